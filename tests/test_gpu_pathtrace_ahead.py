"""Frames traced without a wave callback keep their ray counts on the device and
run shadow waves beside extension waves; with a callback the host reads each
count.  Both trace the same rays: equal counts, and equal images up to the order
in which a pixel's contributions are added."""
import threading

import numpy as np
import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W
from dagbuild import build_dag, random_voxels

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def city():
    torch.cuda.set_device(0)
    return W.SceneSpec(cbq.SCENE_CITY, 9, 31).build()


def _frame(dag, edge_log2, width, height, samples, bounces, on_wave=None, seed=3, materials=None, shift=0.0):
    eye, target = W.city_camera(edge_log2)
    eye = tuple(v + shift for v in eye)
    target = tuple(v + shift for v in target)
    return cbq.pathtrace(dag, width, height, samples, bounces, eye, target,
                         W.city_materials() if materials is None else materials, seed=seed, on_wave=on_wave)


def _close(a, b, terms):
    """Sums of the same `terms` non-negative floats in another order: each addition rounds once
    (2^-24 relative), so two sums differ by at most 2 * terms * 2^-24 of the sum."""
    a, b = a.double(), b.double()
    assert torch.isfinite(a).all()
    assert ((a - b).abs() <= 2.0 * terms * 2.0 ** -24 * torch.maximum(a, b)).all()


@pytest.mark.parametrize("width,height,samples,bounces", [(1, 1, 1, 0), (33, 17, 1, 0), (64, 40, 3, 3), (333, 217, 2, 5),
                                                          (640, 360, 4, 2)])
@pytest.mark.parametrize("layout", [cbq.LAYOUT_REFERENCE, cbq.LAYOUT_COMPACT])
def test_ahead_equals_wave_by_wave(city, layout, width, height, samples, bounces):
    dag = cbq.Dag(*city, layout)
    want, ws = _frame(dag, 9, width, height, samples, bounces, on_wave=lambda *a: None)
    for _ in range(2):  # a new workspace, then the kept one
        got, gs = _frame(dag, 9, width, height, samples, bounces)
        assert (gs["extension_rays"], gs["shadow_rays"]) == (ws["extension_rays"], ws["shadow_rays"])
        _close(got, want, samples * (bounces + 1) * 4)


def test_several_passes(city):
    """More paths than one pass holds: the shadow sets and counters of two passes."""
    dag = cbq.Dag(*city)
    want, ws = _frame(dag, 9, 2048, 2048, 5, 1, on_wave=lambda *a: None)
    got, gs = _frame(dag, 9, 2048, 2048, 5, 1)
    assert (gs["extension_rays"], gs["shadow_rays"]) == (ws["extension_rays"], ws["shadow_rays"])
    _close(got, want, 5 * 2 * 4)


@pytest.mark.parametrize("config", ["integer", "nested", "local", "plain"])
def test_other_forms(config):
    torch.cuda.set_device(0)
    rng = np.random.default_rng(8)
    edge = 32
    at = (1 << 30) if config == "integer" else 0
    nodes, root = build_dag(random_voxels(rng, edge), (at, at, at))
    dag = cbq.Dag(nodes, root)
    if config == "nested":
        dag.set_launch_config(cbq.KERNEL_NESTED)
    elif config == "local":
        dag.set_launch_config(stack=cbq.STACK_LOCAL)
    elif config == "plain":
        dag.set_launch_config(form=cbq.FORM_PLAIN)
    mats = np.full((256, 2, 3), 0.5, np.float32)
    want, ws = _frame(dag, 5, 96, 64, 2, 2, on_wave=lambda *a: None, materials=mats, shift=float(at))
    got, gs = _frame(dag, 5, 96, 64, 2, 2, materials=mats, shift=float(at))
    assert (gs["extension_rays"], gs["shadow_rays"]) == (ws["extension_rays"], ws["shadow_rays"])
    _close(got, want, 2 * 3 * 4)


def test_frames_from_several_threads(city):
    """Frames of one DAG at the same time: one has the kept workspace, the others their own."""
    dag = cbq.Dag(*city)
    want = [_frame(dag, 9, 200, 120, 2, 3, on_wave=lambda *a: None, seed=10 + i)[0] for i in range(4)]
    got = [None] * 4

    def work(i):
        torch.cuda.set_device(0)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(3):
                got[i], _ = _frame(dag, 9, 200, 120, 2, 3, seed=10 + i)
            stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        _close(a, b, 2 * 4 * 4)
