"""Device memory of a frame: 260 bytes a path, and in frames small enough for their
workspace to be kept, traced without a callback, a second shadow set (98 more)."""
import gc

import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SLACK = 8 << 20  # the image, counters, padding, CUDA's own granularity


def _used():
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.fixture(autouse=True)
def nothing_left_over():
    """Device memory of earlier tests is given back before a test looks at what is used."""
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def scene():
    torch.cuda.set_device(0)
    dag = cbq.Dag(*W.SceneSpec(cbq.SCENE_CITY, 9, 31).build())
    _frame(dag, 64, 64, 1)  # kernels and streams
    dag.destroy()
    return W.SceneSpec(cbq.SCENE_CITY, 9, 31).build()


def _frame(dag, width, height, samples, on_wave=None):
    eye, target = W.city_camera(9)
    return cbq.pathtrace(dag, width, height, samples, 1, eye, target, W.city_materials(), seed=3, on_wave=on_wave)


@pytest.mark.parametrize("width,height,samples", [(640, 360, 4), (2048, 2048, 1), (2048, 1024, 6)])
def test_wave_by_wave(scene, width, height, samples):
    dag = cbq.Dag(*scene)
    torch.empty((height, width, 3), device="cuda")  # torch's segment for the image: cached from here on
    before, seen = _used(), []
    _frame(dag, width, height, samples, on_wave=lambda *a: seen.append(_used()))
    assert 0 < max(seen) - before <= 260 * width * height * samples + 12 * width * height + SLACK
    dag.destroy()


def test_kept_between_frames(scene):
    dag = cbq.Dag(*scene)
    before = _used()
    for _ in range(2):
        image, _ = _frame(dag, 640, 360, 4)
    del image
    torch.cuda.empty_cache()
    assert _used() - before <= 358 * 640 * 360 * 4 + SLACK
    _frame(dag, 2048, 2048, 2)  # beyond what is kept
    torch.cuda.empty_cache()
    assert _used() - before <= SLACK
    dag.destroy()


def test_kept_over_all_volumes(scene):
    """Nine volumes that rendered a frame of 330 MB keep 1 GiB together; destroyed, nothing."""
    before = _used()
    dags = [cbq.Dag(*scene) for _ in range(9)]
    volumes = _used() - before
    want = None
    for dag in dags + dags[::-1]:
        image, stats = _frame(dag, 640, 360, 4)
        want = stats if want is None else want
        assert stats["extension_rays"] == want["extension_rays"] and stats["shadow_rays"] == want["shadow_rays"]
    del image
    torch.cuda.empty_cache()
    kept = _used() - before - volumes
    assert 358 * 640 * 360 * 4 * 2 < kept <= (1 << 30) + 9 * (2 << 20) + SLACK
    for dag in dags:
        dag.destroy()
    dag = cbq.Dag(*scene)
    _frame(dag, 640, 360, 4)  # room again
    torch.cuda.empty_cache()
    assert _used() - before > 300 * 640 * 360 * 4
    dag.destroy()
    assert _used() - before <= SLACK
