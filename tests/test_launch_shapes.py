"""A launch shape is the library's own choice exactly where the configuration holds
the values that a fresh handle is read with: reading a configuration and setting
it again, on the same handle or another, changes no launch."""
import subprocess
from pathlib import Path

import pytest

import cubiquity_gb300 as cbq

TESTS = Path(__file__).resolve().parent
PERSISTENT = cbq.FORM_PERSISTENT


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = tmp_path_factory.mktemp("shapes") / "launch_shapes"
    subprocess.run(["g++", "-std=c++17", "-Wall", str(TESTS / "launch_shapes.cpp"), "-o", str(exe)], check=True)
    text = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [(kind, *(int(v) for v in rest)) for kind, *rest in (line.split() for line in text.splitlines())]


def test_only_the_fresh_values_are_automatic(lines):
    automatic = {"volume": set(), "batch": set()}
    for kind, *values in lines:
        if kind in automatic and values[3] == 0:
            automatic[kind].add(tuple(values[:3]))
    assert automatic == {"volume": {(0, 0, PERSISTENT)}, "batch": {(16, 8, PERSISTENT)}}


def test_the_tuner_times_the_automatic_shape(lines):
    tuned = [line[1:] for line in lines if line[0] == "tuned"]
    want = {(form, block, refill, steps, stack) for block in (64, 128, 256) for stack in (0, 1)
            for form, refills in ((cbq.FORM_PLAIN, (0,)), (PERSISTENT, (8, 16, 24)), (cbq.FORM_SORTED, (8, 16, 24)))
            for refill in refills for steps in (4, 8, 16, 32)}
    want |= {(form, block, 0, 0, stack) for form in (PERSISTENT, cbq.FORM_SORTED) for block in (64, 128, 256)
             for stack in (0, 1)}
    assert len(tuned) == len(set(tuned)) and set(tuned) == want


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1000, 100_000])
def test_auto_takes_the_automatic_shape(n):
    """A spread launch has no work counter: intersect_auto leaves the counter in its scratch as it was."""
    torch = pytest.importorskip("torch")
    from cubiquity_gb300 import workloads as W
    torch.cuda.set_device(0)
    spec = W.terrain_scaled(7)
    dag = cbq.Dag(*spec.build())
    (o, d), _ = W.serve_ray_pools(spec, n, 8, 5)
    o, d, scratch = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(), cbq.scratch_for(n)
    want = cbq.intersect_volume(dag, o, d)
    for kw, spread in (({}, True), ({"refill_min": 16, "steps": 8}, False), ({"form": cbq.FORM_SORTED}, False)):
        dag.set_launch_config(**kw)
        scratch.fill_(0x5A)
        got = cbq.intersect_auto(dag, o, d, scratch)
        assert bool((scratch[:8] == 0x5A).all()) == spread, kw
        for k, v in want.items():
            assert torch.equal(v.view(torch.uint8), got[k].view(torch.uint8)), (kw, k)


@pytest.mark.gpu
def test_fresh_batch_has_the_automatic_values():
    torch = pytest.importorskip("torch")
    from cubiquity_gb300 import workloads as W
    torch.cuda.set_device(0)
    spec = W.terrain_scaled(7)
    dag = cbq.Dag(*spec.build())
    (o, d), _ = W.serve_ray_pools(spec, 3000, 8, 5)
    job = (dag, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    batch, other = cbq.Batch([job]), cbq.Batch([job])
    read = batch.config()
    assert (read["refill_min"], read["steps"], read["form"]) == (16, 8, PERSISTENT)
    shape = {k: read[k] for k in ("block", "refill_min", "steps", "registers", "stack", "form")}
    other.set_launch_config(**shape)
    assert other.config() == read
    other.set_config(block=64)
    other.set_config()
    assert other.config() == read
    batch.launch()
    other.launch()
    torch.cuda.synchronize()
    for k, v in batch.outputs[0].items():
        assert torch.equal(v.view(torch.uint8), other.outputs[0][k].view(torch.uint8)), k
