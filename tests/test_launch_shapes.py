"""A launch shape is the library's own choice exactly where the configuration holds
the values that a fresh handle is read with: reading a configuration and setting
it again, on the same handle or another, changes no launch."""
import subprocess
from pathlib import Path

import pytest

import cubiquity_gb300 as cbq

TESTS = Path(__file__).resolve().parent
PERSISTENT = cbq.FORM_PERSISTENT


def test_only_the_fresh_values_are_automatic(tmp_path):
    exe = tmp_path / "launch_shapes"
    subprocess.run(["g++", "-std=c++17", "-Wall", str(TESTS / "launch_shapes.cpp"), "-o", str(exe)], check=True)
    text = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    automatic = {"volume": set(), "batch": set()}
    for kind, refill, steps, form, own in (line.split() for line in text.splitlines()):
        if own == "0":
            automatic[kind].add((int(refill), int(steps), int(form)))
    assert automatic == {"volume": {(0, 0, PERSISTENT)}, "batch": {(16, 8, PERSISTENT)}}


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
