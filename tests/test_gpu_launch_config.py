"""Launch configurations read from one handle and set on another give the same
launches: nothing that is chosen by the library comes back as a fixed shape."""
import numpy as np
import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def scene():
    torch.cuda.set_device(0)
    return W.terrain_scaled(7).build()


@pytest.mark.parametrize("kw", [
    {}, {"refill_min": 12}, {"steps": 4}, {"refill_min": 16, "steps": 8}, {"block": 256}, {"stack": cbq.STACK_LOCAL},
    {"form": cbq.FORM_PLAIN}, {"form": cbq.FORM_SORTED, "steps": 16}, {"kernel": cbq.KERNEL_NESTED, "chunk": 32},
    {"registers": 56}])
def test_volume_configuration_round_trip(scene, kw):
    dag, other = cbq.Dag(*scene), cbq.Dag(*scene)
    dag.set_launch_config(**kw)
    read = dag.launch_config()
    for k in ("refill_min", "steps", "form", "stack", "registers"):
        assert read[k] == kw.get(k, cbq.FORM_PERSISTENT if k == "form" else 0), k
    other.set_launch_config(**read)
    assert other.launch_config() == read
