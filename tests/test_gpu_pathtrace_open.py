"""Frames of an open scene with many bounces: the paths are all gone after a few
depths, and the depths that nothing can come to are not launched."""
import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

AHEAD = 4     # waves queued ahead of the last one whose count the host has looked at
PER_WAVE = 4  # launches: extension, shade, shadow, add


@pytest.fixture(scope="module")
def dag():
    torch.cuda.set_device(0)
    return cbq.Dag(*W.SceneSpec(cbq.SCENE_SPHERES, 7, 7, 1).build())


def _frame(dag, width, height, samples, bounces, on_wave=None):
    return cbq.pathtrace(dag, width, height, samples, bounces, (-150.0, -150.0, 150.0), (64.0, 64.0, 64.0),
                         W.city_materials(), seed=5, on_wave=on_wave)


@pytest.mark.parametrize("bounces", [0, 1, 3, 4, 5, 6, 16, 63, 64])
@pytest.mark.parametrize("width,height,samples,passes", [(1, 1, 1, 1), (97, 61, 2, 1), (640, 360, 1, 1), (2048, 2048, 5, 2)])
def test_depths_without_paths(dag, width, height, samples, passes, bounces):
    if passes > 1 and bounces not in (4, 64):
        pytest.skip("two passes: a short and a long frame")
    waves = []
    want, ws = _frame(dag, width, height, samples, bounces, on_wave=lambda kind, *a: waves.append(kind))
    live = waves.count(0)  # depths with rays
    for _ in range(2):
        got, gs = _frame(dag, width, height, samples, bounces)
        assert (gs["extension_rays"], gs["shadow_rays"]) == (ws["extension_rays"], ws["shadow_rays"])
        assert gs["kernel_launches"] <= 1 + passes + PER_WAVE * min(live + passes * AHEAD, passes * (bounces + 1))
        a, b = got.double(), want.double()
        # Sums of the same non-negative floats in another order: each addition rounds once.
        assert ((a - b).abs() <= 2.0 * samples * (bounces + 1) * 4 * 2.0 ** -24 * torch.maximum(a, b)).all()
