"""Launches without a caller's shape: small ones are spread over the chip's warps
(fewer rays per warp, no work counter), larger ones refill by what their rays
look like.  Around the sizes where the rays per warp change and where spreading
ends, the results are those of the persistent form with an explicit shape."""
import numpy as np
import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

WARPS_PER_SM = 32


@pytest.fixture(scope="module")
def scene():
    torch.cuda.set_device(0)
    warps = torch.cuda.get_device_properties(0).multi_processor_count * WARPS_PER_SM
    nodes, root = W.terrain_scaled(8).build()
    n = 32 * warps + 2048
    (co, cd), _ = W.serve_ray_pools(W.terrain_scaled(8), n, 8, 7)
    wide = W.camera_scaled(8, 512, -(-n // 512)).rays()
    dag = cbq.Dag(nodes, root)
    shaped = cbq.Dag(nodes, root)
    shaped.set_launch_config(refill_min=16, steps=8)
    pools = {k: tuple(torch.from_numpy(a).cuda() for a in v) for k, v in (("collision", (co, cd)), ("camera", wide))}
    return dag, shaped, warps, pools


def _same(a, b, what):
    for k in a:
        assert torch.equal(a[k].view(torch.uint8), b[k].view(torch.uint8)), f"{what}: {k}"


@pytest.mark.parametrize("rays", ["collision", "camera"])
@pytest.mark.parametrize("times,extra", [(0, 1), (0, 31), (0, 33), (1, -1), (1, 0), (1, 1), (2, 1), (16, 17), (31, 1),
                                         (32, -1), (32, 0), (32, 1), (32, 2000)])
def test_spread_sizes(scene, rays, times, extra):
    dag, shaped, warps, pools = scene
    n = times * warps + extra
    o, d = (a[:n] for a in pools[rays])
    for kw in ({}, {"use_tmax": True, "compute_surface_properties": False}, {"max_footprint": 0.01}):
        for width in (0, 512):
            want = cbq.intersect_volume(shaped, o, d, image_width=width, **kw)
            _same(cbq.intersect_volume(dag, o, d, image_width=width, **kw), want, f"{n} {rays} {kw} width {width}")
        counter = torch.zeros(1, dtype=torch.int64, device="cuda")
        _same(cbq.intersect_volume_persistent(dag, o, d, counter, **kw), want, f"persistent {n} {rays} {kw}")
    cut = n // 3
    batch = cbq.Batch([(dag, o[:cut], d[:cut]), (shaped, o[cut:], d[cut:])])
    batch.launch()
    want = cbq.intersect_volume(shaped, o, d)
    got = {k: torch.cat([batch.outputs[0][k], batch.outputs[1][k]]) for k in want}
    _same(got, want, f"batch {n} {rays}")


def test_spread_launch_in_a_capture(scene):
    dag, shaped, warps, pools = scene
    o, d = (a[:3 * warps + 5] for a in pools["collision"])
    out = cbq.alloc_hits(o.shape[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cbq.intersect_volume(dag, o, d, out=out)
    for v in out.values():
        v.zero_()
    graph.replay()
    torch.cuda.synchronize()
    _same(out, cbq.intersect_volume(shaped, o, d), "capture")


@pytest.mark.parametrize("n", [(3 << 19) - 4096, 3 << 19, (3 << 19) + 1, (3 << 19) + 4096])
def test_image_sizes(scene, n):
    """Around the size up to which an image takes one thread per ray: whole bands, ragged ends, host calls."""
    dag, shaped, _, _ = scene
    o, d = W.camera_scaled(8, 512, -(-n // 512)).rays()
    to, td = torch.from_numpy(o[:n]).cuda(), torch.from_numpy(d[:n]).cuda()
    for kw in ({}, {"max_footprint": 0.01}):
        want = cbq.intersect_volume(shaped, to, td, **kw)
        for width in (512, 513):
            _same(cbq.intersect_volume(dag, to, td, image_width=width, **kw), want, f"{n} {kw} width {width}")
    host = cbq.intersect_volume_host(dag, o[:n], d[:n], image_width=512)
    want = cbq.intersect_volume(shaped, to, td)
    for k in want:
        assert want[k].cpu().numpy().tobytes() == host[k].tobytes(), k


@pytest.mark.parametrize("shared_stream", [False, True])
def test_launches_beyond_the_counter_ring(scene, shared_stream):
    """600 persistent launches (a stream's ring holds 256 work counters) from three threads, on streams of
    their own or all on one: every launch traverses all its rays."""
    import threading
    dag, shaped, warps, pools = scene
    o, d = pools["collision"]
    cuts = [o.shape[0] - k for k in (0, 1, 777)]  # beyond the spread sizes
    want = cbq.intersect_volume(shaped, o, d)
    torch.cuda.synchronize()
    one, bad = torch.cuda.Stream(), []

    def run(k):
        torch.cuda.set_device(0)
        stream = one if shared_stream else torch.cuda.Stream()
        n = cuts[k]
        for i in range(200):
            with torch.cuda.stream(stream):
                out = cbq.alloc_hits(n, fields=("hit", "distance"))
                out["distance"].fill_(-1.0)
                cbq.intersect_volume(dag, o[:n], d[:n], out=out, stream=stream)
                same = torch.equal(out["hit"], want["hit"][:n]) and torch.equal(out["distance"], want["distance"][:n])
            if not same:
                bad.append((k, i))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
