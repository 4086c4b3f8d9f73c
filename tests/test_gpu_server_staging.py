"""The server's staging kernels: page-locked rays in and hits out at every
alignment of the hit buffers, sizes around the 16-byte accesses, missing
fields, and requests whose buffers are only partly page-locked; results equal
the host entry point's and nothing outside a buffer is written."""
import numpy as np
import pytest

import cubiquity_gb300 as cbq
from cubiquity_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GUARD = 64


@pytest.fixture(scope="module")
def scene():
    torch.cuda.set_device(0)
    nodes, root = W.terrain_scaled(7).build()
    (co, cd), _ = W.serve_ray_pools(W.terrain_scaled(7), 70000, 8, 5)
    return cbq.Dag(nodes, root), co, cd


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _buffers(n, shift, fields, pinned=True):
    """(whole guarded byte buffers, hit arrays `shift` bytes off their alignment)."""
    whole, out = {}, {}
    for k, like in cbq.alloc_host_hits(n).items():
        if k not in fields:
            continue
        raw = np.full(like.nbytes + 2 * GUARD, 0xA5, np.uint8)
        raw = _pin(raw) if pinned else raw
        whole[k] = raw
        out[k] = np.frombuffer(raw, like.dtype, like.size, GUARD + shift).reshape(like.shape)
    return whole, out


def _check(whole, shift, want):
    for k, raw in whole.items():
        body = want[k].tobytes()
        lo = GUARD + shift
        assert raw[lo:lo + len(body)].tobytes() == body, k
        assert (raw[:lo] == 0xA5).all() and (raw[lo + len(body):] == 0xA5).all(), f"{k}: written outside"


@pytest.mark.parametrize("n", [1, 3, 4, 5, 15, 16, 17, 31, 33, 1000, 8191, 65537])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4, 7, 13])
def test_staged_hits(scene, n, shift):
    dag, co, cd = scene
    want = cbq.intersect_volume_host(dag, co[:n], cd[:n], use_tmax=True)
    server = cbq.Server(device_memory_budget=64 << 20)
    for fields in (cbq.HIT_FIELDS, ("hit", "distance")):
        whole, out = _buffers(n, shift, fields)
        ticket, _ = server.submit(dag, _pin(co[:n]), _pin(cd[:n]), cbq.Query(use_tmax=True), out)
        assert server.wait(ticket, 20_000_000) == 0
        _check(whole, shift, want)
    server.close()


def test_mixed_buffers_in_one_server(scene):
    """Page-locked, pageable and half page-locked requests together, also under load."""
    dag, co, cd = scene
    server = cbq.Server(device_memory_budget=64 << 20, max_inflight_launches=2)
    jobs = []
    for i in range(48):
        n = 1 + 389 * i
        at = (997 * i) % 40000
        o, d = co[at:at + n], cd[at:at + n]
        if i % 3 != 1:
            o = _pin(o)
        if i % 4 != 2:
            d = _pin(d)
        whole, out = _buffers(n, i % 5, cbq.HIT_FIELDS, pinned=i % 3 != 2)
        if i % 6 == 0:  # one field pageable among page-locked ones
            one, view = _buffers(n, i % 5, ("normal",), pinned=False)
            whole.update(one)
            out.update(view)
        ticket, _ = server.submit(dag, o, d, cbq.Query(use_tmax=True), out)
        jobs.append((ticket, whole, i % 5, cbq.intersect_volume_host(dag, co[at:at + n], cd[at:at + n], use_tmax=True)))
    for ticket, whole, shift, want in jobs:
        assert server.wait(ticket, 20_000_000) == 0
        _check(whole, shift, want)
    server.close()


@pytest.mark.parametrize("n", [1, 3, 16, 33, 65536, 196607, 196608, 393216, 655359, 655360, 655361])
def test_host_call_chunks(scene, n):
    """The host entry point around the sizes where its chunk count changes (the first of chunks
    1:2:3:4 has 65,536 rays at least), with page-locked and pageable buffers, all fields and two."""
    dag, co, cd = scene
    o = np.resize(co, (n, 4)).astype(np.float32)
    d = np.resize(cd, (n, 4)).astype(np.float32)
    o[:, 3] += np.arange(n, dtype=np.float32) % 7  # rays that differ from one copy to the next
    dev = cbq.intersect_volume(dag, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda(), use_tmax=True)
    want = {k: v.cpu().numpy() for k, v in dev.items()}
    want["material"] = want["material"].astype(np.uint32)
    for pinned, shift, fields in ((True, 0, cbq.HIT_FIELDS), (True, 5, ("hit", "position")), (False, 0, cbq.HIT_FIELDS)):
        whole, out = _buffers(n, shift, fields, pinned)
        po, pd = (_pin(o), _pin(d)) if pinned else (o, d)
        cbq.intersect_volume_host(dag, po, pd, use_tmax=True, out=out)
        _check(whole, shift, want)
