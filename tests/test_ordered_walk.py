"""The ordered walk's rules where they can go wrong: rays on both sides of its
condition, origins inside, on and behind volumes, volumes in several octants,
volumes at +-2^21, the LOD threshold.  On the CPU a plain restatement of the
rules (ordered_walk.cpp) against the oracle; on the GPU the kernels against the
oracle, bit for bit."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import cubiquity_gb300 as cbq
import oracle
from dagbuild import build_dag, random_voxels

FIELDS = ("hit", "distance", "material", "position", "normal", "voxel", "status")
FOOTPRINTS = (-1.0, 0.0, 0.0035, 0.02, 0.3, 1.0, 2.0)
DIR_MIN, DIR_MAX, ORIGIN_MAX = np.float32(2.0 ** -60), np.float32(2.0 ** 60), np.float32(2.0 ** 21)


def _join(volumes):
    """One DAG of several (nodes, root), each in octants of its own."""
    rows = [np.repeat(np.arange(256, dtype=np.uint32)[:, None], 8, axis=1)]
    top = np.zeros(8, np.uint32)
    for nodes, root in volumes:
        n = nodes.reshape(-1, 8).copy()
        shift = sum(r.shape[0] for r in rows) - 256
        n[256:][n[256:] >= 256] += np.uint32(shift)
        top |= n[root]
        rows.append(n[256:])
    rows.append(top[None])
    all_rows = np.concatenate(rows)
    return all_rows.reshape(-1), all_rows.shape[0] - 1


def _volume(seed):
    """(nodes, root, centre, edge): one random box, or one in each of three octants."""
    rng = np.random.default_rng(4000 + seed)
    edge = 1 << int(rng.integers(2, 7))
    vox = random_voxels(rng, edge)
    if seed % 4 == 3:  # around the origin, in three octants
        boxes = [build_dag(random_voxels(rng, edge), tuple(int(v) for v in o))
                 for o in ((0, 0, 0), (-edge, 0, -edge), (-edge, -edge, 0))]
        return (*_join(boxes), np.zeros(3), 2 * edge)
    if seed % 4 == 2:  # touching +-2^21, the last coordinates of the float positions
        low = tuple(int(v) for v in rng.choice(((1 << 21) - edge, -(1 << 21)), 3))
    else:
        low = tuple(int(v) * edge for v in rng.integers(-64, 64, 3))
    return (*build_dag(vox, low), np.array(low) + edge / 2.0, edge)


def _rays(seed, centre, edge, n=6000):
    rng = np.random.default_rng(9000 + seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    out = rng.random(n)
    o = centre + rng.uniform(-0.5, 0.5, (n, 3)) * edge * np.where(out < 0.4, 1.0, 3.0)[:, None]
    away = out > 0.7  # from outside: towards the volume, or past it, the volume behind
    o[away] = centre + d[away] * -2.0 * edge * rng.choice((1.0, 1.0, -1.0), away.sum())[:, None]
    o[away] += rng.uniform(-0.4, 0.4, (int(away.sum()), 3)) * edge
    snap = rng.random(n) < 0.25  # on voxel faces and centres
    o[snap] = np.round(o[snap] * 2.0) / 2.0
    o4 = np.zeros((n, 4), np.float32)
    d4 = np.zeros((n, 4), np.float32)
    o4[:, :3], d4[:, :3] = o, d
    o4[:, 3] = np.inf
    diagonal = rng.random(n) < 0.1
    d4[diagonal, :3] = rng.choice(np.array([-1.0, 1.0, 0.5], np.float32), (int(diagonal.sum()), 3))
    # Components at the ends of the ordered range, just outside it, and zero.
    odd = np.nonzero(rng.random(n) < 0.2)[0]
    vals = np.array([DIR_MIN, np.nextafter(DIR_MIN, np.float32(0)), 1e-6, 1e-3, DIR_MAX,
                     np.nextafter(DIR_MAX, np.float32(np.inf)), 0.0, 1e30, 1e-30], np.float32)
    d4[odd, rng.integers(0, 3, odd.size)] = rng.choice(vals, odd.size) * rng.choice((-1.0, 1.0), odd.size)
    far = np.nonzero(rng.random(n) < 0.03)[0]
    o4[far, rng.integers(0, 3, far.size)] = rng.choice(
        np.array([ORIGIN_MAX, -ORIGIN_MAX, ORIGIN_MAX - 1, 3e6, -5e7], np.float32), far.size)
    return o4, d4


def _ordered(o, d):
    sign = np.where(d[:, :3] < 0, np.float32(-1), np.float32(1))
    ro = np.abs((o[:, :3] + np.float32(0.5)) * sign)
    rd = np.abs(d[:, :3])
    return ((ro <= ORIGIN_MAX) & (rd >= DIR_MIN) & (rd <= DIR_MAX)).all(axis=1)


def _exit_max(mf):
    fn = getattr(cbq.lib(), "_ZN3cbq18footprint_exit_maxEf")
    fn.argtypes, fn.restype = [ctypes.c_float], ctypes.c_float
    return fn(mf)


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    so = tmp_path_factory.mktemp("walk") / "ordered_walk.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(so),
                    str(Path(__file__).with_name("ordered_walk.cpp"))], check=True)
    lib = ctypes.CDLL(str(so))

    def run(nodes, subdags, o, d, mf):
        n = o.shape[0]
        out = {"hit": np.zeros(n, np.uint8), "distance": np.zeros(n, np.float32), "node": np.zeros(n, np.uint32),
               "fetches": np.zeros(n, np.uint32), "status": np.zeros(n, np.uint8)}
        arr = oracle._subdag_array(subdags)
        lib.ordered_trace(nodes.ctypes.data_as(ctypes.c_void_p), ctypes.byref(arr),
                          o.ctypes.data_as(ctypes.c_void_p), d.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(n),
                          ctypes.c_float(mf), ctypes.c_float(_exit_max(mf)),
                          *[out[k].ctypes.data_as(ctypes.c_void_p) for k in
                            ("hit", "distance", "node", "fetches", "status")])
        return out
    return run


@pytest.mark.parametrize("seed", range(16))
def test_rules_against_the_oracle(seed, orc, walk):
    nodes, root, centre, edge = _volume(seed)
    sd = orc.find_subdags(nodes, root)
    o, d = _rays(seed, centre, edge)
    keep = _ordered(o, d)
    assert 0.3 < keep.mean() < 1.0  # at +-2^21 about half of the origins lie beyond the range
    o, d = np.ascontiguousarray(o[keep]), np.ascontiguousarray(d[keep])
    for mf in FOOTPRINTS:
        want = orc.intersect(nodes, sd, o, d, False, mf)
        fetches = orc.count_fetches(nodes, sd, o, d, False, mf)
        got = walk(nodes, sd, o, d, mf)
        assert not (got["status"] > 3).any()
        own = got["status"] == 0  # the others are handed to the reference's steps
        assert own.mean() > 0.5
        for k in ("hit", "distance"):
            assert np.array_equal(got[k][own].view(np.uint8), want[k][own].view(np.uint8)), (k, mf)
        assert np.array_equal(got["fetches"][own], fetches[own]), mf


@pytest.mark.filterwarnings("ignore:overflow")
def test_footprint_exit_is_the_quotient_s_boundary():
    """t <= s * exit exactly where float32(s / t) > max_footprint, s a power of two."""
    rng = np.random.default_rng(5)
    mfs = np.concatenate([[0.0, 1.0, 0.0035, 3e38, 1e-38, 2e-39, 1e-45, np.float32(1) / 3], rng.random(200),
                          np.exp(rng.uniform(-60, 60, 200))]).astype(np.float32)
    for mf in mfs:
        lim = np.float32(_exit_max(float(mf)))
        t = np.abs(np.float32(1) / mf) if mf > 0 else np.float32(1)
        near = [t]
        for _ in range(40):
            near.append(np.nextafter(near[-1], np.float32(0)))
        near += [np.nextafter(t, np.float32(np.inf))]
        for _ in range(40):
            near.append(np.nextafter(near[-1], np.float32(np.inf)))
        t = np.concatenate([np.array(near, np.float32), np.exp(rng.uniform(-58, 57, 500)).astype(np.float32)])
        for s in (1.0, 2.0, 1024.0, 2.0 ** 20):
            ts = (t * np.float32(s)).astype(np.float32)
            ts = ts[(ts >= 2.0 ** -85) & (ts <= 2.0 ** 83)]
            assert np.array_equal(np.float32(s) / ts > mf, ts <= np.float32(s) * lim), (mf, s)
    assert _exit_max(-1.0) == np.inf and _exit_max(float("inf")) == -1.0 and _exit_max(float("nan")) == -1.0


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(8))
def test_kernels_against_the_oracle(seed, orc):
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    nodes, root, centre, edge = _volume(seed)
    sd = orc.find_subdags(nodes, root)
    o, d = _rays(seed, centre, edge)
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    for mf in FOOTPRINTS:
        want = orc.intersect(nodes, sd, o, d, True, mf)
        for layout in (cbq.LAYOUT_REFERENCE, cbq.LAYOUT_COMPACT):
            dag = cbq.Dag(nodes, root, layout)
            for stack in (cbq.STACK_SHARED, cbq.STACK_LOCAL):
                for form, refill, steps in ((cbq.FORM_PERSISTENT, 0, 8), (cbq.FORM_PERSISTENT, 1, 1),
                                            (cbq.FORM_PLAIN, 0, 32)):
                    dag.set_launch_config(cbq.KERNEL_FLAT, 64, 0, refill, stack, form, steps)
                    got = cbq.intersect_volume(dag, to, td, True, mf)
                    batch = cbq.Batch([(dag, to, td)], True, mf)
                    batch.launch()
                    torch.cuda.synchronize()
                    for what, res in (("call", got), ("batch", batch.outputs[0])):
                        for k in FIELDS:
                            g = res[k].cpu().numpy()
                            w = want[k]
                            if k == "material":
                                g, w = g.astype(np.uint32), w.astype(np.uint32)
                            assert oracle.same_bits_nan_equal(g, w), (what, k, mf, layout, stack, form, refill)


@pytest.mark.gpu
def test_store_beyond_the_tagged_range(orc):
    """2^24 + 1 nodes (padded with unused ones): the walk on the plain store, alone, in a
    batch beside a tagged volume and in a server, against the oracle."""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    small, root, centre, edge = _volume(3)
    nodes = np.zeros(((1 << 24) + 1) * 8, np.uint32)
    nodes[:small.size] = small
    sd = orc.find_subdags(small, root)
    o, d = _rays(3, centre, edge)
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    dag, tagged = cbq.Dag(nodes, root), cbq.Dag(small, root)
    for mf in (-1.0, 0.02):
        want = orc.intersect(small, sd, o, d, True, mf)
        got = cbq.intersect_volume(dag, to, td, True, mf)
        batch = cbq.Batch([(dag, to, td), (tagged, to, td)], True, mf)
        batch.launch()
        server = cbq.Server(device_memory_budget=16 << 20)
        ticket, served = server.submit(dag, o, d, cbq.Query(True, mf))
        assert server.wait(ticket, 20_000_000) == 0
        torch.cuda.synchronize()
        for res in (got, batch.outputs[0], batch.outputs[1], served):
            for k in FIELDS:
                g = res[k] if isinstance(res[k], np.ndarray) else res[k].cpu().numpy()
                assert oracle.same_bits_nan_equal(g.astype(want[k].dtype) if k == "material" else g, want[k]), (k, mf)
        server.close()


@pytest.mark.gpu
@pytest.mark.parametrize("log2", [1, 4, 5, 6, 7])
def test_origins_inside_around_the_table_s_height(log2, orc):
    """Rays from inside volumes whose SubDAG has no table of upper cells (height 5 and below),
    ends right below it (6) and goes on (7), in one octant and in three, both layouts."""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    rng = np.random.default_rng(70 + log2)
    edge = 1 << log2
    for places in (((0, 0, 0),), ((-edge, 0, 0), (0, -edge, -edge), (0, 0, 0)), ((-(1 << 21),) * 3,)):
        nodes, root = _join([build_dag(random_voxels(rng, edge) if log2 > 1 else
                                       rng.integers(0, 2, (2, 2, 2)).astype(np.uint8) * 7, p) for p in places])
        sd = orc.find_subdags(nodes, root)
        n = 4000
        at = np.array(places, np.float64)[rng.integers(0, len(places), n)]
        o = np.zeros((n, 4), np.float32)
        d = rng.normal(size=(n, 4)).astype(np.float32)
        o[:, :3] = at + rng.uniform(-0.5, edge - 0.5, (n, 3))
        snap = rng.random(n) < 0.3
        o[snap, :3] = np.round(o[snap, :3] * 2.0) / 2.0
        o[:, 3] = np.inf
        to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
        for mf in (-1.0, 0.0035, 0.4, 3.0):
            want = orc.intersect(nodes, sd, o, d, True, mf)
            for layout in (cbq.LAYOUT_REFERENCE, cbq.LAYOUT_COMPACT):
                dag = cbq.Dag(nodes, root, layout)
                for stack in (cbq.STACK_SHARED, cbq.STACK_LOCAL):
                    dag.set_launch_config(stack=stack)
                    got = cbq.intersect_volume(dag, to, td, True, mf)
                    for k in FIELDS:
                        g = got[k].cpu().numpy()
                        assert oracle.same_bits_nan_equal(g.astype(want[k].dtype) if k == "material" else g,
                                                          want[k]), (k, mf, layout, stack, places)


@pytest.mark.gpu
@pytest.mark.parametrize("places", [((0, 0, 0),), ((-32, 0, -32),), ((0, 0, 0), (-32, -32, 0)),
                                    ((0, 0, 0), (0, -32, 0), (-32, -32, -32), (-32, 0, 0))])
def test_rays_from_other_octants(places, orc):
    """Volumes in one, two and four octants met from all the others, with crossings of the
    planes between that tie exactly or differ by a few units in the last place."""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    rng = np.random.default_rng(len(places))
    nodes, root = _join([build_dag(random_voxels(rng, 32), p) for p in places])
    sd = orc.find_subdags(nodes, root)
    n = 60000
    o = np.zeros((n, 4), np.float32)
    d = np.zeros((n, 4), np.float32)
    o[:, :3] = rng.integers(-128, 129, (n, 3)) * 0.5 - 0.5
    d[:, :3] = rng.choice(np.array([-2.0, -1.0, -0.5, -0.75, 0.25, 0.75, 1.0, 3.0], np.float32), (n, 3))
    toward = rng.random(n) < 0.5  # through a point near the origin's planes: close calls of their order
    d[toward, :3] = -(o[toward, :3] + np.float32(0.5)) + rng.integers(-1, 2, (int(toward.sum()), 3)) * np.float32(1e-5)
    for a in range(3):
        bump = rng.random(n) < 0.3
        d[bump, a] = np.nextafter(d[bump, a], rng.choice(np.array([-9.0, 9.0], np.float32), int(bump.sum())))
    o[:, 3] = np.inf
    dag = cbq.Dag(nodes, root)
    got = cbq.intersect_volume(dag, torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda())
    want = orc.intersect(nodes, sd, o, d)
    assert 0 < int(want["hit"].sum()) < n
    for k in FIELDS:
        g = got[k].cpu().numpy()
        assert oracle.same_bits_nan_equal(g.astype(want[k].dtype) if k == "material" else g, want[k]), k


@pytest.mark.gpu
@pytest.mark.parametrize("places", [((1 << 23, 0, 0),), ((1 << 23, 0, 1 << 22), (-32, -32, 0), (-32, 0, -32)),
                                    ((0, 0, 0), (-(1 << 22), 0, 0), (-(1 << 31), -32, -32))])
def test_rays_between_octants_of_far_volumes(places, orc):
    """Integer positions: volumes beyond +-2^21 and around the origin met from all octants, from
    origins up to 2^31, directions on both sides of the octant rules' range, and close calls."""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    rng = np.random.default_rng(len(places))
    nodes, root = _join([build_dag(random_voxels(rng, 32), p) for p in places])
    sd = orc.find_subdags(nodes, root)
    n = 60000
    o = np.zeros((n, 4), np.float32)
    d = np.zeros((n, 4), np.float32)
    target = np.array(places, np.float64)[rng.integers(0, len(places), n)] + rng.uniform(0.0, 32.0, (n, 3))
    away = np.exp2(rng.uniform(3.0, 31.0, n))[:, None]
    way = rng.normal(size=(n, 3))
    way /= np.linalg.norm(way, axis=1, keepdims=True)
    o[:, :3] = np.clip(target - way * away, -(2.0 ** 31), 2.0 ** 31)
    d[:, :3] = way
    near = rng.random(n) < 0.4
    o[near, :3] = rng.integers(-128, 129, (int(near.sum()), 3)) * 0.5 - 0.5
    toward = rng.random(n) < 0.3  # through a point near the origin's planes: close calls of their order
    d[toward, :3] = -(o[toward, :3] + np.float32(0.5)) + rng.integers(-1, 2, (int(toward.sum()), 3)) * np.float32(1e-5)
    odd = np.nonzero(rng.random(n) < 0.1)[0]
    vals = np.array([DIR_MIN, np.nextafter(DIR_MIN, np.float32(0)), DIR_MAX,
                     np.nextafter(DIR_MAX, np.float32(np.inf)), 0.0, 1e-38, 1e-30, 1e30], np.float32)
    d[odd, rng.integers(0, 3, odd.size)] = rng.choice(vals, odd.size) * rng.choice((-1.0, 1.0), odd.size)
    beyond = np.nonzero(rng.random(n) < 0.02)[0]
    o[beyond, rng.integers(0, 3, beyond.size)] = rng.choice(
        np.array([2.0 ** 32, -(2.0 ** 32), 4.3e9, -1e12, 1e30], np.float32), beyond.size)
    o[:, 3] = np.inf
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    dag = cbq.Dag(nodes, root)
    for mf in (-1.0, 0.02):
        want = orc.intersect(nodes, sd, o, d, True, mf)
        assert 0 < int(want["hit"].sum()) < n
        for stack, form in ((cbq.STACK_SHARED, cbq.FORM_PERSISTENT), (cbq.STACK_LOCAL, cbq.FORM_PLAIN)):
            dag.set_launch_config(stack=stack, form=form)
            got = cbq.intersect_volume(dag, to, td, True, mf)
            for k in FIELDS:
                g = got[k].cpu().numpy()
                assert oracle.same_bits_nan_equal(g.astype(want[k].dtype) if k == "material" else g, want[k]), (k, mf)


@pytest.mark.gpu
@pytest.mark.parametrize("footprints", [(-1.0,), (0.02,), (-1.0, 0.02, 0.0, -1.0, 1.0, float("inf"), float("nan"))])
def test_requests_with_and_without_lod(footprints, orc):
    """Server groups of requests with and without a footprint, in both layouts, against the oracle."""
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    nodes, root, centre, edge = _volume(3)
    sd = orc.find_subdags(nodes, root)
    o, d = _rays(3, centre, edge, 3000)
    for layout in (cbq.LAYOUT_REFERENCE, cbq.LAYOUT_COMPACT):
        dag = cbq.Dag(nodes, root, layout)
        server = cbq.Server(device_memory_budget=64 << 20)
        asked = [(mf, *server.submit(dag, o, d, cbq.Query(True, mf))) for mf in footprints * 12]
        for mf, ticket, got in asked:
            assert server.wait(ticket, 20_000_000) == 0
            want = orc.intersect(nodes, sd, o, d, True, mf)
            for k in FIELDS:
                g = got[k].astype(want[k].dtype) if k == "material" else got[k]
                assert oracle.same_bits_nan_equal(g, want[k]), (k, mf, layout)
        server.close()


def _parallel_rays(seed, centre, edge, n=6000):
    """Rays with one, two or three components of exactly 0 (or -0), origins on voxel faces and off them."""
    rng = np.random.default_rng(600 + seed)
    o, d = _rays(seed, centre, edge, n)
    for a in range(3):
        zero = rng.random(n) < 0.45
        d[zero, a] = rng.choice(np.array([0.0, -0.0], np.float32), int(zero.sum()))
    aim = rng.random(n) < 0.6  # along the zero axes the origin lies within the volume
    within = (centre + rng.uniform(-0.5, 0.5, (n, 3)) * edge).astype(np.float32)
    o[:, :3] = np.where(aim[:, None] & (d[:, :3] == 0), within, o[:, :3])
    snap = rng.random(n) < 0.3
    o[snap, :3] = np.round(o[snap, :3] * 4.0) / 4.0
    return o, d


def _parallel(o, d):
    """The rays that the ordered walk takes beside those of _ordered."""
    sign = np.where(d[:, :3] < 0, np.float32(-1), np.float32(1))
    ro = (o[:, :3] + np.float32(0.5)) * sign
    rd = np.abs(d[:, :3])
    zero = (rd == 0) & (np.trunc(ro) != ro)
    ok = (np.abs(ro) <= ORIGIN_MAX) & (zero | ((rd >= DIR_MIN) & (rd <= DIR_MAX)))
    return ok.all(axis=1) & ~zero.all(axis=1) & zero.any(axis=1)


@pytest.mark.parametrize("seed", range(12))
@pytest.mark.filterwarnings("ignore:divide by zero")
def test_rules_of_parallel_rays(seed, orc, walk):
    nodes, root, centre, edge = _volume(seed)
    sd = orc.find_subdags(nodes, root)
    o, d = _parallel_rays(seed, centre, edge)
    keep = _parallel(o, d)
    assert keep.sum() > 200
    o, d = np.ascontiguousarray(o[keep]), np.ascontiguousarray(d[keep])
    for mf in FOOTPRINTS:
        want = orc.intersect(nodes, sd, o, d, False, mf)
        fetches = orc.count_fetches(nodes, sd, o, d, False, mf)
        got = walk(nodes, sd, o, d, mf)
        assert not (got["status"] > 3).any()
        own = got["status"] == 0
        assert own.mean() > 0.5
        for k in ("hit", "distance"):
            assert np.array_equal(got[k][own].view(np.uint8), want[k][own].view(np.uint8)), (k, mf)
        assert np.array_equal(got["fetches"][own], fetches[own]), mf


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(8))
def test_kernels_on_parallel_rays(seed, orc):
    torch = pytest.importorskip("torch")
    torch.cuda.set_device(0)
    nodes, root, centre, edge = _volume(seed)
    sd = orc.find_subdags(nodes, root)
    o, d = _parallel_rays(seed, centre, edge)
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    for mf in (-1.0, 0.0035, 0.3):
        want = orc.intersect(nodes, sd, o, d, True, mf)
        for layout in (cbq.LAYOUT_REFERENCE, cbq.LAYOUT_COMPACT):
            dag = cbq.Dag(nodes, root, layout)
            for stack, form in ((cbq.STACK_SHARED, cbq.FORM_PERSISTENT), (cbq.STACK_LOCAL, cbq.FORM_PLAIN)):
                dag.set_launch_config(stack=stack, form=form)
                got = cbq.intersect_volume(dag, to, td, True, mf)
                batch = cbq.Batch([(dag, to, td)], True, mf)
                batch.launch()
                torch.cuda.synchronize()
                for what, res in (("call", got), ("batch", batch.outputs[0])):
                    for k in FIELDS:
                        g = res[k].cpu().numpy()
                        assert oracle.same_bits_nan_equal(g.astype(want[k].dtype) if k == "material" else g,
                                                          want[k]), (what, k, mf, layout, stack)
