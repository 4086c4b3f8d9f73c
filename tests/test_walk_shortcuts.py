"""Two shortcuts of the ordered walk where they can go wrong, restated on the CPU
against the reference's arithmetic: the octants around the origin from products
instead of quotients, and the descent by voxel coordinates."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

TESTS = Path(__file__).resolve().parent
F3 = np.ctypeslib.ndpointer(np.float32, flags="C")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = tmp_path_factory.mktemp("rules") / "walk_shortcuts.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    str(TESTS / "walk_shortcuts.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.octants_differ.restype = lib.descents_differ.restype = ctypes.c_uint64
    lib.octants_differ.argtypes = [ctypes.c_uint64, F3, F3, ctypes.POINTER(ctypes.c_uint64)]
    lib.descents_differ.argtypes = [ctypes.c_uint64, F3, F3, np.ctypeslib.ndpointer(np.int32), ctypes.c_int]
    return lib


def _directions(rng, n):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d = d.astype(np.float32)
    some = rng.random((n, 3)) < 0.1
    d[some] = rng.choice(np.array([1.0, -1.0, 0.5, 1e-6, -1e-6, 2.0 ** -60, -(2.0 ** 60), 3e10], np.float32), some.sum())
    return d


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("reach", [4.0, 1e4, 2.0 ** 21, 2.0 ** 32])
def test_octants(rules, seed, reach):
    rng = np.random.default_rng(100 * seed + int(np.log2(reach)))
    n = 4000
    d = _directions(rng, n)
    o = rng.uniform(-reach, reach, (n, 3))
    close = rng.random(n) < 0.6  # through the planes at the same time, or nearly
    t = rng.uniform(0.0, 1.0, n) * reach / np.abs(d).max(1)
    o[close] = (-d.astype(np.float64) * t[:, None])[close] - 0.5
    o = o.astype(np.float32)
    nudge = rng.random((n, 3)) < 0.3
    o[nudge] = np.nextafter(o, np.float32(np.inf) * rng.choice((-1, 1), (n, 3)).astype(np.float32))[nudge]
    on = rng.random((n, 3)) < 0.1
    o[on] = np.round(o[on]) - np.float32(0.5)  # on a plane; some of them at the origin's
    o[rng.random((n, 3)) < 0.05] = -0.5
    o = np.ascontiguousarray(np.clip(o, -reach + 1, reach - 1).astype(np.float32))
    decided = ctypes.c_uint64()
    assert rules.octants_differ(n, o, np.ascontiguousarray(d), ctypes.byref(decided)) == 0
    assert decided.value > 100 * n  # of 256 sets of SubDAGs, most calls


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("height", [1, 2, 6, 11, 20])
def test_descents(rules, seed, height):
    rng = np.random.default_rng(1000 * seed + height)
    n = 4000
    size = 1 << height
    for place in ("origin", "low", "high"):
        low = {"origin": np.zeros(3), "low": np.full(3, -(2 ** 21)), "high": np.full(3, 2 ** 21 - size)}[place]
        low = low.astype(np.int32)
        d = _directions(rng, n)
        o = low + rng.uniform(-0.01, 1.01, (n, 3)) * size - 0.5
        on = rng.random((n, 3)) < 0.4
        o[on] = np.round(o[on] * 2.0) / 2.0  # on voxel faces and centres, and on the box's own
        o = np.clip(o, -(2 ** 21) + 1, 2 ** 21 - 1).astype(np.float32)
        edge = rng.random((n, 3)) < 0.2
        o[edge] = np.nextafter(o, np.float32(np.inf) * rng.choice((-1, 1), (n, 3)).astype(np.float32))[edge]
        assert rules.descents_differ(n, np.ascontiguousarray(o), np.ascontiguousarray(d), low, height) == 0
