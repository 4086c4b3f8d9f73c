"""The copies of a cbq_intersect_host call: every byte of a host array once, to its
chunk's place on the device, and no pitched copy beyond CUDA's largest pitch."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

TESTS = Path(__file__).resolve().parent
MAX_PITCH = 2 ** 31 - 1


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("copies") / "host_copies"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", str(TESTS / "host_copies.cpp"), "-o", str(exe)], check=True)
    return exe


def _copies(program, n, overlaps, bytes_per_ray, max_pitch=MAX_PITCH):
    text = subprocess.run([str(program), str(n), str(int(overlaps)), str(bytes_per_ray), str(max_pitch)], check=True,
                          capture_output=True, text=True).stdout
    return [tuple(int(v) for v in line.split()) for line in text.splitlines()]


@pytest.mark.parametrize("n", [1, 31, 196607, 196608, 393215, 393216, 655360, 655363, 1 << 20])
@pytest.mark.parametrize("overlaps", [False, True])
@pytest.mark.parametrize("bytes_per_ray", [1, 12])
@pytest.mark.parametrize("max_pitch", [MAX_PITCH, 1000])
def test_every_byte_once(program, n, overlaps, bytes_per_ray, max_pitch):
    host, dev = np.zeros(n * bytes_per_ray, np.uint8), np.zeros(n * bytes_per_ray, np.uint8)
    for _, h, d, width, pitch, rows in _copies(program, n, overlaps, bytes_per_ray, max_pitch):
        assert rows == 1 or width <= pitch <= max_pitch
        for r in range(rows):
            host[h + r * pitch:h + r * pitch + width] += 1
            dev[d + r * width:d + (r + 1) * width] += 1
    assert (host == 1).all() and (dev == 1).all()


@pytest.mark.parametrize("n", [(1 << 27) - 1, 1 << 27, (1 << 29) - 4, 1 << 29, (1 << 30) + 5, (1 << 32) + 77])
@pytest.mark.parametrize("overlaps", [False, True])
def test_largest_pitch(program, n, overlaps):
    for bytes_per_ray in (1, 4, 12, 16):
        copies = _copies(program, n, overlaps, bytes_per_ray)
        assert sum(width * rows for _, _, _, width, _, rows in copies) == n * bytes_per_ray
        assert all(rows == 1 or pitch <= MAX_PITCH for *_, pitch, rows in copies)
        if not overlaps:  # all rays in one plain copy
            assert [c[1:4] + c[5:] for c in copies] == [(0, 0, n * bytes_per_ray, 1)]
