"""Which host buffers kernels may read and write: those that lie in one CUDA
allocation or registration from their first byte to their last (cbq_hostmem.hpp).
A buffer that only starts in page-locked memory is left to the copy calls."""
import shutil
import subprocess
from pathlib import Path

import pytest

TESTS = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path_factory.mktemp("ranges") / "host_ranges"
    subprocess.run([nvcc, "-std=c++17", str(TESTS / "host_ranges.cpp"), "-o", str(exe)], check=True)
    return exe


def _lines(*command):
    text = subprocess.run([str(c) for c in command], check=True, capture_output=True, text=True, timeout=120).stdout
    return {name: tuple(int(v) for v in rest) for name, *rest in (line.split() for line in text.splitlines())}


def test_range_rule(program):
    assert _lines(program) == {"all": (1,), "inside": (1,), "one_past": (0,), "longer": (0,), "before": (0,),
                               "last_byte": (1,), "at_end": (0,), "empty_range": (0,), "huge": (0,), "wraps": (0,)}


@pytest.mark.gpu
def test_classification(program):
    """(whole, usable by kernels, the same from a fresh thread)"""
    yes, no = (1, 1, 1), (0, 0, 1)
    assert _lines(program, "device") == {
        "registered": yes, "registered_part": yes, "registered_end": yes, "over_the_end_of_it": no,
        "all_but_its_first": yes, "before_it": no, "two_registrations": no, "starts_pageable": no,
        "ends_pageable": no, "hole_between": no, "pageable": no, "locked": yes, "locked_tail": yes,
        "past_locked": no, "managed": yes, "past_managed": no, "device_memory": (1, 0, 1)}
