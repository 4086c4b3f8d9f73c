"""A DAG for whose walk there is no memory: the node store alone, with a warning."""
import subprocess
from pathlib import Path

TESTS = Path(__file__).resolve().parent
CSRC = TESTS.parent / "cubiquity_gb300" / "csrc"


def test_store_memory(tmp_path):
    exe = tmp_path / "store_memory"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", str(TESTS / "store_memory.cpp"),
                    str(CSRC / "cbq_host.cpp"), str(CSRC / "cbq_builder.cpp"), "-o", str(exe)], check=True)
    text = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    # memory, wanted, allocated?, bytes, all of it, warnings
    assert [tuple(map(int, line.split())) for line in text.splitlines()] == [
        (3000, 3000, 1, 3000, 1, 0), (3000, 1000, 1, 1000, 1, 0),
        (2999, 3000, 1, 1000, 0, 1), (2999, 1000, 1, 1000, 1, 0),
        (1000, 3000, 1, 1000, 0, 1), (1000, 1000, 1, 1000, 1, 0),
        (999, 3000, 0, 0, 0, 0), (999, 1000, 0, 0, 0, 0)]
