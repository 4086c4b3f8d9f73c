"""Work counters of persistent launches: zero when taken, one ring and one lock per stream."""
import subprocess
from pathlib import Path

TESTS = Path(__file__).resolve().parent


def test_counter_rings(tmp_path):
    exe = tmp_path / "counter_rings"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", str(TESTS / "counter_rings.cpp"), "-o", str(exe)],
                   check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout == "ok\n", run.stdout + run.stderr
