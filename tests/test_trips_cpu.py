"""The index arithmetic of the grid build's kernels over lists of nearly 2^31 entries, on
the CPU: a trip past the end must not wrap to a negative index."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_trips_cover_the_list_and_end(tmp_path):
    exe = str(tmp_path / "trips_test")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", "trips_test.cpp"), "-o", exe])
    assert subprocess.check_output([exe], timeout=120).decode().strip() == "ok"
