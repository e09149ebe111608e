"""The test of slice tables for overlap, checked on the host by
tests/cpp/test_overlap.cpp against every pair of ranges."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
BIN = os.path.join(HERE, "cpp", "_build", "test_overlap")


def test_overlap_of_slice_tables():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "cpp")], check=True)
    r = subprocess.run([BIN], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok 160000")
