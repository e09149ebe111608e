"""The 60-product form of GF(2^16) multiplication behind the tensor-core kernel,
checked on the host by tests/cpp/test_bilinear.cpp: every pair of basis
elements and 20000 random pairs against shift-and-add multiplication."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
BIN = os.path.join(HERE, "cpp", "_build", "test_bilinear")


def test_products_reproduce_gf_multiplication():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "cpp")], check=True)
    r = subprocess.run([BIN], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok 20256")
