"""Host decisions around CUDA calls: failing ones (a wait, an allocation) and which
kernels get launched, on the host by tests/cpp/test_faults.cpp, which puts its own
functions in the runtime's place: no GPU takes part."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
BIN = os.path.join(HERE, "cpp", "_build", "test_faults")


@pytest.mark.parametrize("case", ["repair_sync", "forms", "tune_fails", "batch_room", "tune_room", "get_plan",
                                  "inverse_routes", "upload_parts"])
def test_failing_call(case):
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "cpp")], check=True)
    r = subprocess.run([BIN, case], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout == "ok\n"
