"""What serving reserves for a job covers what the library takes for it in a batch, for
jobs on the lookup tables and on the tensor cores (whose symbol forms are 1.9 times
the slices, padded to whole stages of 256 inputs).  The library's own allocations,
on the host (tests/cpp/test_faults.cpp)."""
import os
import subprocess

import numpy as np
import pytest

from par2gpu.serve import ServedJob

HERE = os.path.dirname(os.path.abspath(__file__))
BIN = os.path.join(HERE, "cpp", "_build", "test_faults")


@pytest.mark.parametrize("kind", ["create", "repair"])
@pytest.mark.parametrize("k,n,S", [(20, 2, 4096), (100, 30, 65536), (100, 90, 65536), (257, 50, 65536),
                                   (300, 200, 16386), (2048, 205, 65536), (4000, 9, 65536), (4000, 2, 65536),
                                   (270, 15, 1 << 20), (600, 300, 65536)])
def test_reservation_covers_the_batch(kind, k, n, S):
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "cpp")], check=True)
    r = subprocess.run([BIN, "job_bytes", kind, str(k), str(n), str(S)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    took = int(r.stdout.split()[0])
    src = np.lib.stride_tricks.as_strided(np.zeros(1, np.uint8), (k, S), (0, 0))
    job = ServedJob(0, kind, src, r=n, missing=np.arange(n) if kind == "repair" else None)
    # apart from the outputs, which are the caller's
    reserved = job.scratch_bytes() - n * S
    # what else a batch allocates: tables of pointers and work items, a decode matrix
    small = 8 * (2 * k + 6 * n) + 8 * (k + n) + 2 * n * n + 64 * (S // 512 + 1) * (n // 208 + 1) * 60 + (1 << 16)
    assert took <= reserved + small, (took, reserved)
