"""Batches that verify what their other jobs write: the checksums are those of the
rebuilt and created slices, also where a verification has slices that nothing
writes beside them."""
import hashlib
import zlib

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def sums(rows):
    return (np.stack([np.frombuffer(hashlib.md5(r.tobytes()).digest(), np.uint8) for r in rows]),
            np.array([zlib.crc32(r.tobytes()) for r in rows], np.uint32))


@pytest.mark.parametrize("k,S,m", [(40, 4096, 5), (300, 1 << 16, 30), (700, 8194, 120)])
@pytest.mark.parametrize("graph", [False, True])
def test_verify_what_the_batch_writes(k, S, m, graph):
    import torch

    import par2gpu

    rng = np.random.default_rng(k)
    data = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(m, dtype=np.uint32)
    rec = oracle.encode(data, exps)
    missing = np.sort(rng.choice(k, m, replace=False))
    pitch = (S + 15) // 16 * 16

    def up(a):
        t = torch.zeros((len(a), pitch), dtype=torch.uint8, device="cuda")
        t[:, :S] = torch.from_numpy(a)
        return t

    d, d_rec = up(data), up(rec)
    fresh = torch.zeros((m, pitch), dtype=torch.uint8, device="cuda")
    lost = torch.from_numpy(missing)
    other = rng.integers(0, 256, (33, S), dtype=np.uint8)
    d_other = up(other)
    gone = set(missing.tolist())
    with par2gpu.Context(0) as ctx:
        jobs = [
            # the whole set, its missing slices rebuilt in place by the next job
            {"kind": par2gpu.JOB_VERIFY, "k": k, "slice_bytes": S, "src": [d[i] for i in range(k)]},
            {"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S, "missing": missing, "exps": exps,
             "src": [d[i] for i in range(k) if i not in gone], "recovery": [d_rec[j] for j in range(m)],
             "out": [d[int(i)] for i in missing]},
            {"kind": par2gpu.JOB_CREATE, "k": k - m, "slice_bytes": S, "exps": exps,
             "src": [d[i] for i in range(k) if i not in gone], "out": [fresh[j] for j in range(m)]},
            {"kind": par2gpu.JOB_VERIFY, "k": m, "slice_bytes": S, "src": [fresh[j] for j in range(m)]},
            {"kind": par2gpu.JOB_VERIFY, "k": 33, "slice_bytes": S, "src": [d_other[j] for j in range(33)]},
        ]
        batch = par2gpu.Batch(ctx, jobs, graph=graph)
        created = oracle.encode(np.delete(data, missing, axis=0), exps)
        for _ in range(2):
            d[lost] = 0x5A
            fresh.zero_()
            torch.cuda.synchronize()
            assert batch.run() == [par2gpu.OK] * len(jobs)
            for j, rows in ((0, data), (3, created), (4, other)):
                md5, crc = sums(rows)
                assert np.array_equal(batch.results[j]["md5"], md5), j
                assert np.array_equal(batch.results[j]["crc"], crc), j
        batch.close()
