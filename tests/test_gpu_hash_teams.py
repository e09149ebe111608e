"""Checksums over every number of teams (32 slices each) that an SM's block can
hold, one to eight, with whole and ragged chunks of 128 bytes, and groups of
several sizes in a batch."""
import hashlib
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def expect(a):
    return (np.array([list(hashlib.md5(r.tobytes()).digest()) for r in a], np.uint8),
            np.array([zlib.crc32(r.tobytes()) for r in a], np.uint32))


@pytest.mark.parametrize("n,S", [(1, 128), (32, 130), (33, 64), (4736, 2), (4737, 320), (9473, 126),
                                 (18945, 256), (37889, 192)])
def test_teams(ctx, n, S):
    import torch

    a = np.random.default_rng(n).integers(0, 256, (n, S), dtype=np.uint8)
    d = torch.zeros((n, (S + 15) // 16 * 16), dtype=torch.uint8, device="cuda")
    d[:, :S] = torch.from_numpy(a)
    ptrs = d.data_ptr() + np.arange(n, dtype=np.uint64) * np.uint64(d.shape[1])
    md5, crc = ctx.hash_slices(ptrs, S, device=True)
    want_md5, want_crc = expect(a)
    assert np.array_equal(md5, want_md5)
    assert np.array_equal(crc, want_crc)


def test_groups_in_a_batch(ctx):
    import torch

    import par2gpu

    rng = np.random.default_rng(5)
    sets, jobs = [], []
    for n, S in [(1, 2), (33, 130), (70, 64), (5, 1000), (64, 128), (96, 4096), (31, 318)]:
        a = rng.integers(0, 256, (n, S), dtype=np.uint8)
        d = torch.zeros((n, (S + 15) // 16 * 16), dtype=torch.uint8, device="cuda")
        d[:, :S] = torch.from_numpy(a)
        sets.append((a, d))
        jobs.append({"kind": par2gpu.JOB_VERIFY, "k": n, "slice_bytes": S, "src": [d[i] for i in range(n)]})
    b = par2gpu.Batch(ctx, jobs)
    for _ in range(2):
        assert all(s == 0 for s in b.run())
        for (a, _), res in zip(sets, b.results):
            want_md5, want_crc = expect(a)
            assert np.array_equal(res["md5"], want_md5)
            assert np.array_equal(res["crc"], want_crc)
    b.close()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 1000])
def test_verdicts(ctx, n):
    """One wrong bit of an expected checksum is one damaged slice."""
    S = 70
    rng = np.random.default_rng(n)
    a = rng.integers(0, 256, (n, S), dtype=np.uint8)
    md5, crc = expect(a)
    bad = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 5)]))
    for t, i in enumerate(bad):
        if t % 2:
            crc[i] ^= np.uint32(1 << int(rng.integers(0, 32)))
        else:
            md5[i, rng.integers(0, 16)] ^= np.uint8(1 << int(rng.integers(0, 8)))
    got = ctx.verify_slices([a[i] for i in range(n)], S, md5, crc)
    assert np.array_equal(np.flatnonzero(~got), bad)
