"""Decode matrices at the sizes where their kernels change: one warp of rows,
the one-launch inverse (up to 128 rows), full and short segments of the
quotients' recurrence (16 per polynomial), a warp per coefficient, the small
elimination's table copy (above 16 rows) and the direct correction (up to 8
exponents outside the window)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def check(ctx, m, exps):
    rng = np.random.default_rng(m + len(exps))
    k = 3 * m + 5
    missing = np.sort(rng.choice(k, m, replace=False))
    c = oracle.par2_constants(k)[missing]
    want = oracle.invert(np.array([[oracle.gf_pow(int(x), int(e)) for x in c] for e in exps], dtype=np.uint16))
    assert want is not None
    assert np.array_equal(ctx.reconstruction_matrix(k, missing, exps), want)


@pytest.mark.parametrize("first", [0, 5])
@pytest.mark.parametrize("m", [1, 3, 31, 32, 33, 127, 128, 129, 144, 145, 160, 161, 162, 257])
def test_consecutive_exponents(ctx, m, first):
    check(ctx, m, np.arange(first, first + m))


@pytest.mark.parametrize("m", [2, 15, 16, 17])
def test_small_eliminations(ctx, m):
    check(ctx, m, np.concatenate([np.arange(m - 1), [1000]]))


@pytest.mark.parametrize("m", [97, 129, 150])
@pytest.mark.parametrize("g", [1, 7, 8, 9, 16, 17])
def test_replaced_rows(ctx, m, g):
    lost = 1 + 3 * np.arange(g)
    check(ctx, m, np.concatenate([np.setdiff1d(np.arange(m), lost), 40000 + 7 * np.arange(g)]))


@pytest.mark.parametrize("m", [128, 129, 300])
def test_repeated_constant_is_singular(ctx, m):
    import par2gpu

    missing = np.concatenate([[5], np.arange(100, 98 + m), [5 + 32768]])
    with pytest.raises(par2gpu.Par2GpuError) as ei:
        ctx.reconstruction_matrix(40000, missing, np.arange(m))
    assert ei.value.code == par2gpu.ESINGULAR


def test_inverses_of_a_batch(ctx):
    """Repairs whose inverses share a launch (up to 128 consecutive exponents),
    among larger and gapped ones and an unrepairable one."""
    import par2gpu
    import torch

    rng = np.random.default_rng(9)
    S, jobs, want = 64, [], []
    for m, first, gap in [(1, 0, 0), (31, 3, 0), (32, 0, 0), (33, 7, 0), (40, 0, 1), (128, 0, 0), (129, 1, 0)]:
        k = m + 9
        src = rng.integers(0, 256, (k, S), dtype=np.uint8)
        exps = first + np.arange(m) + (np.arange(m) >= m // 2) * gap
        rng.shuffle(exps)
        missing = np.sort(rng.choice(k, m, replace=False))
        d = torch.from_numpy(np.delete(src, missing, axis=0)).cuda()
        rec = torch.from_numpy(oracle.encode(src, exps.astype(np.uint32))).cuda()
        out = torch.full((m, S), 0x5A, dtype=torch.uint8, device="cuda")
        jobs.append({"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S, "src": list(d), "missing": missing,
                     "exps": exps, "recovery": list(rec), "out": list(out)})
        want.append((out, src[missing], d, rec))
    k = 32780
    d = torch.zeros((1, S), dtype=torch.uint8, device="cuda")
    out = torch.full((2, S), 0x5A, dtype=torch.uint8, device="cuda")
    jobs.insert(3, {"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S, "src": [d[0]] * (k - 2),
                    "missing": np.array([5, 5 + 32768]), "exps": np.arange(2), "recovery": [d[0], d[0]],
                    "out": list(out)})
    b = par2gpu.Batch(ctx, jobs)
    st = b.run()
    assert [s != 0 for s in st] == [j == 3 for j in range(len(jobs))], st
    assert st[3] == par2gpu.ESINGULAR
    assert bool((out == 0x5A).all())
    for o, w, _, _ in want:
        assert np.array_equal(o.cpu().numpy(), w)
    b.close()
