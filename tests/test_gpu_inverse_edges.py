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
