"""Encodes and repairs from host memory whose inputs come up in parts: few parts of
columns that do not fill the SMs, as many as there can be of those that do, and
problems that the parts send to the lookup tables."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,S,r", [(128, 2050, 40), (191, 4096, 70), (300, 20480, 30), (700, 1026, 209),
                                   (1487, 716, 60), (200, 51202, 40), (160, 114688, 9), (520, 98306, 17)])
def test_host_parts(k, S, r):
    import par2gpu

    rng = np.random.default_rng(k)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(r, dtype=np.uint32)
    # the oracle on the first and the last columns (it is column by column)
    cols = np.r_[0:min(512, S), max(512, S - 512):S] if S > 1024 else np.arange(S)
    want = oracle.encode(np.ascontiguousarray(src[:, cols]), exps)
    missing = np.sort(rng.choice(k, r, replace=False))
    with par2gpu.Context(0) as ctx:
        rec = ctx.encode_array(src, exps)
        assert np.array_equal(rec[:, cols], want)
        damaged = src.copy()
        damaged[missing] = 0
        got = ctx.repair_array(damaged, missing, exps, rec)
    assert np.array_equal(np.asarray(got), src[missing])
