"""The tensor-core multiply-accumulate at the ends of its range: as many inputs as calls
take, with sums as large as they get, and problems whose symbol forms exceed the 12
GiB that a call holds of them and run in column chunks (one input's forms are 480
times its slice, so that a few inputs of 28 MiB do)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def pin(ctx, k, r, S, parts=1):
    ctx.set_plan(k, r, S, 16, -(-r // 16) * 16, 1, parts, 16, tile_symbols=256, inputs_per_stage=256)


@pytest.fixture()
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


# two sets of accumulators up to 80 outputs, one above
@pytest.mark.parametrize("ndst", [17, 96])
@pytest.mark.parametrize("nsrc", [21845, 32768, 32769, 43691, 65534, 65535])
def test_sums_of_all_inputs(ctx, nsrc, ndst):
    """Every input alike, so that a product's sum is 0 or the number of inputs; and the
    last third of them random."""
    n = 300
    rng = np.random.default_rng(nsrc + ndst)
    row = rng.integers(0, 65536, n).astype(np.uint16)
    row[:4] = [0xFFFF, 0, 1, 0x8000]
    col = rng.integers(0, 65536, ndst).astype(np.uint16)
    col[:4] = [0xFFFF, 0x8000, 1, 0]
    src = np.broadcast_to(row, (nsrc, n)).copy()
    coeff = np.broadcast_to(col[:, None], (ndst, nsrc)).copy()
    pin(ctx, nsrc, ndst, 2 * n)
    for mixed in (False, True):
        if mixed:
            src[-(nsrc // 3):] = rng.integers(0, 65536, (nsrc // 3, n))
            coeff[:, -(nsrc // 3):] = rng.integers(0, 65536, (ndst, nsrc // 3))
        got = np.zeros((ndst, n), np.uint16)
        ctx.muladd_region(list(got), list(src), coeff, 0, n)
        keep = [0, 1, 2, 3, 5, ndst - 1]
        want = np.zeros((len(keep), n), np.uint16)
        oracle.muladd_region(list(want), list(src), coeff[keep], 0, n)
        assert np.array_equal(got[keep], want), mixed


# two and three chunks; a last one with an odd number of tiles and an odd symbol
@pytest.mark.parametrize("S", [(28 << 20) + 2, (56 << 20) + 254])
@pytest.mark.parametrize("parts", [1, 4])
def test_column_chunks(ctx, S, parts):
    import torch

    k, r = 3, 2
    rng = np.random.default_rng(S)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.array([1, 5], np.uint32)
    pin(ctx, k, r, S, parts)
    pitch = (S + 31) // 16 * 16
    d_src = torch.zeros((k, pitch), dtype=torch.uint8, device="cuda")
    d_src[:, :S] = torch.from_numpy(src)
    d_out = torch.full((r, pitch), 0xA5, dtype=torch.uint8, device="cuda")
    ctx.encode(d_src, S, exps, d_out, device=True)
    want = torch.from_numpy(oracle.encode(src, exps)).cuda()
    assert torch.equal(d_out[:, :S], want)
    assert bool((d_out[:, S:] == 0xA5).all())
    # added to what is there: the same products again leave the accumulators empty
    c = oracle.power_matrix(oracle.par2_constants(k), exps)
    ctx.muladd_region(d_out, d_src, c, 0, S // 2, device=True)
    assert not bool(d_out[:, :S].any())
    assert bool((d_out[:, S:] == 0xA5).all())


@pytest.mark.parametrize("parts", [1, 4])
def test_repair_in_column_chunks(ctx, parts):
    import torch

    import par2gpu

    k, m, S = 4, 2, (28 << 20) + 2
    rng = np.random.default_rng(parts)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    pin(ctx, m, m, S, parts)  # both passes: two present, two missing
    pitch = (S + 15) // 16 * 16

    def up(a):
        t = torch.zeros((len(a), pitch), dtype=torch.uint8, device="cuda")
        t[:, :S] = torch.from_numpy(np.ascontiguousarray(a))
        return t

    present, out = up(src[[1, 3]]), torch.full((m, pitch), 0x5A, dtype=torch.uint8, device="cuda")
    exps = np.array([2, 3], np.uint32)
    rec = up(oracle.encode(src, exps))
    # the same exponent twice: nothing is written
    with pytest.raises(par2gpu.Par2GpuError) as ei:
        ctx.repair(k, S, [0, 2], present, [2, 2], rec, out, device=True)
    assert ei.value.code == par2gpu.ESINGULAR
    assert bool((out == 0x5A).all())
    ctx.repair(k, S, [0, 2], present, exps, rec, out, device=True)
    assert torch.equal(out[:, :S], torch.from_numpy(src[[0, 2]]).cuda())
