"""The launch that prepares a multiply-accumulate (coefficients, inputs, zeroed
outputs), at the edges of its blocks: 256 records, 8 tiles of planes, 4096
bytes of an output, 32 rows x 128 inputs of the 4-bit coefficients -- over
outputs that hold other bytes before."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def check(ctx, k, r, S):
    import torch

    rng = np.random.default_rng(k * r + S)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = rng.integers(0, 65535, r).astype(np.uint32)
    exps[0] = 0
    pitch = (S + 31) // 16 * 16
    d_src = torch.zeros((k, pitch), dtype=torch.uint8, device="cuda")
    d_src[:, :S] = torch.from_numpy(src)
    d_out = torch.full((r, pitch), 0xA5, dtype=torch.uint8, device="cuda")
    ctx.encode([d_src[i].data_ptr() for i in range(k)], S, exps,
               [d_out[o].data_ptr() for o in range(r)], device=True)
    got = d_out.cpu().numpy()
    assert np.array_equal(got[:, :S], oracle.encode(src, exps))
    assert (got[:, S:] == 0xA5).all()


@pytest.mark.parametrize("k,r,S,splits", [(1, 1, 4, 1), (51, 5, 4100, 3), (64, 4, 4096, 2), (257, 1, 8196, 4),
                                          (33, 8, 2052, 5), (8, 3, 2048, 8), (9, 3, 4092, 1)])
def test_tables(ctx, k, r, S, splits):
    ctx.set_plan(k, r, S, 8, 1, 1, splits)
    check(ctx, k, r, S)


@pytest.mark.parametrize("k,r,S,parts", [(1, 1, 2, 1), (127, 32, 514, 2), (128, 33, 4098, 3), (129, 64, 512, 1),
                                         (193, 209, 6, 1), (65, 417, 262, 4)])
def test_tensor(ctx, k, r, S, parts):
    blocks = -(-r // 208)
    rows = -(-(-(-r // blocks)) // 16) * 16
    ctx.set_plan(k, r, S, 16, rows, blocks, parts, 16, tile_symbols=256, inputs_per_stage=256)
    check(ctx, k, r, S)
