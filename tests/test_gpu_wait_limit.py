"""Waits inside the tensor-core kernel that run out: the kernel ends, the call
reports P2G_ETIMEOUT, and the context goes on working.  The limit is set to one
failing try, so that every role of a CTA gives up, at whichever of its waits is the
first not to be over at once."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def pin(ctx, k, r, S, parts):
    blocks = -(-r // 208)
    rows = -(-(-(-r // blocks)) // 16) * 16
    ctx.set_plan(k, r, S, 16, rows, blocks, parts, 16, tile_symbols=256, inputs_per_stage=256)


# one and two tiles in a CTA, one and two warpgroups reading a tile's results, one
# and two sets of accumulators, all products in a CTA and one; as many inputs as
# keep a product busy for longer than a try may suspend its thread
@pytest.mark.parametrize("S", [256, 512, 4096])
@pytest.mark.parametrize("r,parts", [(16, 1), (48, 1), (48, 60), (208, 1), (208, 4)])
def test_call_ends_and_reports(S, r, parts):
    import torch

    import par2gpu

    k = 32000
    rng = np.random.default_rng(S + r + parts)
    src = torch.randint(0, 256, (k, S), dtype=torch.uint8, device="cuda")
    out = torch.zeros((r, S), dtype=torch.uint8, device="cuda")
    exps = np.arange(r, dtype=np.uint32)
    small = rng.integers(0, 256, (70, S), dtype=np.uint8)
    with par2gpu.Context(0) as ctx:
        pin(ctx, k, r, S, parts)
        pin(ctx, 70, r, S, parts)
        for _ in range(2):
            ctx.set_wait_limit(1)
            with pytest.raises(par2gpu.Par2GpuError) as ei:
                ctx.encode(src, S, exps, out, device=True)
            assert ei.value.code == par2gpu.ETIMEOUT
            # reported once; calls with the usual limit are not affected
            ctx.set_wait_limit(0)
            assert np.array_equal(ctx.encode_array(small, exps), oracle.encode(small, exps))
