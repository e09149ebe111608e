"""Calls whose outputs lie over their inputs on the device: every input is read
before an output is written, whatever plan the shape has.  Slices of thousands of
tiles, so that a launch which zeroed outputs beside the inputs' conversion would
have zeroed some before they were read."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def pin(ctx, k, r, S, plan):
    if plan == "tables split":
        ctx.set_plan(k, r, S, 8, 1, 1, min(4, k))
    elif plan.startswith("tensor"):
        ctx.set_plan(k, r, S, 16, 16, 1, int(plan.split()[1]), 16, tile_symbols=256, inputs_per_stage=256)


@pytest.mark.parametrize("plan", ["own", "tensor 1", "tensor 4", "tensor 60"])
def test_mul_slice(ctx, plan):
    import torch

    n = 2 << 20
    rng = np.random.default_rng(1)
    x = rng.integers(0, 65536, n).astype(np.uint16)
    pin(ctx, 1, 1, 2 * n, plan)
    want = np.zeros((1, n), np.uint16)
    oracle.muladd_region([want[0]], [x], np.array([[0x1234]], np.uint16), 0, n)
    for _ in range(3):
        d = torch.from_numpy(x.view(np.uint8).copy()).cuda()
        ctx_call(ctx, d, n)
        assert np.array_equal(d.cpu().numpy().view(np.uint16), want[0])


def ctx_call(ctx, d, n):
    import par2gpu

    par2gpu.check(par2gpu.lib().p2g_mul_slice(ctx.h, 0x1234, d.data_ptr(), n, par2gpu.DEVICE_PTRS))


# outputs over sources, and straddling two of them
@pytest.mark.parametrize("shift", [0, 4096])
@pytest.mark.parametrize("plan", ["own", "tables split", "tensor 1", "tensor 4"])
@pytest.mark.parametrize("k,r,S", [(20, 2, 1 << 18), (300, 7, 1 << 16), (600, 8, 12 * 1024 + 4)])
def test_encode(ctx, k, r, S, plan, shift):
    import torch

    rng = np.random.default_rng(k + r)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(r, dtype=np.uint32)
    pin(ctx, k, r, S, plan)
    want = oracle.encode(src, exps)
    pitch = (S + 15) // 16 * 16
    at = rng.choice(k - 1, r, replace=False) if shift == 0 else np.arange(r) * 2
    for _ in range(3):
        d = torch.zeros((k, pitch), dtype=torch.uint8, device="cuda")
        d[:, :S] = torch.from_numpy(src)
        base = d.data_ptr()
        outs = [base + int(i) * pitch + shift for i in at]
        ctx.encode([base + i * pitch for i in range(k)], S, exps, outs, device=True)
        flat = d.flatten().cpu().numpy()
        for e, i in enumerate(at):
            lo = int(i) * pitch + shift
            assert np.array_equal(flat[lo:lo + S], want[e]), e


@pytest.mark.parametrize("plan", ["own", "tensor 1", "tensor 4"])
def test_region(ctx, plan):
    """Accumulators that are sources too."""
    import torch

    k, r, n = 64, 8, 40001
    rng = np.random.default_rng(5)
    x = rng.integers(0, 65536, (k, 40008)).astype(np.uint16)
    coeff = rng.integers(0, 65536, (r, k)).astype(np.uint16)
    pin(ctx, k, r, 2 * n, plan)
    want = np.ascontiguousarray(x[3:3 + r, :n])
    oracle.muladd_region(list(want), list(x), coeff, 0, n)
    d = torch.from_numpy(x.view(np.uint8).copy()).cuda()
    ctx.muladd_region([d[3 + o] for o in range(r)], [d[i] for i in range(k)], coeff, 0, n, device=True)
    got = d.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[3:3 + r, :n], want)
    assert np.array_equal(got[3 + r:], x[3 + r:]) and np.array_equal(got[:3], x[:3])
