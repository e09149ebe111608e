"""Repairs of slices on the device, whose passes are queued before the
inversion's outcome is known up to 96 rows: results on both sides of that size,
and a singular matrix leaving the outputs alone with every kind of plan for the
last pass."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def pointers(t):
    return [t[i].data_ptr() for i in range(t.shape[0])]


def setup(k, S, missing, exps):
    import torch

    rng = np.random.default_rng(k + S)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    rec = oracle.encode(src, exps)
    pitch = (S + 15) // 16 * 16

    def up(a):
        t = torch.zeros((len(a), pitch), dtype=torch.uint8, device="cuda")
        t[:, :S] = torch.from_numpy(np.ascontiguousarray(a))
        return t

    out = torch.full((len(missing), pitch), 0x5A, dtype=torch.uint8, device="cuda")
    return src, up(np.delete(src, missing, axis=0)), up(rec), out


def pin(ctx, m, S, plan):
    if plan == "split":
        ctx.set_plan(m, m, S, 8, -(-m // 8) if m <= 24 else 13, 1, min(m, 3))
    elif plan == "tensor":
        ctx.set_plan(m, m, S, 16, -(-m // 16) * 16, 1, 1, 16, tile_symbols=256, inputs_per_stage=256)
    elif plan == "tensor split":
        ctx.set_plan(m, m, S, 16, -(-m // 16) * 16, 1, 4, 16, tile_symbols=256, inputs_per_stage=256)


@pytest.mark.parametrize("plan", ["own", "split", "tensor", "tensor split"])
@pytest.mark.parametrize("m,gap", [(1, 0), (13, 0), (13, 1), (96, 1), (97, 0), (97, 1)])
def test_repair(ctx, m, gap, plan):
    k, S = 120, 4096 + 4 * m
    missing = np.sort(np.random.default_rng(m).choice(k, m, replace=False))
    exps = np.arange(m) + (np.arange(m) >= m // 2) * gap
    src, present, rec, out = setup(k, S, missing, exps)
    pin(ctx, m, S, plan)
    ctx.repair(k, S, missing, pointers(present), exps, pointers(rec), pointers(out), device=True)
    assert np.array_equal(out.cpu().numpy()[:, :S], src[missing])


@pytest.mark.parametrize("plan", ["own", "split", "tensor", "tensor split"])
@pytest.mark.parametrize("m,gap", [(3, 0), (3, 1), (100, 0)])
def test_singular_leaves_the_outputs(ctx, m, gap, plan):
    """c_i = c_{i + 32768}: losing both slices of such a pair is unrepairable."""
    import par2gpu

    k, S = 32780, 64
    missing = np.concatenate([[5], np.arange(100, 98 + m), [5 + 32768]])
    exps = np.arange(m) + (np.arange(m) == m - 1) * gap
    src, present, rec, out = setup(k, S, missing, exps)
    pin(ctx, m, S, plan)
    with pytest.raises(par2gpu.Par2GpuError) as ei:
        ctx.repair(k, S, missing, pointers(present), exps, pointers(rec), pointers(out), device=True)
    assert ei.value.code == par2gpu.ESINGULAR
    assert bool((out == 0x5A).all())
