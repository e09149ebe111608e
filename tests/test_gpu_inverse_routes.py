"""Closed-form inverses on both sides of the sizes at which one CTA makes them: alone,
beside a repair's first pass, and as the only repair of a batch."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def up(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("m", [56, 63, 64, 65, 96])
def test_matrix(ctx, m):
    rng = np.random.default_rng(m)
    k = 3 * m
    missing = np.sort(rng.choice(k, m, replace=False))
    exps = 2 + rng.permutation(m)
    c = oracle.par2_constants(k)[missing]
    want = oracle.invert(np.array([[oracle.gf_pow(int(x), int(e)) for x in c] for e in exps], dtype=np.uint16))
    assert np.array_equal(ctx.reconstruction_matrix(k, missing, exps), want)


@pytest.mark.parametrize("m", [64, 65, 96])
def test_repair_and_lone_job(ctx, m):
    import par2gpu
    import torch

    rng = np.random.default_rng(m)
    k, S = 2 * m + 7, 512
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = rng.permutation(m).astype(np.uint32)
    missing = np.sort(rng.choice(k, m, replace=False))
    present, rec = up(np.delete(src, missing, axis=0)), up(oracle.encode(src, exps))
    out = torch.full((m, S), 0x5A, dtype=torch.uint8, device="cuda")
    ctx.repair(k, S, missing, present, exps, rec, out, device=True)
    assert np.array_equal(out.cpu().numpy(), src[missing])
    out.fill_(0x5A)
    job = {"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S, "src": present, "missing": missing, "exps": exps,
           "recovery": rec, "out": out}
    b = par2gpu.Batch(ctx, [job])
    assert b.run() == [par2gpu.OK]
    assert np.array_equal(out.cpu().numpy(), src[missing])
    b.close()


@pytest.mark.parametrize("m", [3, 100])
def test_lone_singular_job(ctx, m):
    import par2gpu
    import torch

    k, S = 32780, 64
    missing = np.concatenate([[5], np.arange(100, 98 + m), [5 + 32768]])
    d = torch.zeros((1, S), dtype=torch.uint8, device="cuda")
    out = torch.full((m, S), 0x5A, dtype=torch.uint8, device="cuda")
    b = par2gpu.Batch(ctx, [{"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S, "src": [d[0]] * (k - m),
                             "missing": missing, "exps": np.arange(m), "recovery": [d[0]] * m, "out": out}])
    assert b.run() == [par2gpu.ESINGULAR]
    assert bool((out == 0x5A).all())
    b.close()
