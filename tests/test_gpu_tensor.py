"""The tensor-core multiply-accumulate against the oracle, bit for bit, at the
edges of its tiles: 64 inputs per product and 256 per stage, 16 rows per
accumulator group, 80 rows (two sets of accumulators below, one above), 208
rows per block, 128 symbols per tile and 256 per tile pair, odd last symbols,
and every way the 60 products are dealt out."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import par2gpu

    with par2gpu.Context(0) as c:
        yield c


def pin(ctx, k, r, S, parts=1):
    blocks = -(-r // 208)
    rows = -(-(-(-r // blocks)) // 16) * 16
    ctx.set_plan(k, r, S, 16, rows, blocks, parts, 16, tile_symbols=256, inputs_per_stage=256)


@pytest.mark.parametrize("k", [1, 63, 64, 65, 256, 257, 600])
@pytest.mark.parametrize("r", [1, 16, 17, 80, 81, 208, 209])
def test_inputs_and_outputs(ctx, k, r):
    rng = np.random.default_rng(1000 * k + r)
    S = int(rng.choice([2, 254, 256, 258, 510, 514, 1026]))
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(r, dtype=np.uint32)
    pin(ctx, k, r, S)
    assert np.array_equal(ctx.encode_array(src, exps), oracle.encode(src, exps))


@pytest.mark.parametrize("S", [2, 4, 6, 256, 512, 514, 766, 768, 770, 4098])
@pytest.mark.parametrize("parts", [1, 2, 7, 30, 60])
def test_columns_and_parts(ctx, S, parts):
    k, r = 70, 20
    rng = np.random.default_rng(S + parts)
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = rng.integers(0, 65535, r).astype(np.uint32)
    pin(ctx, k, r, S, parts)
    assert np.array_equal(ctx.encode_array(src, exps), oracle.encode(src, exps))


@pytest.mark.parametrize("parts", [1, 4])
def test_accumulates_and_stays_in_bounds(ctx, parts):
    """The region call adds to what the accumulators hold, and nothing past a
    slice's last (odd) symbol is touched."""
    import torch

    nsrc, ndst, n = 130, 33, 777
    rng = np.random.default_rng(parts)
    pin(ctx, nsrc, ndst, 2 * n, parts)
    src = rng.integers(0, 65536, (nsrc, 784)).astype(np.uint16)
    dst = rng.integers(0, 65536, (ndst, 784)).astype(np.uint16)
    coeff = rng.integers(0, 65536, (ndst, nsrc)).astype(np.uint16)
    d_src = torch.from_numpy(src.view(np.uint8)).cuda()
    d_dst = torch.from_numpy(dst.view(np.uint8)).cuda()
    ctx.muladd_region([d_dst[i] for i in range(ndst)], [d_src[i] for i in range(nsrc)], coeff, 0,
                      n, device=True)
    got = d_dst.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[:, n:], dst[:, n:])
    want = dst[:, :n].copy()
    exp, log = tables()
    for i in range(nsrc):
        row = src[i, :n]
        for o in range(ndst):
            if coeff[o, i]:
                want[o] ^= np.where(row != 0, exp[log[row] + log[coeff[o, i]]], 0).astype(np.uint16)
    assert np.array_equal(got[:, :n], want)


def tables():
    exp = np.zeros(131070, np.uint16)
    log = np.zeros(65536, np.int64)
    b = 1
    for i in range(65535):
        exp[i] = exp[i + 65535] = b
        log[b] = i
        b <<= 1
        if b & 0x10000:
            b ^= 0x1100B
    return exp, log


@pytest.mark.parametrize("k", [300, 1024])
def test_host_groups(ctx, k):
    """Host sources go up and are accumulated in groups of whole 64 inputs."""
    rng = np.random.default_rng(k)
    r, S = 40, 6146
    src = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(r, dtype=np.uint32)
    pin(ctx, k, r, S)
    assert np.array_equal(ctx.encode_array(src, exps), oracle.encode(src, exps))


def test_many_inputs_reset_the_accumulators(ctx):
    """Above 1092 inputs the 60 products' sums need more than the 16 bits kept
    between two settings of the accumulators; all-ones symbols and coefficients
    make the sums as large as they get."""
    k, r, S = 9000, 5, 256
    src = np.full((k, S), 0xFF, np.uint8)
    src[::3] = np.random.default_rng(3).integers(0, 256, src[::3].shape, dtype=np.uint8)
    exps = np.array([0, 1, 2, 65534, 7], np.uint32)
    pin(ctx, k, r, S)
    assert np.array_equal(ctx.encode_array(src, exps), oracle.encode(src, exps))


def test_repair_through_the_tensor_cores(ctx):
    rng = np.random.default_rng(9)
    k, m, S = 700, 90, 1030
    data = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(m, dtype=np.uint32)
    pin(ctx, k, m, S)
    pin(ctx, k - m, m, S)
    pin(ctx, m, m, S)
    rec = ctx.encode_array(data, exps)
    missing = np.sort(rng.choice(k, m, replace=False))
    assert np.array_equal(ctx.repair_array(data, missing, exps, rec), data[missing])


def test_set_plan_rejects_other_tensor_shapes(ctx):
    import par2gpu

    for warps, rows, blocks, parts, wpg, stage in [(8, 208, 1, 1, 16, 256), (16, 192, 1, 1, 16, 256),
                                                   (16, 208, 2, 1, 16, 256), (16, 208, 1, 61, 16, 256),
                                                   (16, 208, 1, 1, 16, 1)]:
        with pytest.raises(par2gpu.Par2GpuError) as ei:
            ctx.set_plan(300, 205, 4096, warps, rows, blocks, parts, wpg, tile_symbols=256,
                         inputs_per_stage=stage)
        assert ei.value.code == par2gpu.EINVAL


def test_batch_problems_on_the_tensor_cores(ctx):
    """A batch whose large problems go to the tensor cores (in parts, with
    odd last symbols, next to problems that stay with the tables and to a
    column range); every job equals the oracle."""
    import par2gpu
    import torch

    rng = np.random.default_rng(77)
    jobs, want, outs, keep = [], [], [], []
    for k, S, r, cols in [(700, 16386, 120, None), (1500, 4098, 209, None), (64, 2050, 30, None),
                          (520, 8192, 90, (2048, 6144)), (5, 4096, 1, None)]:
        src = rng.integers(0, 256, (k, S), dtype=np.uint8)
        exps = np.arange(r, dtype=np.uint32)
        pitch = (S + 15) // 16 * 16
        d = torch.zeros((k, pitch), dtype=torch.uint8, device="cuda")
        d[:, :S] = torch.from_numpy(src).cuda()
        o = torch.full((r, pitch), 7, dtype=torch.uint8, device="cuda")
        job = {"kind": par2gpu.JOB_CREATE, "k": k, "slice_bytes": S,
               "src": [d[i] for i in range(k)], "exps": exps, "out": [o[e] for e in range(r)]}
        full = oracle.encode(src, exps)
        expect = np.full((r, pitch), 7, np.uint8)
        a, b = cols or (0, S)
        expect[:, a:b] = full[:, a:b]
        if cols:
            job["col_begin"], job["col_end"] = cols
        jobs.append(job)
        want.append(expect)
        outs.append(o)
        keep.append(d)
    k, S, m = 900, 8190, 100
    data = rng.integers(0, 256, (k, S), dtype=np.uint8)
    exps = np.arange(m, dtype=np.uint32)
    rec = oracle.encode(data, exps)
    missing = np.sort(rng.choice(k, m, replace=False))
    pitch = (S + 15) // 16 * 16
    d = torch.zeros((k, pitch), dtype=torch.uint8, device="cuda")
    d[:, :S] = torch.from_numpy(data).cuda()
    d_rec = torch.zeros((m, pitch), dtype=torch.uint8, device="cuda")
    d_rec[:, :S] = torch.from_numpy(rec).cuda()
    o = torch.full((m, pitch), 7, dtype=torch.uint8, device="cuda")
    lost = set(missing.tolist())
    jobs.append({"kind": par2gpu.JOB_REPAIR, "k": k, "slice_bytes": S,
                 "src": [d[i] for i in range(k) if i not in lost], "missing": missing, "exps": exps,
                 "recovery": [d_rec[j] for j in range(m)], "out": [o[j] for j in range(m)]})
    expect = np.full((m, pitch), 7, np.uint8)
    expect[:, :S] = data[missing]
    want.append(expect)
    outs.append(o)
    for graph in (False, True):
        for o in outs:
            o.fill_(7)
        torch.cuda.synchronize()
        batch = par2gpu.Batch(ctx, jobs, graph=graph)
        for _ in range(2):
            assert batch.run() == [par2gpu.OK] * len(jobs)
        for j, (o, w) in enumerate(zip(outs, want)):
            assert np.array_equal(o.cpu().numpy(), w), (graph, j)
        batch.close()
