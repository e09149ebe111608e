"""Who reports a device wait that ran out: the batch whose kernels gave up, and it
alone, while calls and other batches of the same context run beside it; and the
accumulators of the shuffle2x hooks, all of them, until the last is finished."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def timed_out(fn):
    import par2gpu

    with pytest.raises(par2gpu.Par2GpuError) as ei:
        fn()
    assert ei.value.code == par2gpu.ETIMEOUT


@pytest.mark.parametrize("graph", [False, True])
def test_each_batch_reports_its_own(graph):
    import torch

    import par2gpu

    rng = np.random.default_rng(3)
    k, S, r = 32000, 4096, 208  # goes to the tensor cores
    big = torch.randint(0, 256, (k, S), dtype=torch.uint8, device="cuda")
    big_out = torch.zeros((r, S), dtype=torch.uint8, device="cuda")
    job = {"kind": par2gpu.JOB_CREATE, "k": k, "slice_bytes": S, "exps": np.arange(r), "src": big, "out": big_out}
    # a singular repair beside it keeps its own status
    lost = np.array([5, 5 + 32768])
    bad = {"kind": par2gpu.JOB_REPAIR, "k": 32780, "slice_bytes": 64, "missing": lost, "exps": np.arange(2),
           "src": [big[0]] * 32778, "recovery": [big[0], big[1]], "out": [big_out[0], big_out[1]]}
    src = rng.integers(0, 256, (300, S), dtype=np.uint8)
    want = oracle.encode(src, np.arange(20))
    d_src = torch.from_numpy(src).cuda()
    d_out = torch.zeros((20, S), dtype=torch.uint8, device="cuda")
    good = {"kind": par2gpu.JOB_CREATE, "k": 300, "slice_bytes": S, "exps": np.arange(20), "src": d_src, "out": d_out}
    with par2gpu.Context(0) as ctx:
        ctx.set_wait_limit(1)
        x = par2gpu.Batch(ctx, [job, bad], graph=graph)
        ctx.set_wait_limit(0)
        y = par2gpu.Batch(ctx, [good], graph=graph)
        for _ in range(2):
            d_out.zero_()
            torch.cuda.synchronize()
            x.launch()
            y.launch()
            assert np.array_equal(ctx.encode_array(src, np.arange(20)), want)
            assert y.wait() == [par2gpu.OK]
            assert np.array_equal(d_out.cpu().numpy(), want)
            timed_out(x.wait)
            assert x.statuses() == [par2gpu.ETIMEOUT, par2gpu.ESINGULAR]
        # the same batch with the usual limit
        x.close()
        x = par2gpu.Batch(ctx, [job, bad], graph=graph)
        assert x.run() == [par2gpu.OK, par2gpu.ESINGULAR]
        ctx.encode(big, S, np.arange(r), torch.zeros_like(big_out), device=True)
        x.close()
        y.close()


def test_hooks_report_for_every_accumulator():
    import par2gpu

    rng = np.random.default_rng(4)
    nsrc, ndst, n = 16000, 48, 512
    src = rng.integers(0, 65536, (nsrc, n)).astype(np.uint16)
    coeff = rng.integers(1, 65536, (ndst, nsrc)).astype(np.uint16)
    small = rng.integers(0, 256, (64, 1024), dtype=np.uint8)
    want = oracle.encode(small, np.arange(3))
    with par2gpu.Context(0) as ctx:
        ctx.set_plan(nsrc, ndst, 2 * n, 16, 48, 1, 1, 16, tile_symbols=256, inputs_per_stage=256)

        def accumulate(limit):
            dst = np.zeros((ndst, n), np.uint16)
            for b in list(dst) + list(src):
                ctx.prepare_shuffle2x(b)
            ctx.muladd_region_shuffle2x(list(dst), list(src), coeff, 0, n)
            ctx.set_wait_limit(limit)
            return dst

        dst = accumulate(1)
        timed_out(lambda: ctx.finish_shuffle2x(dst[0]))
        ctx.set_wait_limit(0)
        assert np.array_equal(ctx.encode_array(small, np.arange(3)), want)
        for o in range(1, ndst):
            timed_out(lambda: ctx.finish_shuffle2x(dst[o]))
        # a finished accumulator is the caller's again
        ctx.finish_shuffle2x(dst[0])
        dst = accumulate(0)
        for o in range(ndst):
            ctx.finish_shuffle2x(dst[o])
        ref = np.zeros((4, n), np.uint16)
        oracle.muladd_region(list(ref), list(src), coeff[:4], 0, n)
        assert np.array_equal(dst[:4], ref)
