"""The bounded waits of the FP64 kernel's bulk-copy loaders: with a poll limit of 0 every
wait gives up at once, as if its copy had not landed in time.  The kernel has to end, the
call to report it, and the next call to run the whole list again."""
import os
import sys

import numpy as np
import pytest

from tsc_tri_t1t2j1j2_b200 import Context
from tsc_tri_t1t2j1j2_b200._lib import TscError
from tsc_tri_t1t2j1j2_b200.blocksparse import Problem, random_psi

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.gpu
def test_wait_that_runs_out_ends_the_kernel_and_the_list_restarts():
    sl, el, ints, data, off, n = bench.make_superblock()   # lists of 37 and 79 GFLOP
    psi = data[off:off + n]
    ctx = Context(**bench.MODEL)
    try:
        ctx.set_autotune(False)
        ctx.set_superblock_flat(sl, el, ints, data)
        want = ctx.model_wave(psi)
        for _ in range(2):
            ctx.set_bulk_wait_limit(0)
            with pytest.raises(TscError) as ei:
                ctx.model_wave(psi)
            assert ei.value.code == -3 and "bounded wait" in str(ei.value)
            ctx.set_bulk_wait_limit(1 << 20)
            assert np.array_equal(ctx.model_wave(psi), want)
    finally:
        ctx.close()


def big_batch(rng, d=1500):
    """One sector, two terms: 27 GFLOP a product, so both lists are staged by bulk copies."""
    P = Problem(d=[d], e=[d])
    P.left = [(0, [rng.standard_normal((d, d)) + 0j]) for _ in range(2)]
    P.right = [(0, [rng.standard_normal((d, d)) + 0j])]
    P.terms = [(1.0, 0, 0), (0.5, 1, 0)]
    return P


@pytest.mark.gpu
def test_asynchronous_call_is_reported_by_the_next_one_that_waits():
    """blocksparse_apply in FP64 returns before its kernels run, so their wait that ran out
    belongs to it whoever reads the status word: synchronize, or a later call before it runs."""
    import torch
    rng = np.random.default_rng(3)
    P = big_batch(rng)
    ctx = Context(4, 4)
    try:
        ctx.blocksparse_set([P])
        x = torch.from_numpy(random_psi(rng, [P])).cuda()
        out = torch.empty_like(x)
        torch.cuda.synchronize()

        def apply():
            ctx.blocksparse_apply(x.data_ptr(), out.data_ptr(), Context.FP64)

        apply()
        ctx.synchronize()
        want = out.clone()
        torch.cuda.synchronize()
        for waiting in (ctx.synchronize, lambda: ctx.blocksparse_set([P]),
                        lambda: ctx.blocksparse_apply(x.data_ptr(), out.data_ptr(), Context.SPLIT_BF16)):
            ctx.set_bulk_wait_limit(0)
            apply()
            ctx.set_bulk_wait_limit(1 << 20)
            with pytest.raises(TscError) as ei:
                waiting()
            assert ei.value.code == -3 and "earlier call" in str(ei.value) and "FP64" in str(ei.value)
            waiting()   # reported once; the call itself is sound
        apply()
        ctx.synchronize()
        assert torch.equal(out, want)
    finally:
        ctx.close()


@pytest.mark.gpu
def test_replays_of_a_captured_call_are_reported():
    """A caller may capture the asynchronous call in a graph of its own: synchronize reports
    a wait that ran out in a replay, although no call of the context launched it."""
    import torch
    rng = np.random.default_rng(4)
    P = big_batch(rng)
    ctx = Context(4, 4)
    try:
        ctx.blocksparse_set([P])
        x = torch.from_numpy(random_psi(rng, [P])).cuda()
        out = torch.empty_like(x)
        torch.cuda.synchronize()
        ctx.blocksparse_apply(x.data_ptr(), out.data_ptr(), Context.FP64)
        ctx.synchronize()
        want = out.clone()
        graph, good = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
        for g, limit in ((graph, 0), (good, 1 << 20)):
            ctx.set_bulk_wait_limit(limit)
            with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(ctx.stream)):
                ctx.blocksparse_apply(x.data_ptr(), out.data_ptr(), Context.FP64)
        ctx.synchronize()   # nothing has run yet
        graph.replay()
        torch.cuda.synchronize()
        with pytest.raises(TscError):
            ctx.synchronize()
        out.zero_()
        good.replay()
        torch.cuda.synchronize()
        ctx.synchronize()
        assert torch.equal(out, want)
        del graph, good
    finally:
        ctx.close()
