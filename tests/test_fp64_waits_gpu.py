"""The bounded waits of the FP64 kernel's bulk-copy loaders: with a poll limit of 0 every
wait gives up at once, as if its copy had not landed in time.  The kernel has to end, the
call to report it, and the next call to run the whole list again."""
import os
import sys

import numpy as np
import pytest

from tsc_tri_t1t2j1j2_b200 import Context
from tsc_tri_t1t2j1j2_b200._lib import TscError

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
