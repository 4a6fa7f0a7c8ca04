"""Rounding of the FP64 H.psi where the products of two block operators are its largest
terms and of one size: normal random values on the YC4x24 m=4000 superblock, whose lists
hold the longest sums.  The first kernels' largest element error against the oracle is
1.2e-14 of the largest element; the oracle's own adds 0.2e-14.  Summing the couplings
between the blocks last built first gave 2.5e-14."""
import os
import sys

import numpy as np
import pytest

from tsc_tri_t1t2j1j2_b200 import Context

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.gpu
def test_equal_terms_at_m4000():
    sb = bench.make_superblock(fixture=bench.FIXTURE3)
    sl, el, ints, data, off, n = sb
    ctx = Context(**bench.MODEL3)
    try:
        ctx.set_autotune(False)
        ctx.set_superblock_flat(sl, el, ints, data)
        got = ctx.model_wave(data[off:off + n])
    finally:
        ctx.close()
    ref, *_ = bench.cpu_hpsi(sb, 1, bench.MODEL3)
    assert np.max(np.abs(got - ref)) <= 1.4e-14 * np.max(np.abs(ref))
