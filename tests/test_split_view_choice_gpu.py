"""tsc_set_split_view_sharing(-1): one coefficient-folded view per term unless those would
pass 4 GiB, then one view per operator block."""
import os
import sys

import pytest

from tsc_tri_t1t2j1j2_b200 import Context

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1, 2])   # folded views of 1.4 and 5.1 GiB
def test_automatic_sharing_keeps_folded_views_under_4_gib(scale):
    sl, el, ints, data, off, _ = bench.make_superblock(scale=scale)
    got = {}
    for shared in (True, None):
        ctx = Context(**bench.MODEL)
        try:
            ctx.set_precision(Context.SPLIT_BF16)
            ctx.set_split_view_sharing(shared)
            ctx.set_superblock_flat(sl, el, ints, data)
            got[shared] = ctx.split_views()["operators"][0]
        finally:
            ctx.close()
    if scale == 1:
        assert 3 * got[True] < got[None] <= 4 << 30
    else:
        assert got[None] == got[True]
