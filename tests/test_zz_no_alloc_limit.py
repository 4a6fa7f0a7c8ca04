"""The fixed scratch of tsc_hpsi_noalloc: the last superblocks that fit with the basic
schedule (4 waves of 888 CTAs with 32x32 tiles; sizes measured in steps of 3) are taken,
whatever schedule their lists are cut for, and the first that do not fit are refused.
The answer is tsc_hpsi_device's, from the same lists: equal."""
import pytest

from tsc_tri_t1t2j1j2_b200._lib import TscError

TSC_E_LIMIT = -6


@pytest.mark.gpu
@pytest.mark.parametrize("precision, nx, last, first", [("fp64", 12, 303, 306), ("fp64", 24, 285, 288),
                                                        ("split", 12, 306, 309), ("split", 24, 303, 306)])
def test_limit(precision, nx, last, first):
    import torch
    from perf import cases
    for m in (last, first):
        st = cases.prepare(dict(call="hpsi", precision=precision, nx=nx, m=m), 3)
        ctx, x = st["ctx"], st["psi"]
        try:
            want = cases.run(st)
            out = torch.full_like(x, float("nan"))
            torch.cuda.synchronize()
            if m == last:
                ctx.hpsi_noalloc(x.data_ptr(), out.data_ptr())
                torch.cuda.synchronize()
                assert torch.equal(out, want)
            else:
                with pytest.raises(TscError) as e:
                    ctx.hpsi_noalloc(x.data_ptr(), out.data_ptr())
                assert e.value.code == TSC_E_LIMIT
        finally:
            ctx.close()
