"""The element-wise kernel at the edges of its 32x32 tiles: block enlargement and operator
merges (masked sums, transposes and diagonals of sub-blocks) for both sides of a lattice, as
part of a renormalisation whose sectors run from 1 to 2, 8, 20, 31-33 and past 64 rows,
against plain torch.

Bound: an element is u^H O u' with unit vectors u, u' of at most D elements and O a sum of at
most 64 terms, so it is at most |O| off by 8 (2 D + 64) 2^-53 |O|.  |O| is under 64 times the
norm of all operators together: no coefficient is over 8 here, no operator in over 8 terms.
"""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("nx, m", [(12, 23), (12, 131), (12, 400), (24, 131)])
def test_enlargement_tile_edges(nx, m, side):
    from perf import cases
    case = dict(call="renormalize", nx=nx, m=m, side=side)
    state = cases.prepare(case, 9)
    try:
        ints, data = cases.run(state)
    finally:
        state["ctx"].close()
    ref_ints, ref = cases.exact(case, 9)
    assert np.array_equal(np.asarray(ints), np.asarray(ref_ints))
    model = state["args"][1]
    norm = np.sqrt(sum(np.vdot(a, a).real for b in [model.ham, *sum(model.ops, [])] for a in b.mats))
    d = max(s[2] for s in cases.enlarged(cases.block_dims(nx, m)))
    ref = ref.cpu().numpy() if hasattr(ref, "cpu") else np.asarray(ref)
    assert np.max(np.abs(data - ref)) <= 8 * (2 * d + 64) * 2.0 ** -53 * 64 * norm
