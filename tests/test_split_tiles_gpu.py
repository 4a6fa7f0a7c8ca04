"""The split-precision kernel at the edges of its tiles and accumulator segments:
block-sparse products whose dimensions sit on and beside the 128 x 64 tiles, the
K steps of 16 and the segments of at most 8 of them, against numpy.

Bound, relative to sum |alpha| |L| |X| |R|^T element by element: three BF16 slices
keep an element to 2^-24, the slice products left out weigh 3 * 2^-24, and one
segment adds at most 16 MMAs into an FP32 accumulator, each losing at most 2^-23 of
the sum; with the complex product's two real ones and two products in a row that is
below 4 * (5 * 2^-24 + 17 * 2^-23) = 9.3e-6.
"""
import numpy as np
import pytest

from test_fp64_tiles_gpu import problem, reference
from tsc_tri_t1t2j1j2_b200 import Context
from tsc_tri_t1t2j1j2_b200.blocksparse import random_psi

DIMS = [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 145, 257]


@pytest.mark.gpu
@pytest.mark.parametrize("alphas", [(1.0,), (0.7, -1.3, 2.0, 1e-3, 5.0), (0.3 + 0.4j, -1.0, 1j)],
                         ids=["one", "real", "complex"])
def test_split_tile_edges(alphas):
    import torch
    rng = np.random.default_rng(11)
    P = problem(rng, DIMS, DIMS[::-1], [complex(a) for a in alphas])
    ctx = Context(4, 4)
    try:
        ctx.blocksparse_set([P])
        x = random_psi(rng, [P])
        dx = torch.from_numpy(x).cuda()
        out = torch.full_like(dx, float("nan"))
        torch.cuda.synchronize()
        ctx.blocksparse_apply(dx.data_ptr(), out.data_ptr(), Context.SPLIT_BF16)
        got = out.cpu().numpy()
    finally:
        ctx.close()
    ref, bound = reference(P, x, lambda d, e, t: 1.0, 9.3e-6)
    assert np.all(np.abs(got - ref) <= bound)
