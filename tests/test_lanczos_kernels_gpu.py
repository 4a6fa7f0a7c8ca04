"""The Lanczos vector kernels where their split of a vector changes: vectors below
one block of 256, of a few blocks, on both sides of one block of each of the 592
(151,552 elements) and of one 1024-element piece of each (606,208), against the same
recurrence in numpy on the engine's own H.psi (eigen.f90:4-199, Gram-Schmidt of
block.f90:1251-1289).

Bound: every scalar of an iteration is a sum of n products, within 64 units of
2^-53 for the tree sums used, and a Ritz value moves by at most the sum of the
errors of its l <= 100 iterations times the operator's norm, here the lowest
eigenvalue's magnitude up to a small factor: 100 * 64 * 2^-53 = 7e-13, and 1e-11
with that factor.  The returned vector is normalised to 1e-12; it differs from the
recurrence's by at most that error over the relative gap above the lowest Ritz value,
1e-8 for a gap of 1e-3, so their overlap is 1 to the square of it, within 1e-12.
(The couplings are random, so H is not exactly Hermitian and the energy of the
vector is not its Ritz value.)
"""
import numpy as np
import pytest


def numpy_lanczos(h, x, lanzero):
    basis = [x / np.linalg.norm(x)]
    w = h(basis[0])
    alpha, beta = [np.vdot(basis[0], w).real], []
    ritz = alpha[0]
    for it in range(2, 101):
        w = w - alpha[-1] * basis[-1] - (beta[-1] * basis[-2] if beta else 0.0)
        beta.append(np.linalg.norm(w))
        w = w / beta[-1]
        w = w - sum(np.vdot(v, w).real * v for v in basis)
        basis.append(w / np.linalg.norm(w))
        w = h(basis[-1])
        alpha.append(np.vdot(basis[-1], w).real)
        low = np.linalg.eigvalsh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))[0]
        if abs(low - ritz) <= lanzero:
            z = np.linalg.eigh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))[1][:, 0]
            x = sum(c * v for c, v in zip(z, basis))
            return low, it, x / np.linalg.norm(x)
        ritz = low
    raise AssertionError("not converged")


@pytest.mark.gpu
@pytest.mark.parametrize("m, lo, hi", [(8, 1, 256), (40, 1280, 1536), (420, 140000, 151552), (440, 151553, 170000),
                                       (845, 560000, 606208), (870, 606209, 660000)])
def test_vector_sizes(m, lo, hi):
    from perf import cases
    st = cases.prepare(dict(call="lanczos", nx=12, m=m, lanzero=1e-3), 5)
    ctx, psi = st["ctx"], st["psi"]
    try:
        assert lo <= psi.size <= hi
        ref, iters, y = numpy_lanczos(ctx.model_wave, psi, 1e-3)
        for graph in (True, False):
            ctx.set_lanczos_graph(graph)
            x, e0, it = ctx.lanczos_memo_new(psi, 1e-3)
            assert it == iters
            assert abs(e0 - ref) <= 1e-11 * abs(ref)
            assert abs(np.linalg.norm(x) - 1.0) <= 1e-12
            assert 1.0 - abs(np.vdot(x, y)) <= 1e-12
    finally:
        ctx.close()
