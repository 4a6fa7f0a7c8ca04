"""The FP64 grouped kernel at the edges of its tiles: block-sparse products whose
sector dimensions sit on and beside the 8-wide sub-tiles, the 32x32 and 64x48
tiles and the chunks of 16 of the inner dimension, staged by cp.async and by bulk
copies, against numpy.

Bound: a product of inner dimension d followed by one of inner dimension e, summed
over t terms, by the three-multiplication form (each real sum at most twice the
complex magnitudes), is within 8 (d + e + t) 2^-53 of sum |alpha| |L| |X| |R|^T,
element by element.
"""
import numpy as np
import pytest

from tsc_tri_t1t2j1j2_b200 import Context
from tsc_tri_t1t2j1j2_b200.blocksparse import Problem, random_psi

SMALL = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40]
LARGE = [1, 3, 8, 17, 33, 47, 48, 49, 63, 64, 65, 97, 129, 200]


def problem(rng, d, e, alphas):
    P = Problem(d=list(d), e=list(e))

    def blocks(s, dims):
        return [rng.standard_normal((dims[i + s], dims[i])) + 1j * rng.standard_normal((dims[i + s], dims[i]))
                if 0 <= i + s < len(dims) else None for i in range(len(dims))]

    P.left = [(s, blocks(s, P.d)) for s in (0, 1, -1)]
    P.right = [(s, blocks(s, P.e)) for s in (0, 1, -1)]
    P.terms = [(a, k % 3, k % 3) for k, a in enumerate(alphas)]
    return P


def reference(P, x, weight=lambda d, e, t: d + e + t, unit=8 * 2.0 ** -53):
    out, bound, off = [], [], 0
    X = []
    for d, e in zip(P.d, P.e):
        X.append(x[off:off + d * e].reshape((d, e), order="F"))
        off += d * e
    for j in range(P.K):
        y = np.zeros((P.d[j], P.e[j]), complex)
        b = np.zeros((P.d[j], P.e[j]))
        for al, a, c in P.terms:
            i = j - P.left[a][0]
            if not 0 <= i < P.K:
                continue
            L, R = P.left[a][1][i], P.right[c][1][i]
            y += al * (L @ X[i] @ R.conj().T)
            b += weight(P.d[i], P.e[i], len(P.terms)) * abs(al) * (abs(L) @ abs(X[i]) @ abs(R).T)
        out.append(y.ravel(order="F"))
        bound.append(unit * b.ravel(order="F"))
    return np.concatenate(out), np.concatenate(bound)


@pytest.mark.gpu
@pytest.mark.parametrize("tile", ["32x32", "64x48", "64x48 bulk"])
@pytest.mark.parametrize("alphas", [(1.0,), (0.7, -1.3, 2.0, 1e-3, 5.0), (0.3 + 0.4j, -1.0, 1j)],
                         ids=["one", "real", "complex"])
def test_tile_edges(tile, alphas):
    import torch
    rng = np.random.default_rng(7)
    if tile == "32x32":
        d, e = SMALL, SMALL[::-1]
    else:   # past 8 (32) GFLOP in each phase through the last sector, where the large tile (bulk copies) takes over
        big = 1650 if "bulk" in tile else 1100
        d, e = LARGE + [big], LARGE[::-1] + [big + 9]
    P = problem(rng, d, e, [complex(a) for a in alphas])
    ctx = Context(4, 4)
    try:
        n, _, flops = ctx.blocksparse_set([P])
        assert (flops >= 16e9) == (tile != "32x32") and (flops >= 64e9) == ("bulk" in tile)
        x = random_psi(rng, [P])
        dx = torch.from_numpy(x).cuda()
        out = torch.full_like(dx, float("nan"))
        torch.cuda.synchronize()
        got = []
        for _ in range(2):   # the job counter starts over
            ctx.blocksparse_apply(dx.data_ptr(), out.data_ptr(), Context.FP64)
            torch.cuda.synchronize()
            got.append(out.cpu().numpy())
    finally:
        ctx.close()
    assert np.array_equal(got[0], got[1])
    ref, bound = reference(P, x)
    assert np.all(np.abs(got[0] - ref) <= bound)
