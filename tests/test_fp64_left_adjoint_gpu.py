"""The FP64 grouped kernel with a conjugate-transposed left operand at the edges of its
tiles: the left-to-right wavefunction transformation, whose first list is U^H psi and whose
second multiplies by T^H, on sectors without spin (every recoupling coefficient is one).
Sector dimensions sit beside the 8-wide sub-tiles, the 32x32 and 64x48 tiles and the chunks
of 16 of the inner dimension; one large sector takes the lists to the larger kernels.

Bound, element by element, for the result before it is normalised: as in
test_fp64_tiles_gpu, 8 (D + E + 1) 2^-53 of |U|^H |psi| |T|^H.  The norm divides by a sum
whose longest chain is under 100 additions, so it adds norm(bound) / norm(result) + 100 2^-53
of each element.
"""
import numpy as np
import pytest

from tsc_tri_t1t2j1j2_b200 import Context
from tsc_tri_t1t2j1j2_b200.layout import Basis, Block, Wave

# (rows of U, columns of U, rows and columns of T) per sector
SMALL = [(1, 1, 1, 1), (3, 2, 5, 7), (8, 8, 8, 8), (17, 9, 15, 31), (33, 16, 31, 32), (47, 33, 40, 17), (16, 40, 3, 33)]
LARGE = SMALL + [(63, 64, 49, 48), (65, 49, 65, 47), (130, 65, 97, 64), (50, 129, 18, 97)]


def random(rng, r, c):
    return rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))


@pytest.mark.gpu
@pytest.mark.parametrize("tile,sizes", [("32x32", SMALL), ("64x48", LARGE + [(1037, 1101, 1001, 1029)]),
                                        ("64x48 bulk", LARGE + [(1651, 1590, 1685, 1613)])])
def test_left_adjoint_tile_edges(tile, sizes):
    for k in (0, 1):   # GFLOP of the two lists: the kernel each runs on
        gf = 8e-9 * sum(c * e * (d if k == 0 else f) for d, c, f, e in sizes)
        assert (gf >= 8) == (tile != "32x32") and (gf >= 32) == ("bulk" in tile)
    rng = np.random.default_rng(11)
    n = len(sizes)
    q = [(2 * k, 2 * (n - k)) for k in range(n)]   # electrons left and right
    U = [random(rng, d, c) for d, c, _, _ in sizes]
    T = [random(rng, f, e) for _, _, f, e in sizes]
    X = [random(rng, d, e) for d, _, _, e in sizes]

    def basis(side, dims):
        return Basis(4, sum(dims), np.array([[s[side], 0, m, 1] for s, m in zip(q, dims)], np.int32),
                     np.array([[s[side], 0, 0, 0, 0, m] for s, m in zip(q, dims)], np.int32))

    def block(side, mats):
        return Block(4, 0, 0, np.array([[s[side], 0, 0, *a.shape] for s, a in zip(q, mats)], np.int32), mats,
                     sum(a.shape[1] for a in mats))

    def wave(rows, cols, vec):
        return Wave(4, 4, np.array([[s[0], 0, s[1], 0, r, c] for s, r, c in zip(q, rows, cols)], np.int32), vec)

    old = wave([s[0] for s in sizes], [s[3] for s in sizes], np.concatenate([x.ravel(order="F") for x in X]))
    new = wave([s[1] for s in sizes], [s[2] for s in sizes], None)
    ctx = Context(4, 4)
    try:
        got = ctx.wave_trans(0, basis(0, [s[1] for s in sizes]), basis(1, [s[3] for s in sizes]), block(0, U),
                             block(1, T), old, new).vec
    finally:
        ctx.close()
    ref = np.concatenate([(u.conj().T @ x @ t.conj().T).ravel(order="F") for u, x, t in zip(U, X, T)])
    bound = np.concatenate([(8 * 2.0 ** -53 * (u.shape[0] + t.shape[1] + 1) * (abs(u).T @ abs(x) @ abs(t).T)).ravel(order="F")
                            for u, x, t in zip(U, X, T)])
    norm = np.linalg.norm(ref)
    bound = bound + np.abs(ref) * (np.linalg.norm(bound) / norm + 100 * 2.0 ** -53)
    assert np.all(np.abs(got * norm - ref) <= bound)
