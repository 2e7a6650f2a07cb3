"""Triangular solves with few right-hand sides at the edges of their launches:
tile sizes that are no multiple of the 32-row block, one column, a full and an
overfull 8-column block, the 32-column blocks, low-rank and dense off-diagonal
tiles.  Reference: scipy's substitution with the same factor, uncompressed.

Tolerance: every product is a sum of at most NB terms and the diagonal blocks
are applied as explicit inverses, whose error is bounded by NB eps cond(L_kk) a
block; both sweeps together stay below 2 N eps cond(L) relative to the solution,
times 10 for the constants.
"""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

EPS = 2.0 ** -52


@pytest.mark.parametrize("nb,nt,band", [(333, 4, 1), (64, 5, 2), (250, 4, 4), (97, 1, 1)])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 33, 70])
def test_solve_matches_substitution(ctx, nb, nt, band, nrhs):
    from hicma_parsec_b200 import tlr
    n = nb * nt
    prob = tlr.Problem(kind=tlr.KIND_SQEXP_2D, noise=1e-2, seed=nb)
    A = tlr.TLRMatrix(ctx, n, nb, nb // 2, 1)
    try:
        # nb 64: tiles this small are rejected by the rank rule next to the diagonal
        info = A.generate(prob, 1e-8)
        b = band if info == 0 else max([band] + [m - k + 1 for m, k in A.rejected_tiles()])
        if b > 1:
            A.band_regenerate(prob, min(b, nt))
        assert A.potrf(1e-8) == 0
        L = np.tril(A.uncompress())
        B = np.random.default_rng(nrhs).standard_normal((n, nrhs))
        X = A.solve(B)
        ref = sl.solve_triangular(L, sl.solve_triangular(L, B, lower=True), lower=True, trans="T")
        tol = 20 * n * EPS * np.linalg.cond(L)
        assert np.linalg.norm(X - ref) <= tol * np.linalg.norm(ref)
        assert np.array_equal(A.solve(B[:, 0]), A.solve(B[:, 0]))
    finally:
        A.close()
