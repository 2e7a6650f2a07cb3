"""Tile Cholesky and inverse at the edges of its block tasks: one and two block
columns, an odd and an even number of block rows below the diagonal (row pairs),
partial last blocks, odd leading dimensions (the path without 16-byte copies),
and every number of CTAs from the smallest.  Reference: numpy.

Tolerances: blocked Cholesky and forward substitution are backward stable with a
constant of about n; the tile's condition is below 1e6, so ||L L^T - A|| / ||A|| <=
10 n eps and ||X L - I|| <= 10 n eps cond(L) hold with room.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

EPS = 2.0 ** -52


def tile(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n))
    return G @ G.T / n + 0.05 * np.eye(n)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 192, 257, 320, 511, 769, 1024])
@pytest.mark.parametrize("pad", [0, 1, 2])
def test_potrf_tile_edges(ctx, n, pad):
    from hicma_parsec_b200 import tlr
    lib, lda = tlr.load_library(), n + pad
    A = tile(n, n)
    h = np.full((n, lda), 7.0)
    h[:, :n] = A.T
    for grid, inverse in ((0, True), (2, True), (0, False)):
        ctx.set_tuning(32, grid)
        dA = torch.from_numpy(h.copy()).cuda()
        dX = torch.full((n, n), 3.0, dtype=torch.float64, device="cuda")
        info = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        try:
            rc = lib.hicma_tlr_k_potrf(ctx.h, n, dA.data_ptr(), lda, dX.data_ptr() if inverse else None,
                                       info.data_ptr(), 0)
        finally:
            ctx.set_tuning(32, 0)
        assert rc == 0, tlr.last_error()
        assert int(info.item()) == 0
        out = dA.cpu().numpy()
        L = out[:, :n].T
        assert np.array_equal(np.triu(L, 1), np.zeros((n, n)))
        assert np.array_equal(out[:, n:], h[:, n:])       # nothing written past the tile
        assert np.linalg.norm(L @ L.T - A) <= 10 * n * EPS * np.linalg.norm(A)
        if inverse:
            X = dX.cpu().numpy().T
            assert np.array_equal(np.triu(X, 1), np.zeros((n, n)))
            assert np.linalg.norm(X @ L - np.eye(n)) <= 10 * n * EPS * np.linalg.cond(L) * np.sqrt(n)


@pytest.mark.parametrize("n,bad", [(64, 0), (200, 130), (700, 699), (700, 64), (700, 385)])
def test_potrf_tile_reports_the_pivot(ctx, n, bad):
    from hicma_parsec_b200 import tlr
    A = tile(n, n + bad)
    A[bad, bad] = -1.0
    dA = torch.from_numpy(A.T.copy()).cuda()
    dX = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rc = tlr.load_library().hicma_tlr_k_potrf(ctx.h, n, dA.data_ptr(), n, dX.data_ptr(), info.data_ptr(), 1000)
    assert rc == 0
    assert int(info.item()) == 1000 + bad + 1
