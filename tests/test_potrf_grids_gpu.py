"""Tile Cholesky and inverse on every kind of grid: two CTAs, odd counts, half the
device (beside a panel's updates) and all of it.  A block's products are summed in the
same order whoever forms it, so the bits do not depend on the grid."""
import numpy as np
import pytest

from test_potrf_tile_gpu import EPS, tile

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [129, 320, 705, 1350])
def test_grids_agree(ctx, n):
    from hicma_parsec_b200 import tlr
    lib, A = tlr.load_library(), tile(n, n)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    out = []
    for grid in (2, 3, 5, 16, 37, nsm // 2, nsm, 0):
        ctx.set_tuning(32, grid)
        dA = torch.from_numpy(A.T.copy()).cuda()
        dX = torch.full((n, n), 3.0, dtype=torch.float64, device="cuda")
        info = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        try:
            assert lib.hicma_tlr_k_potrf(ctx.h, n, dA.data_ptr(), n, dX.data_ptr(), info.data_ptr(), 0) == 0
        finally:
            ctx.set_tuning(32, 0)
        assert int(info.item()) == 0
        out.append((dA.cpu().numpy().T, dX.cpu().numpy().T))
    L, X = out[0]
    assert np.linalg.norm(L @ L.T - A) <= 10 * n * EPS * np.linalg.norm(A)
    for l, x in out[1:]:
        assert np.array_equal(l, L) and np.array_equal(x, X)


def test_lookahead_does_not_change_the_factor(ctx):
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=2, beta=0.1, noise=0.1)
    A, B = tlr.TLRMatrix(ctx, 2700, 270, 130, 1), tlr.TLRMatrix(ctx, 2700, 270, 130, 1)
    try:
        assert A.generate(prob, 1e-8) == 0
        B.copy_from(A)
        assert A.potrf(1e-8) == 0 and B.potrf(1e-8, lookahead=0) == 0
        assert A.logdet() == B.logdet() and np.array_equal(A.uncompress(), B.uncompress())
    finally:
        A.close()
        B.close()
