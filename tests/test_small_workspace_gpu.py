"""Updates and compressions in the smallest workspace that each needs with Householder QRs:
the block QRs and the wide core SVD, which want more scratch, leave them to it there.
The sizes below are what one task needs, in arrays of doubles rounded up to 256 bytes."""
import ctypes

import numpy as np
import pytest

from test_core_svd_gpu import EPS, orth, update

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def arrays(*counts):
    return sum((8 * n + 1 + 255) // 256 * 256 for n in counts)


def panel(nb):
    pb = 200 * 1024 // (nb * 8 + 1)
    return next((p for p in (32, 16, 8, 4) if pb >= p), 2)


def workspace(main):
    """Workspace whose bulk part (seven eighths of it) holds `main` bytes."""
    return (main * 8 // 7 + 4095) // 2048 * 2048


def update_bytes(nb, rc, ra, rb):
    K, pb = rc + ra, panel(nb)
    tri = lambda n: (-(-n // pb) + 1) * pb * pb
    b = 3 * arrays(nb * K) + arrays(ra, K, tri(ra), tri(K), rc * ra, rc * ra, nb * ra, ra * ra) + 6 * arrays(K * K)
    return b + (arrays(K * K + 4 * K + 16) if K > 160 else 0) + arrays(rb * ra) + 1024


def compress_bytes(nb, s):
    pb = panel(nb)
    b = 4 * arrays(nb * s) + 2 * arrays(s) + 2 * arrays((-(-s // pb) + 1) * pb * pb) + 3 * arrays(s * s)
    return b + (arrays(s * s + 4 * s + 16) if s > 160 else 0) + 1024


@pytest.mark.parametrize("nb, rc, ra", [(70, 40, 25), (100, 99, 1), (300, 60, 6), (300, 150, 150), (1000, 66, 1),
                                        (2000, 65, 5), (900, 100, 70), (1030, 300, 150), (1400, 350, 350)])
def test_update_in_the_smallest_workspace(nb, rc, ra):
    from hicma_parsec_b200 import tlr
    rng = np.random.default_rng(nb + ra)
    K = rc + ra
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, ra), orth(rng, nb, ra)
    Cv, Y = orth(rng, nb, rc) * np.linspace(3.0, 1.0, rc), orth(rng, nb, ra)
    ref = Cu @ Cv.T - Au @ Y.T
    s = np.linalg.svd(ref, compute_uv=False)
    with tlr.Context(0, workspace(256 + update_bytes(nb, rc, ra, ra))) as ctx:
        r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, 1e-6, K)
    assert r == int((s >= 1e-6).sum())
    # backward stable QRs and core, as for the core SVD's edges
    assert np.linalg.norm(U @ V.T - ref, 2) <= 100 * K * EPS * s[0] + (s[r] if r < len(s) else 0.0)


@pytest.mark.parametrize("nb, maxrank", [(80, 70), (170, 150), (300, 60), (1000, 100), (600, 250), (1500, 480)])
def test_compress_in_the_smallest_workspace(nb, maxrank):
    from hicma_parsec_b200 import tlr
    rng = np.random.default_rng(nb)
    k = min(maxrank, nb // 2 - 1)      # numerical rank, below half the tile
    T = (orth(rng, nb, k) * np.linspace(2.0, 1.0, k)) @ orth(rng, nb, k).T
    s = min(maxrank + 10, nb)
    dA = torch.from_numpy(np.ascontiguousarray(T.T)).cuda()
    dU = torch.zeros((maxrank, nb), dtype=torch.float64, device="cuda")
    dV = torch.zeros_like(dU)
    r = ctypes.c_int()
    torch.cuda.synchronize()
    with tlr.Context(0, workspace(arrays(nb * s, s * s, 1, 1) + compress_bytes(nb, s))) as ctx:
        st = tlr.load_library().hicma_tlr_k_compress(ctx.h, nb, dA.data_ptr(), dU.data_ptr(), dV.data_ptr(), maxrank,
                                                     1e-8, ctypes.byref(r))
        assert st == 0, tlr.last_error()
    assert r.value == k
    U, V = dU.cpu().numpy()[:k].T, dV.cpu().numpy()[:k].T
    # the range finder and the core lose 100 s eps; nothing is truncated at 1e-8
    assert np.linalg.norm(U @ V.T - T, 2) <= 100 * s * EPS * 2.0 * np.sqrt(nb)


@pytest.mark.parametrize("nb, cap, acc, beta", [(400, 190, 1e-9, 0.1), (600, 250, 1e-10, 0.05)])
def test_generate_in_the_smallest_workspace(nb, cap, acc, beta):
    """The samples grow past 64 columns and the block QRs do not fit: the same ranks as with
    room within 1, as for the two QR paths, and the same tiles to the accuracy."""
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=2, beta=beta, noise=0.1)
    s = min(cap + 10, nb)
    out = []
    for ws in (1 << 30, workspace(arrays(nb * s, s * s, 9, nb * nb) + 1024 + compress_bytes(nb, s))):
        with tlr.Context(0, ws) as ctx:
            A = tlr.TLRMatrix(ctx, 4 * nb, nb, cap, 1)
            assert A.generate(prob, acc) == 0
            out.append([A.tile(m, n) for m, n in ((1, 0), (2, 0), (2, 1))])
            A.close()
    assert max(U.shape[1] for U, _ in out[0]) > 32      # more than the first 64 samples serve
    for (U0, V0), (U1, V1) in zip(*out):
        assert abs(U0.shape[1] - U1.shape[1]) <= 1
        T = U0 @ V0.T
        assert np.linalg.norm(T - U1 @ V1.T) <= 2.0 * acc * np.linalg.norm(T)


@pytest.mark.parametrize("odd", [1, 8, 100, 1234])
def test_workspace_of_any_size(odd):
    """A workspace that is no multiple of anything: its two parts start aligned."""
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=2, beta=0.1, noise=0.1)
    out = []
    for ws in (64 << 20, (64 << 20) + odd):
        with tlr.Context(0, ws) as ctx:
            A = tlr.TLRMatrix(ctx, 1280, 256, 120, 1)
            assert A.generate(prob, 1e-8) == 0
            assert A.potrf(1e-8) == 0
            out.append((A.logdet(), A.rank_map()))
            A.close()
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("nt, nb, band, nrhs", [(1, 96, 1, 1), (2, 100, 1, 3), (6, 128, 1, 1), (6, 128, 2, 8), (6, 130, 1, 9),
                                                (5, 200, 3, 70)])
def test_solve_in_the_smallest_workspace(nt, nb, band, nrhs):
    """The right-hand sides, one block row of them and the low-rank products: what a solve
    needs without a second copy of the right-hand sides.  Same products in the same
    order as with one, so the same bits."""
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=2, beta=0.1, noise=0.1)
    n, cap = nt * nb, nb // 2 - 1
    b = np.random.default_rng(n).standard_normal((n, nrhs))
    small = workspace(arrays(n * nrhs, nt * cap * nrhs + 1, nb * nrhs))
    with tlr.Context(0, 64 << 20) as ctx, tlr.Context(0, small) as tight:
        A, B = tlr.TLRMatrix(ctx, n, nb, cap, band), tlr.TLRMatrix(tight, n, nb, cap, band)
        info = A.generate(prob, 1e-7)
        if info:
            A.band_regenerate(prob, max(m - k for m, k in A.rejected_tiles()) + 1)
        assert A.potrf(1e-7) == 0
        B.copy_from(A)
        x, y = A.solve(b.copy()), B.solve(b.copy())
        assert np.array_equal(x, y)
        # and it is the solution: the factor holds A to acc, the nugget 0.1 bounds its inverse
        D = A.uncompress()
        L = np.tril(D)
        assert np.linalg.norm(L @ (L.T @ x) - b) <= 1e-9 * np.linalg.norm(b)
        A.close()
        B.close()
