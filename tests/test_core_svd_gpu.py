"""Core SVD of a recompression at the edges of its kernels: the one-CTA kernel's
width instances (16 to 96), the cluster sizes (4, 8 and 16 CTAs) and the cores
whose T does not fit the cluster's shared memory, with full, truncated, graded
and rank-deficient spectra.  Reference: numpy on the same factors in FP64.

Tolerances: the two QRs and the core are backward stable, so the update is the
truncated SVD of a matrix within p(K) eps sigma_1 of the exact one; the
truncation threshold lies in a gap of at least a factor 3 of the spectrum, which
at most doubles that.  p(K) = 100 K covers the constants of the three steps.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

EPS = 2.0 ** -52


def orth(rng, n, k):
    return np.linalg.qr(rng.standard_normal((n, k)))[0]


def update(ctx, nb, Cu, Cv, Au, Av, Bu, Bv, acc, maxrank, fixed_rank=0):
    from hicma_parsec_b200 import tlr
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    ra, rb, rc = Au.shape[1], Bu.shape[1], Cu.shape[1]
    dCu = torch.zeros((maxrank, nb), dtype=torch.float64, device="cuda")
    dCv = torch.zeros_like(dCu)
    dCu[:rc], dCv[:rc] = dev(Cu), dev(Cv)
    dAu, dAv, dBu, dBv = dev(Au), dev(Av), dev(Bu), dev(Bv)
    r = ctypes.c_int(rc)
    torch.cuda.synchronize()
    st = tlr.load_library().hicma_tlr_k_lr_update(ctx.h, nb, dAu.data_ptr(), dAv.data_ptr(), ra, dBu.data_ptr(),
                                                  dBv.data_ptr(), rb, dCu.data_ptr(), dCv.data_ptr(),
                                                  ctypes.byref(r), acc, maxrank, fixed_rank)
    assert st == 0, tlr.last_error()
    return r.value, dCu.cpu().numpy()[:r.value].T, dCv.cpu().numpy()[:r.value].T


@pytest.mark.parametrize("K", [2, 7, 16, 17, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 130, 160, 161, 257, 448, 449, 700])
@pytest.mark.parametrize("spectrum", ["graded", "flat", "deficient"])
def test_core_svd_edges(ctx, K, spectrum):
    nb = max(320, 2 * K + 40)
    rng = np.random.default_rng(17 * K + len(spectrum))
    rc = K // 2
    ra = K - rc
    decay = {"graded": 10.0 ** np.linspace(1.0, -9.0, K), "flat": np.linspace(2.0, 1.0, K),
             "deficient": np.where(np.arange(K) < (K + 3) // 4, 1.0, 0.0)}[spectrum]
    Cu, Au = orth(rng, nb, rc), orth(rng, nb, ra)
    Cv = orth(rng, nb, rc) * decay[1::2]
    # Y = Bu (Bv^T Av) with Bv = Av: Y = Bu
    Av = orth(rng, nb, ra)
    Y = orth(rng, nb, ra) * decay[0::2]
    if spectrum == "deficient" and ra > 1:
        Au[:, -1] = Au[:, 0]          # a dependent column on the U side
    Qu, Ru = np.linalg.qr(np.hstack([Cu, Au]))
    Qv, Rv = np.linalg.qr(np.hstack([Cv, -Y]))
    u, s, vt = np.linalg.svd(Ru @ Rv.T)
    if spectrum == "flat":
        acc = 1e-8                    # nothing truncated
    else:
        # a gap of a factor 3 or more, as deep as the spectrum has one well above rounding
        gaps = [i for i in range(1, K) if s[i - 1] > 1e-10 and s[i - 1] > 3.0 * max(s[i], 1e-300)]
        acc = float(np.sqrt(s[gaps[-1] - 1] * max(s[gaps[-1]], s[gaps[-1] - 1] / 9.0))) if gaps else 1e-8
    r_ref = int((s >= acc).sum())
    # the block's own dot products Bv^T Av = I only to rounding: Bu carries Y
    r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, acc, max(K, 1))
    assert r == r_ref
    ref = (Qu @ u[:, :r]) * s[:r] @ (Qv @ vt[:r].T).T
    assert np.linalg.norm(U @ V.T - ref, 2) <= 100 * K * EPS * s[0]
    assert np.abs(U.T @ U - np.eye(r)).max() <= 100 * K * EPS
    assert np.abs(np.linalg.norm(V, axis=0) - s[:r]).max() <= 100 * K * EPS * s[0]


@pytest.mark.parametrize("K,fixed", [(12, 5), (40, 40), (90, 33), (150, 70), (300, 300)])
def test_core_svd_fixed_rank(ctx, K, fixed):
    """fixed_rank keeps that many columns whatever the accuracy (zero columns past the numerical rank)."""
    nb = 700
    rng = np.random.default_rng(K)
    rc = K // 2
    Cu, Au, Cv, Av = orth(rng, nb, rc), orth(rng, nb, K - rc), orth(rng, nb, rc), orth(rng, nb, K - rc)
    Y = orth(rng, nb, K - rc)
    r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, 1e-8, K, fixed)
    assert r == fixed
    s = np.linalg.svd(Cu @ Cv.T - Au @ Y.T, compute_uv=False)
    assert abs(np.linalg.norm(U @ V.T) - np.sqrt((s[:fixed] ** 2).sum())) <= 100 * K * EPS * np.linalg.norm(s[:fixed])


@pytest.mark.parametrize("nb", [21, 33, 64, 100, 257, 1030])
@pytest.mark.parametrize("K", [5, 17, 40, 64])
def test_narrow_qr_row_slices(ctx, nb, K):
    """Stacks up to 64 columns with few rows: the clusters of CTAs that share a
    matrix when a launch has few of them get partial, single or no row chunks."""
    K = min(K, nb - 1)
    rng = np.random.default_rng(nb * 100 + K)
    rc = K // 2
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, K - rc), orth(rng, nb, K - rc)
    Cv, Y = orth(rng, nb, rc) * np.linspace(3.0, 1.0, rc), orth(rng, nb, K - rc)
    ref = Cu @ Cv.T - Au @ Y.T
    s = np.linalg.svd(ref, compute_uv=False)
    r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, 1e-6, max(K, 1))
    assert r == int((s >= 1e-6).sum())
    # backward stable QRs and core: 100 K eps sigma_1, plus what the truncation at 1e-6 may drop
    assert np.linalg.norm(U @ V.T - ref, 2) <= 100 * K * EPS * s[0] + (s[r] if r < len(s) else 0.0)
    assert np.abs(U.T @ U - np.eye(r)).max() <= 100 * K * EPS
