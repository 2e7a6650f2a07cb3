"""Wide core SVDs whose columns, sorted values or pivot column lie in the workspace
instead of shared memory.  Only cores of thousands of columns need that, so a low
shared memory limit (read when a context is created) brings small ones there; the
arithmetic is the same, so the results are the same bits."""
import numpy as np
import pytest

from test_core_svd_gpu import EPS, orth, update

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [66, 97, 161, 300, 449])
@pytest.mark.parametrize("spectrum", ["full", "deficient"])
def test_core_in_the_workspace(monkeypatch, K, spectrum):
    from hicma_parsec_b200 import tlr
    nb = K + 70
    rng = np.random.default_rng(K)
    rc = K // 2
    ra = K - rc
    keep = K if spectrum == "full" else K // 3
    decay = np.where(np.arange(K) < keep, np.linspace(2.0, 1.0, K), 0.0)
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, ra), orth(rng, nb, ra)
    Cv, Y = orth(rng, nb, rc) * decay[1::2][:rc], orth(rng, nb, ra) * decay[0::2][:ra]
    out = []
    # everything in shared memory where it fits, the pivot column alone from K = 300 on, nothing
    for limit in (None, "60000", "0"):
        if limit is None:
            monkeypatch.delenv("HICMA_TLR_CORE_SMEM", raising=False)
        else:
            monkeypatch.setenv("HICMA_TLR_CORE_SMEM", limit)
        with tlr.Context(0, 512 << 20) as ctx:
            out.append(update(ctx, nb, Cu, Cv, Au, Av, Y, Av, 1e-8, K))
    for r, U, V in out[1:]:
        assert r == out[0][0] == min(keep, K)
        assert np.array_equal(U, out[0][1]) and np.array_equal(V, out[0][2])


@pytest.mark.parametrize("K, keep", [(900, 900), (1500, 260), (2600, 100)])
def test_cores_beyond_shared_memory(ctx, K, keep):
    """Cores whose columns never fit the shared memory of a cluster: full and low numerical
    rank.  Tolerance as for the core SVD's edges."""
    nb = K + 70
    rng = np.random.default_rng(K)
    rc = K // 2
    ra = K - rc
    decay = np.where(np.arange(K) < keep, np.linspace(2.0, 1.0, K), 0.0)
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, ra), orth(rng, nb, ra)
    Cv, Y = orth(rng, nb, rc) * decay[1::2][:rc], orth(rng, nb, ra) * decay[0::2][:ra]
    Qu, Ru = np.linalg.qr(np.hstack([Cu, Au]))
    Qv, Rv = np.linalg.qr(np.hstack([Cv, -Y]))
    s = np.linalg.svd(Ru @ Rv.T, compute_uv=False)
    r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, 1e-8, K)
    assert r == keep
    assert np.linalg.norm(U @ V.T - (Cu @ Cv.T - Au @ Y.T), 2) <= 100 * K * EPS * s[0]
    assert np.abs(U.T @ U - np.eye(r)).max() <= 100 * K * EPS
    assert np.abs(np.linalg.norm(V, axis=0) - s[:r]).max() <= 100 * K * EPS * s[0]
