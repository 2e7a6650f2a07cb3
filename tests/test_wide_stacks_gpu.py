"""Updates whose stacks are wider than tall (K = rc + ra > nb: ranks above half the tile),
by the default QRs and with HICMA_TLR_QR=householder.  Reference: numpy in FP64.

Tolerance: as for the core SVD's edges, 100 K eps sigma_1 for the product, plus the
largest singular value that is dropped; 100 K eps sigma_1 / sigma_r for the
orthogonality of the new U, whose r-th column is determined to that by the product."""
import numpy as np
import pytest

from test_core_svd_gpu import EPS, orth, update

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [None, "householder"])
@pytest.mark.parametrize("nb, rc, ra, lo", [(33, 30, 20, -3), (40, 36, 36, -9), (64, 64, 64, -2), (65, 65, 65, -2),
                                            (100, 70, 31, -6), (100, 70, 70, -6), (100, 100, 100, -2), (150, 140, 140, -4),
                                            (150, 10, 150, -6), (200, 200, 199, -6), (257, 250, 250, -3)])
def test_update_wider_than_tall(monkeypatch, mode, nb, rc, ra, lo):
    from hicma_parsec_b200 import tlr
    if mode:
        monkeypatch.setenv("HICMA_TLR_QR", mode)
    else:
        monkeypatch.delenv("HICMA_TLR_QR", raising=False)
    rng = np.random.default_rng(1000 * nb + ra)
    K = rc + ra
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, ra), orth(rng, nb, ra)
    Cv = orth(rng, nb, rc) * 10.0 ** np.linspace(0, lo, rc)
    Y = orth(rng, nb, ra) * 10.0 ** np.linspace(0, lo, ra)
    ref = Cu @ Cv.T - Au @ Y.T
    s = np.linalg.svd(ref, compute_uv=False)
    # cut in the widest gap of the upper half of the spectrum's logarithm
    i = int(np.argmax(s[nb // 2:-1] / s[nb // 2 + 1:])) + nb // 2
    acc = float(np.sqrt(s[i] * s[i + 1]))
    with tlr.Context(0, 512 << 20) as ctx:
        r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, acc, K)
    assert r == i + 1
    assert np.linalg.norm(U @ V.T - ref, 2) <= s[r] + 100 * K * EPS * s[0]
    assert np.abs(U.T @ U - np.eye(r)).max() <= 100 * K * EPS * s[0] / s[r - 1]


@pytest.mark.parametrize("nb, rc, ra, what", [(100, 70, 70, "zero"), (100, 70, 70, "dependent"), (60, 40, 40, "zero"),
                                              (150, 100, 120, "dependent"), (150, 20, 150, "zero"), (200, 0, 200, "zero"),
                                              (140, 70, 70, "dependent"), (128, 64, 64, "dependent"), (300, 150, 150, "dependent"),
                                              (71, 35, 36, "dependent"), (141, 70, 70, "dependent")])
def test_new_directions_after_a_gap(nb, rc, ra, what):
    """The first new columns bring nothing (zero, or copies of old ones), the last ones do: with
    K > nb the basis is not full when nb columns are through, with K = nb the rounding errors
    of the copies fill it exactly."""
    from hicma_parsec_b200 import tlr
    rng = np.random.default_rng(nb + rc)
    K = rc + ra
    Cu, Au, Av = orth(rng, nb, rc), orth(rng, nb, ra), orth(rng, nb, ra)
    gap = min(ra - 10, max(rc, 40))
    Au[:, :gap] = 0.0 if what == "zero" else Cu[:, np.arange(gap) % max(rc, 1)]
    Cv, Y = orth(rng, nb, rc) * np.linspace(3.0, 1.0, rc), orth(rng, nb, ra) * np.linspace(2.0, 1.0, ra)
    ref = Cu @ Cv.T - Au @ Y.T
    s = np.linalg.svd(ref, compute_uv=False)
    acc = 1e-6
    with tlr.Context(0, 512 << 20) as ctx:
        r, U, V = update(ctx, nb, Cu, Cv, Au, Av, Y, Av, acc, max(K, 1))
    assert r == int((s >= acc).sum())
    assert np.linalg.norm(U @ V.T - ref, 2) <= 100 * K * EPS * s[0] + (s[r] if r < len(s) else 0.0)
    assert np.abs(U.T @ U - np.eye(r)).max() <= 100 * K * EPS * s[0] / s[r - 1]
