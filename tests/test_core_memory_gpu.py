"""Wide core SVDs whose columns, sorted values or pivot column lie in the workspace
instead of shared memory.  Only cores of thousands of columns need that, so a low
shared memory limit (read when a context is created) brings small ones there; the
arithmetic is the same, so the results are the same bits."""
import numpy as np
import pytest

from test_core_svd_gpu import orth, update

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
