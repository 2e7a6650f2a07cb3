"""A staging ring so small that it wraps many times in every panel (its size is read when
a context is created): the same launches on the same data, so the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, n, nb, cap, acc, prec", [
    (2, 2700, 270, 130, 1e-8, 0),     # narrow stacks, the exact case of the reference
    (2, 2700, 270, 130, 1e-8, 1),     # FP32 products by norm
    (3, 2500, 250, 124, 1e-9, 0),     # narrow and wide stacks side by side
    (4, 2400, 200, 99, 1e-6, 0),      # wide stacks, cores of several widths
])
def test_wrapping_ring_changes_nothing(monkeypatch, kind, n, nb, cap, acc, prec):
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=kind, beta=0.1, noise=0.1)
    b = np.random.default_rng(n).standard_normal((n, 3))
    out = []
    for size in (None, "40960", "20480"):
        if size is None:
            monkeypatch.delenv("HICMA_TLR_STAGE_BYTES", raising=False)
        else:
            monkeypatch.setenv("HICMA_TLR_STAGE_BYTES", size)
        with tlr.Context(0, 1 << 30) as ctx:
            ctx.set_precision(prec)
            A = tlr.TLRMatrix(ctx, n, nb, cap, 1)
            info = A.generate(prob, acc)
            if info:
                A.band_regenerate(prob, max(m - k for m, k in A.rejected_tiles()) + 1)
            assert A.potrf(acc) == 0
            out.append((A.rank_map(), A.logdet(), A.solve(b.copy()), A.uncompress()))
            A.close()
    for other in out[1:]:
        for x, y in zip(out[0], other):
            assert np.array_equal(np.asarray(x), np.asarray(y))
