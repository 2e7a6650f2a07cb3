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


def test_a_failed_factorization_leaves_the_context_usable(monkeypatch):
    """Rings too small for the task arrays of one launch or another of a panel: the
    factorization fails there, on the bulk or on the side stream, and the next solve is as
    ever."""
    from hicma_parsec_b200 import tlr
    prob = tlr.Problem(kind=4, beta=0.1, noise=0.1)
    n, nb, cap = 4800, 200, 99
    b = np.random.default_rng(0).standard_normal((n, 2))
    monkeypatch.delenv("HICMA_TLR_STAGE_BYTES", raising=False)
    with tlr.Context(0, 1 << 30) as ctx:
        A, F = tlr.TLRMatrix(ctx, n, nb, cap, 1), tlr.TLRMatrix(ctx, n, nb, cap, 1)
        if A.generate(prob, 1e-6):
            A.band_regenerate(prob, max(m - k for m, k in A.rejected_tiles()) + 1)
        F.copy_from(A)
        assert F.potrf(1e-6) == 0
        x = F.solve(b.copy())
        failed = 0
        for size in range(4096, 49152, 4096):
            monkeypatch.setenv("HICMA_TLR_STAGE_BYTES", str(size))
            with tlr.Context(0, 1 << 30) as tight:
                B, G = tlr.TLRMatrix(tight, n, nb, cap, 1), tlr.TLRMatrix(tight, n, nb, cap, 1)
                B.copy_from(A)
                G.copy_from(F)
                try:
                    assert B.potrf(1e-6) == 0
                except tlr.TLRError as e:
                    assert "staging failed" in str(e)
                    failed += 1
                assert np.array_equal(G.solve(b.copy()), x)
                B.copy_from(A)
                B.close()
                G.close()
        assert failed >= 3
