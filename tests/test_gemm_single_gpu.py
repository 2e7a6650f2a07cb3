"""Single products at the edges of their two forms: inner dimensions around 16 and 128,
outputs of one tile, of partial tiles and of one and two waves of CTAs, the four
transpositions, even and odd leading dimensions (16- and 8-byte copies).

Reference: torch in FP64.  Tolerance: a sum of k products, each side rounded in its own
order: |difference| <= 2 (k + 2) eps (|alpha| |A| |B| + |beta| |C|), entry by entry."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

EPS = 2.0 ** -52


@pytest.mark.parametrize("m, n, k", [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 127, 17), (130, 70, 128), (70, 130, 129),
                                     (1530, 1536, 40), (1530, 1500, 300), (1600, 1590, 200),
                                     (1985, 2048, 500), (1985, 2048, 520)])
@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("pad", [0, 1])
def test_products(m, n, k, ta, tb, pad):
    from hicma_parsec_b200 import tlr
    lib = tlr.load_library()
    g = torch.Generator(device="cuda").manual_seed(m + 7 * n + k)
    rnd = lambda r, c: torch.randn(c, r + pad, dtype=torch.float64, device="cuda", generator=g)   # column-major, ld r + pad
    A, B, C = rnd(k if ta else m, m if ta else k), rnd(n if tb else k, k if tb else n), rnd(m, n)
    a, b = A[:, :k if ta else m].T, B[:, :n if tb else k].T
    a, b = (a.T if ta else a), (b.T if tb else b)
    alpha, beta = -0.75, 1.25
    ref = alpha * (a @ b) + beta * C[:, :m].T
    bound = 2 * (k + 2) * EPS * (abs(alpha) * (a.abs() @ b.abs()) + abs(beta) * C[:, :m].T.abs())
    kept = C[:, m:].clone()
    rc = lib.hicma_tlr_k_dgemm(ta, tb, m, n, k, ctypes.c_double(alpha), A.data_ptr(), A.shape[1], B.data_ptr(),
                               B.shape[1], ctypes.c_double(beta), C.data_ptr(), C.shape[1],
                               torch.cuda.current_stream().cuda_stream)
    assert rc == 0, tlr.last_error()
    assert bool(((C[:, :m].T - ref).abs() <= bound).all())
    assert torch.equal(C[:, m:], kept)
