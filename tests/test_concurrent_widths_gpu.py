"""Contexts on threads whose launches of one kernel need different amounts of shared
memory at the same time: every update succeeds and gives the rank and factors that
it gives alone."""
import ctypes
import threading

import numpy as np
import pytest

from test_core_svd_gpu import orth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


class Update:
    """A recompression C - A B^T of numerical rank 8 (so that the launches, not the
    rotations, take the time) on device buffers of its own."""

    def __init__(self, nb, K):
        from hicma_parsec_b200 import tlr
        self.lib, self.ctx, self.nb, self.K = tlr.load_library(), tlr.Context(0, 512 << 20), nb, K
        rng = np.random.default_rng(K)
        self.rc, self.ra = K // 2, K - K // 2
        U, V = orth(rng, nb, 8), orth(rng, nb, 8)
        Cu, Au, Av = orth(rng, nb, self.rc), U @ rng.standard_normal((8, self.ra)), orth(rng, nb, self.ra)
        Cv, Y = np.zeros((nb, self.rc)), V @ rng.standard_normal((8, self.ra))
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
        self.Au, self.Av, self.Y = dev(Au), dev(Av), dev(Y)
        self.C0 = torch.zeros((2, K, nb), dtype=torch.float64, device="cuda")
        self.C0[0, :self.rc], self.C0[1, :self.rc] = dev(Cu), dev(Cv)
        self.C = torch.empty_like(self.C0)
        self.stream = torch.cuda.Stream()

    def __call__(self):
        with torch.cuda.stream(self.stream):
            self.C.copy_(self.C0)
        self.stream.synchronize()
        r = ctypes.c_int(self.rc)
        st = self.lib.hicma_tlr_k_lr_update(self.ctx.h, self.nb, self.Au.data_ptr(), self.Av.data_ptr(), self.ra,
                                            self.Y.data_ptr(), self.Av.data_ptr(), self.ra, self.C[0].data_ptr(),
                                            self.C[1].data_ptr(), ctypes.byref(r), 1e-6, self.K, 0)
        return st, r.value

    def factors(self):
        return self.C[:, :8].cpu().numpy()


@pytest.mark.parametrize("mode, sizes, loops", [
    # core SVD on clusters of 4 CTAs with 58 KB each, and of 8 with 78 to 178 KB
    (None, ((400, 280), (500, 420)) + 6 * ((200, 70),), 600),
    # Householder QRs: 32-column panels of long stacks, and of short ones
    ("householder", ((780, 70), (700, 70)) + 6 * ((200, 70),), 1500),
])
def test_widths_side_by_side(monkeypatch, mode, sizes, loops):
    from hicma_parsec_b200 import tlr
    if mode:
        monkeypatch.setenv("HICMA_TLR_QR", mode)
    else:
        monkeypatch.delenv("HICMA_TLR_QR", raising=False)
    ups = [Update(nb, K) for nb, K in sizes]
    try:
        alone = []
        for u in ups:
            assert u() == (0, 8), tlr.last_error()
            alone.append(u.factors())
        bad = []
        left = threading.Semaphore(0)   # released by each of the first two threads when it is done

        def wide(q):
            for _ in range(loops):
                got = ups[q]()
                if got != (0, 8):
                    bad.append((q, got, tlr.last_error()))
            left.release()

        def narrow(q):
            while left._value < 2:
                got = ups[q]()
                if got != (0, 8):
                    bad.append((q, got, tlr.last_error()))

        threads = [threading.Thread(target=wide if q < 2 else narrow, args=(q,)) for q in range(len(sizes))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, (len(bad), bad[:3])
        for u, a in zip(ups, alone):
            assert np.array_equal(u.factors(), a)
    finally:
        for u in ups:
            u.ctx.close()
