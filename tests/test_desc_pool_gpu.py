"""Descriptor memory from the device's pool: reused regions are zero-filled, contexts
on threads share the pool, the last context gives it back."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from hicma_parsec_b200 import tlr

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("nt, nb, cap, band", [(1, 64, 8, 1), (3, 96, 40, 1), (4, 64, 16, 2)])
def test_reused_storage_is_zero(nt, nb, cap, band):
    rng = np.random.default_rng(nt)
    with tlr.Context(0, 256 << 20) as ctx:
        for _ in range(2):
            A = tlr.TLRMatrix(ctx, nt * nb, nb, cap, band)
            for m in range(nt):
                for n in range(max(0, m - band + 1), m + 1):
                    D = A.tile(m, n)
                    assert not np.any(np.asarray(D))
                    A.set_tile(m, n, rng.standard_normal((nb, nb)))
            A.close()


def test_threads_share_the_pool():
    prob = tlr.Problem(kind=2, noise=0.1)

    def work(out, q):
        with tlr.Context(0, 512 << 20) as ctx:
            res = []
            for n in (1024, 2048, 1024, 4096):
                A = tlr.TLRMatrix(ctx, n, 256, 127, 1)
                assert A.generate(prob, 1e-8) == 0
                assert A.potrf(1e-8) == 0
                res.append(A.logdet())
                A.close()
            out[q] = res

    out = {}
    work(out, "alone")
    threads = [threading.Thread(target=work, args=(out, q)) for q in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for q in range(3):
        assert out[q] == out["alone"]


GIVES_BACK = """
import torch
from hicma_parsec_b200 import tlr
keep = tlr.Context(0, 256 << 20)
free0 = torch.cuda.mem_get_info(0)[0]
tlr.TLRMatrix(keep, 8 * 2048, 2048, 2048, 1).close()     # 8 dense tiles + 28 full slots: 2.1 GB
assert free0 - torch.cuda.mem_get_info(0)[0] >= 1 << 30  # kept for the next descriptor
keep.close()
torch.cuda.synchronize()
assert torch.cuda.mem_get_info(0)[0] >= free0
"""


def test_last_context_gives_the_memory_back():
    # in a process of its own: contexts of other tests share this process's pool
    r = subprocess.run([sys.executable, "-c", GIVES_BACK], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
