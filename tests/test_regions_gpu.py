"""Memory kept for the next descriptors goes to another allocation of the library that
needs it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import torch
from hicma_parsec_b200 import tlr
torch.zeros(1, device="cuda")
keep = tlr.Context(0, 256 << 20)
tlr.TLRMatrix(keep, 8 * 2048, 2048, 2048, 1).close()      # 2.1 GB, kept
free = torch.cuda.mem_get_info(0)[0]
with tlr.Context(0, free + (1 << 30)) as big:             # more than is free without it
    assert torch.cuda.mem_get_info(0)[0] < 2 << 30
    try:
        tlr.TLRMatrix(big, 8 * 2048, 2048, 2048, 1)
    except tlr.TLRError as e:                             # nothing is left for a descriptor
        assert e.code == tlr.ERR_OOM
    else:
        raise AssertionError("2.1 GB out of less than 2")
A = tlr.TLRMatrix(keep, 8 * 2048, 2048, 2048, 1)          # and again once that context is gone
A.close()
keep.close()
"""


def test_kept_memory_is_found_when_it_is_needed():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=REPO, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
