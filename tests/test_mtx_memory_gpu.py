"""Matrix Market text with little device memory free (csrc/cuda/k_mtx.cu): where
there is room for what the host parser needs but not for the text beside it,
the text is still read."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import sys
sys.path[:0] = [%r]
import numpy as np, torch
from rvsp import read_mtx
n = 2000
body = b"\\n".join(b"%%d %%d %%d" %% (i + 1, i + 1, i) for i in range(n))
head = b"%%%%%%%%MatrixMarket matrix coordinate real general\\n%%d %%d %%d\\n" %% (n, n, n)
def same(M):
    assert np.array_equal(M.row_ptr.cpu().numpy(), np.arange(n + 1))
    assert np.array_equal(M.col_idx.cpu().numpy(), np.arange(n))
    assert np.array_equal(M.values.cpu().numpy(), np.arange(n, dtype=np.float32))
same(read_mtx(head + body, device=True))  # loads the kernels
text = head + body + b" " * (128 << 20)
from cuda.bindings import runtime as rt
def take(size):
    err, p = rt.cudaMalloc(size)
    assert err == rt.cudaError_t.cudaSuccess
    return p
def free():
    return torch.cuda.mem_get_info()[0] >> 20
hog = [take((free() - 200) << 20)]
while free() > 80:
    hog.append(take(2 << 20))
low = free()
while True:  # 2 MB more each time, until the text has its place on the device
    before = free()
    same(read_mtx(text, device=True))
    if before - free() > 100:
        break
    rt.cudaFree(hog.pop())
print("read with", low, "to", before, "MB")
assert low < 128 < before
"""


def test_text_of_most_of_the_free_memory():
    r = subprocess.run([sys.executable, "-c", SCRIPT % str(ROOT / "rv-sparse_b200")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "read with" in r.stdout
