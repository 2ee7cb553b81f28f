"""The arrays of one-shot results own their memory: numpy resizes them in
place, and they outlive the call, the other arrays and the interpreter's
modules."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from rvsp import gen, spgemm_csr, spgemm_typed
from rvsp import _lib as L
from rvsp.api import _Owner

ROOT = Path(__file__).resolve().parents[1]


def _block(values):
    malloc = C.CDLL(None).malloc
    malloc.restype, malloc.argtypes = C.c_void_p, [C.c_size_t]
    p = malloc(values.nbytes)
    C.memmove(p, values.ctypes.data, values.nbytes)
    return p


def _owns(a):
    return a.flags.owndata and a.base is None and a.flags.writeable and a.flags.c_contiguous


@pytest.mark.parametrize("n", [1, 7, 1 << 20])
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.float64])
def test_array_over_a_block(dtype, n):
    owner = _Owner(L.load())
    want = np.arange(n).astype(dtype)
    m = L.CsrMatrix()
    m.values = p = _block(want)
    a = owner.take(m, "values", n, dtype)
    assert m.values is None and a.ctypes.data == p and _owns(a)
    assert a.dtype == dtype and np.array_equal(a, want)
    b = a[: n // 2 + 1].copy()  # arrays made later are numpy's own
    assert np.array_equal(b, want[: n // 2 + 1])
    a.resize(3 * n, refcheck=False)
    assert np.array_equal(a[:n], want) and not a[n:].any()
    a.resize(1, refcheck=False)
    assert a[0] == want[0] and _owns(a)


def test_without_the_hook():
    owner = _Owner(L.load())
    owner.make = None
    want = np.arange(5, dtype=np.float32)
    m = L.CsrMatrix()
    m.values, m.owns_data = _block(want), 1
    a = owner.take(m, "values", 5, np.float32)
    owner.lib.rvsp_csr_destroy(C.byref(m))
    assert _owns(a) and np.array_equal(a, want)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["f32", "f64", "i8"])
@pytest.mark.parametrize("n", [40, 30000])
def test_results(kind, n):
    M = gen.uniform_rows(n, n, 5, 2)
    if kind == "f32":
        R = spgemm_csr(M, M)
        out = [R.row_ptr, R.col_idx, R.values]
    else:
        v = np.ones(M.nnz, np.float64 if kind == "f64" else np.int8)
        a = (M.rows, M.cols, M.row_ptr, M.col_idx, v)
        out = list(spgemm_typed(a, a, kind))
    for x in out:
        assert _owns(x)
        was = x.copy()
        x.resize(x.size + 100, refcheck=False)
        assert np.array_equal(x[:-100], was) and not x[-100:].any()


@pytest.mark.gpu
def test_last_array_at_exit():
    code = ("import sys; sys.path[:0] = [%r]\n"
            "from rvsp import gen, spgemm_csr\n"
            "M = gen.uniform_rows(30000, 30000, 5, 2)\n"
            "sys.kept = spgemm_csr(M, M).values\n" % str(ROOT / "rv-sparse_b200"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and not r.stderr, r.stderr
