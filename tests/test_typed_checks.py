"""Argument checks of the FP64 and INT8 one-shot products give their codes
whether or not a device can be used, below and above the size from which the
device looks at the columns."""
import numpy as np
import pytest

from conftest import HAS_GPU
from rvsp import _lib as L
from rvsp import gen, spgemm_typed


@pytest.mark.parametrize("entries", [1 << 10, 1 << 16])
@pytest.mark.parametrize("kind,fault,status", [
    ("f64", "range", L.ERROR_INVALID_ARGUMENT), ("f64", "order", L.ERROR_INVALID_CSR),
    ("i8", "range", L.ERROR_INVALID_CSR), ("i8", "order", L.ERROR_INVALID_CSR),
    ("f64", None, L.ERROR_UNSUPPORTED_BACKEND), ("i8", None, L.ERROR_UNSUPPORTED_BACKEND)])
def test_codes_without_a_device(kind, fault, status, entries):
    if HAS_GPU and fault is None:
        pytest.skip("a device is there")
    M = gen.uniform_rows(entries // 8, entries // 8, 4, 3)
    ci, v = M.col_idx.copy(), np.ones(M.nnz, np.float64 if kind == "f64" else np.int8)
    if fault == "range":
        ci[-1] = M.cols
    elif fault == "order":
        ci[4:6] = ci[4:6][::-1].copy()
    good = (M.rows, M.cols, M.row_ptr, M.col_idx, v)
    with pytest.raises(L.RvspError) as e:
        spgemm_typed(good, good[:3] + (ci, v), kind)
    assert e.value.status == status
