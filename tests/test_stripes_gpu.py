"""Stripe rows (csrc/cuda/k_stripe.cu): heavy rows cut by columns.

Columns, values and numeric-only repeats are bit-identical to the oracle at
the widths where the accumulator, the bitmap words, the stripes and the class
itself end, for B rows from empty to longer than a step, for columns spread
evenly and bunched into a few words, and for signed zeros, infinities and NaN.
A C whose columns are not the product's is reported.
"""
import numpy as np
import pytest

from oracle import oracle
from rvsp import CSR, Descriptor, DeviceCSR, RvspError, gen
from rvsp import _lib as L

pytestmark = pytest.mark.gpu


def _rows(rng, lengths, cols, power):
    """CSR rows of the given lengths; columns bunch towards 0 as power grows."""
    out = []
    for n in lengths:
        c = np.unique((cols * rng.random(3 * n + 8) ** power).astype(np.int64))
        out.append(np.sort(rng.choice(c, size=min(n, c.size), replace=False)))
    rp = np.concatenate([[0], np.cumsum([x.size for x in out])])
    ci = np.concatenate(out)
    return CSR(len(out), cols, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))


def _operands(b_cols, power, seed):
    rng = np.random.default_rng(seed)
    inner = 900
    lengths = rng.choice([0, 1, 2, 5, 31, 32, 33, 70, 400], size=inner)
    B = _rows(rng, np.minimum(lengths, b_cols), b_cols, power)
    A = _rows(rng, [0, 1, 31, 32, 33, 64, 65, 200, 600, 899, 17, 128, 450], inner, 1.0)
    return A, B


def _device(A, B, algo=L.ALGO_CUDA_PLAIN):
    d = Descriptor(algo=algo, memory=L.MEM_DEVICE)
    a, b = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
    ws, nnz = d.work_estimation(a, b)
    c = DeviceCSR.empty(A.rows, B.cols, nnz)
    import torch
    return d, a, b, c, torch.zeros(max(ws, 1), dtype=torch.uint8, device="cuda")


def _same(c, A, B, what):
    rp, ci, cv, _ = oracle.spgemm(A, B)
    got = c.to_host(ci.size)
    assert np.array_equal(got.row_ptr, rp), what
    assert np.array_equal(got.col_idx, ci), what
    nan = np.isnan(cv)
    assert np.array_equal(np.isnan(got.values), nan), what
    assert np.array_equal(got.values.view(np.uint32)[~nan], cv.view(np.uint32)[~nan]), what


@pytest.mark.parametrize("power", [1.0, 6.0])
@pytest.mark.parametrize("b_cols", [1025, 2048, 4096, 4097, 20011, 65536, 65537, 131072, 131073])
def test_widths(b_cols, power):
    A, B = _operands(b_cols, power, b_cols)
    d, a, b, c, ws = _device(A, B)
    d.compute(a, b, c, ws)
    d.synchronize()
    _same(c, A, B, "fill")
    sym, num = d.class_counts()
    assert sym["b8192"] + sym["dense"] > 0
    assert power > 1 or num["b8192"] + num["dense"] > 0
    A2 = A.with_values((A.values * np.float32(-0.75)).astype(np.float32))
    a2 = DeviceCSR.from_host(A2)
    for _ in range(2):
        d.compute(a2, b, c, ws)
        d.synchronize()
        _same(c, A2, B, "repeat")
    d.close()


def test_values_that_cancel_or_are_not_finite():
    A, B = _operands(30000, 2.0, 5)
    rng = np.random.default_rng(6)
    for M in (A, B):
        M.values[:] = rng.choice(np.array([0.0, -0.0, 1.0, -1.0], np.float32), M.nnz)
    B.values[rng.choice(B.nnz, 40, replace=False)] = np.inf
    B.values[rng.choice(B.nnz, 20, replace=False)] = np.nan
    d, a, b, c, ws = _device(A, B)
    for what in ("fill", "repeat"):
        d.compute(a, b, c, ws)
        d.synchronize()
        _same(c, A, B, what)
    d.close()


@pytest.mark.parametrize("b_cols", [3000, 60000])
def test_columns_of_another_product_are_reported(b_cols):
    A, B = _operands(b_cols, 1.0, 7)
    d, a, b, c, ws = _device(A, B)
    d.compute(a, b, c, ws)
    d.synchronize()
    host = c.to_host(d.c_nnz)
    # a heavy row with columns missing: one of its columns moves up by one
    n = np.diff(host.row_ptr)
    row = int(np.nonzero((n > 1024) & (n < b_cols - 100))[0][0])
    p0, p1 = host.row_ptr[row], host.row_ptr[row + 1]
    gaps = np.nonzero(np.diff(host.col_idx[p0:p1]) > 1)[0]
    c.col_idx[int(p0 + gaps[gaps.size // 2])] += 1
    d.compute(a, b, c, ws)
    with pytest.raises(RvspError) as e:
        d.synchronize()
    assert e.value.status == L.ERROR_DEVICE
    c.col_idx[int(p0 + gaps[gaps.size // 2])] -= 1
    d.compute(a, b, c, ws)
    d.synchronize()
    _same(c, A, B, "after the error")
    d.close()


def test_hub_rows_and_every_row_heavy():
    # a graph whose hub row is many items, and a product all of whose rows
    # are of one stripe class (no row list)
    A = gen.rmat(13, 16, seed=3)
    d, a, b, c, ws = _device(A, A)
    d.compute(a, b, c, ws)
    d.synchronize()
    _same(c, A, A, "hub rows")
    d.close()
    rng = np.random.default_rng(9)
    X = _rows(rng, [300] * 40, 500, 1.0)
    Y = _rows(rng, [60] * 500, 40000, 1.0)
    d, a, b, c, ws = _device(X, Y)
    d.compute(a, b, c, ws)
    d.synchronize()
    _same(c, X, Y, "every row")
    assert d.class_counts()[1]["dense"] == 40
    d.close()
