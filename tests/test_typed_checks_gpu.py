"""Argument checks of the FP64 and INT8 one-shot products on either side of the
size from which the columns are checked on the device: every planted fault
must give the status that the host's checks give in their order, and the
arrays of a result must outlive each other."""
import numpy as np
import pytest

from oracle import oracle
from rvsp import _lib as L
from rvsp import gen, spgemm_typed

pytestmark = pytest.mark.gpu

BAD_ARG, BAD_CSR = L.ERROR_INVALID_ARGUMENT, L.ERROR_INVALID_CSR


def operands(kind, entries):
    """A and B with entries/2 entries each, four a row"""
    n = entries // 8
    out = []
    for seed in (1, 2):
        M = gen.uniform_rows(n, n, 4, seed)
        v = np.arange(1, M.nnz + 1)
        v = v / 7.0 if kind == "f64" else (v % 5 + 1).astype(np.int8)
        out.append([M.rows, M.cols, M.row_ptr.copy(), M.col_idx.copy(), v])
    return out


def plant(M, fault):
    n, rp, ci = M[1], M[2], M[3]
    if fault == "range":
        ci[-1] = n
    elif fault == "negative":
        ci[0] = -1
    elif fault == "unsorted":
        ci[4:6] = ci[4:6][::-1].copy()
    elif fault == "duplicate":
        ci[5] = ci[4]
    elif fault == "row_ptr":
        rp[3] = rp[2] - 1
    elif fault == "first":
        rp[0] = 1


@pytest.mark.parametrize("entries", [(1 << 15) - 8, 1 << 15])
@pytest.mark.parametrize("kind", ["f64", "i8"])
@pytest.mark.parametrize("faults,f64,i8", [
    ([(0, "range")], BAD_ARG, BAD_CSR),
    ([(1, "negative")], BAD_ARG, BAD_CSR),
    ([(1, "unsorted")], BAD_CSR, BAD_CSR),
    ([(0, "duplicate")], BAD_CSR, BAD_CSR),
    ([(0, "unsorted"), (1, "range")], BAD_ARG, BAD_CSR),
    ([(1, "row_ptr")], BAD_ARG, BAD_CSR),
    ([(0, "first")], BAD_CSR, BAD_CSR),
])
def test_fault(kind, entries, faults, f64, i8):
    ops = operands(kind, entries)
    for which, fault in faults:
        plant(ops[which], fault)
    with pytest.raises(L.RvspError) as e:
        spgemm_typed(tuple(ops[0]), tuple(ops[1]), kind)
    assert e.value.status == (f64 if kind == "f64" else i8)


@pytest.mark.parametrize("entries", [(1 << 15) - 8, 1 << 15])
@pytest.mark.parametrize("kind", ["f64", "i8"])
def test_result_arrays_are_their_own(kind, entries):
    a, b = (tuple(M) for M in operands(kind, entries))
    want = oracle.spgemm_typed(a, b, kind)
    got = []
    for k in range(3):  # one array of each of three results is kept
        got.append(spgemm_typed(a, b, kind)[k])
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and g.tobytes() == w.tobytes()
        assert g.flags.writeable and g.flags.c_contiguous


def test_kept_result_memory_is_not_shared():
    """destroyed results give their arrays to later ones, live ones never"""
    a, b = (tuple(M) for M in operands("f64", 1 << 17))
    want = oracle.spgemm_typed(a, b, "f64")
    twice = oracle.spgemm_typed(a[:4] + (a[4] * 2,), b, "f64")
    for _ in range(3):
        live = spgemm_typed(a, b, "f64")
        other = spgemm_typed(a[:4] + (a[4] * 2,), b, "f64")
        for g, h, w, t in zip(live, other, want, twice):
            assert g.tobytes() == w.tobytes() and h.tobytes() == t.tobytes()
        del live, other
