"""Host arrays that rvsp_csr_destroy keeps for later one-shot results
(csrc/host/alloc.c): none in a process that makes no products, and all of them
back at the end of the last thread that made some, or when asked for."""
import ctypes as C
import threading

import numpy as np
import pytest

from rvsp import _lib as L
from rvsp import gen, spgemm_typed


class _MallInfo(C.Structure):
    _fields_ = [(n, C.c_size_t) for n in ("arena", "ordblks", "smblks", "hblks", "hblkhd",
                                          "usmblks", "fsmblks", "uordblks", "fordblks",
                                          "keepcost")]


def _in_use():
    """Bytes of live malloc blocks."""
    f = C.CDLL(None).mallinfo2
    f.restype = _MallInfo
    m = f()
    return m.uordblks + m.hblkhd


def _make_and_destroy(lib, size=8 << 20):
    """A matrix that owns two large malloc blocks."""
    malloc = C.CDLL(None).malloc
    malloc.restype, malloc.argtypes = C.c_void_p, [C.c_size_t]
    m = L.CsrMatrix()
    m.col_idx, m.values, m.owns_data = malloc(size), malloc(size), 1
    lib.rvsp_csr_destroy(C.byref(m))


def test_none_without_products():
    lib = L.load()
    lib.rvsp_release_kept_results()
    before = _in_use()
    _make_and_destroy(lib)
    assert _in_use() - before < 1 << 20


def _product():
    M = gen.uniform_rows(20000, 20000, 8, 1)
    a = (M.rows, M.cols, M.row_ptr, M.col_idx, M.values.astype(np.float64))
    return spgemm_typed(a, a, "f64")


@pytest.mark.gpu
def test_kept_until_the_last_thread_ends():
    lib = L.load()
    made, go = threading.Barrier(3), [threading.Event(), threading.Event()]

    def work(i):
        _product()
        made.wait()
        go[i].wait()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    made.wait()
    lib.rvsp_release_kept_results()
    before = _in_use()
    _make_and_destroy(lib)
    assert _in_use() - before > 15 << 20
    lib.rvsp_release_kept_results()
    assert _in_use() - before < 1 << 20
    _make_and_destroy(lib)
    go[0].set()
    threads[0].join()
    assert _in_use() - before > 15 << 20  # the other thread lives
    go[1].set()
    threads[1].join()
    # (this thread may have made products of its own in earlier tests)
    if _in_use() - before > 1 << 20:
        lib.rvsp_release_kept_results()
    assert _in_use() - before < 1 << 20
