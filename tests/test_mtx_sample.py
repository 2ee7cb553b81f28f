"""Matrix Market texts that the device would hand back are not sent to it: the
call returns before it needs one (csrc/cuda/k_mtx.cu)."""
import ctypes as C

import numpy as np
import pytest

from conftest import HAS_GPU
from rvsp import _lib as L

ODD = {"signed": "+%d %d %g", "long": "%d %d %.50f", "inf": "%d %d inf", "small": "%d %d %ge-70"}
PLAIN = {"ordinary": "%d %d %.17g", "pattern": "%d %d", "few odd": "%d %d %g"}


def _parsed(fmt, lines, fields, odd=()):
    rng = np.random.default_rng(1)
    out = []
    for i in range(lines):
        f = ODD["signed"] if i in odd else fmt
        v = (i % 100 + 1, i // 100 + 1, rng.uniform(-1, 1))
        out.append(f % v[:f.count("%")])
    text = ("\n".join(out) + "\n").encode()
    lib = L.load()
    col, val, nnz, parsed = C.c_void_p(), C.c_void_p(), C.c_int32(), C.c_int(7)
    rows = lines // 100 + 100
    st = lib.rvsp_cuda_mtx_to_csr(None, text, len(text), fields, lines, rows, rows, 0,
                                  C.c_void_p(16), C.byref(col), C.byref(val), C.byref(nnz),
                                  C.byref(parsed))
    return st, parsed.value


@pytest.mark.parametrize("lines", [1500, 4000, 40000])
@pytest.mark.parametrize("kind", sorted(ODD))
def test_odd_texts_need_no_device(kind, lines):
    assert _parsed(ODD[kind], lines, 3) == (L.SUCCESS, 0)


@pytest.mark.skipif(HAS_GPU, reason="a device is there")
@pytest.mark.parametrize("lines", [1500, 40000])
@pytest.mark.parametrize("kind", sorted(PLAIN))
def test_other_texts_go_to_the_device(kind, lines):
    odd = range(0, lines, 20) if kind == "few odd" else ()
    st, parsed = _parsed(PLAIN[kind], lines, 2 if kind == "pattern" else 3, odd)
    assert st != L.SUCCESS and parsed == 0
