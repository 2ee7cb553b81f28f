"""Stripe rows where C, memory or the index range end (csrc/cuda/k_stripe.cu).

A call whose row pointers do not give a heavy row its analysed length reports
it and leaves that row alone, whether the row grew or shrank, in a fill and in
a numeric-only repeat.  B may have more than 2^30 entries.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from rvsp import CSR, DeviceCSR, RvspError
from rvsp import _lib as L

pytestmark = pytest.mark.gpu

SENTINEL = 123.0


def _stream():
    import torch
    return C.c_void_p(torch.cuda.current_stream().cuda_stream or 1)


def _rows(rng, lengths, cols):
    out = [np.sort(rng.choice(cols, size=min(n, cols), replace=False)) for n in lengths]
    rp = np.concatenate([[0], np.cumsum([x.size for x in out])])
    ci = np.concatenate(out)
    return CSR(len(out), cols, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))


def _operands(b_cols, seed, rows=(0, 3, 200, 40, 1, 600, 90, 2, 450)):
    rng = np.random.default_rng(seed)
    B = _rows(rng, rng.choice([0, 1, 5, 33, 70], size=800), b_cols)
    return _rows(rng, rows, 800), B


class _Plan:
    """A plan with the analysis of A * B and the product's arrays."""

    def __init__(self, A, B):
        import torch
        self.lib = L.load()
        self.a, self.b = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
        self.h = C.c_void_p()
        L.check(self.lib.rvsp_cuda_plan_create(C.byref(self.h)), "plan")
        self.rp = torch.zeros(A.rows + 1, dtype=torch.int32, device="cuda")

    def analyse(self):
        a, b, total = self.a, self.b, C.c_int64()
        L.check(self.lib.rvsp_cuda_symbolic(
            self.h, _stream(), a.rows, b.rows, b.cols, a.row_ptr.data_ptr(),
            a.col_idx.data_ptr(), b.row_ptr.data_ptr(), b.col_idx.data_ptr(),
            self.rp.data_ptr(), C.byref(total)), "symbolic")
        return total.value

    def numeric(self, rp, ci, cv, fill):
        import torch
        a, b = self.a, self.b
        size = max(self.lib.rvsp_cuda_numeric_workspace_bytes(self.h), 256)
        ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
        L.check(self.lib.rvsp_cuda_numeric(
            self.h, _stream(), a.row_ptr.data_ptr(), a.col_idx.data_ptr(), a.values.data_ptr(),
            b.row_ptr.data_ptr(), b.col_idx.data_ptr(), b.values.data_ptr(), rp.data_ptr(),
            ci.data_ptr(), cv.data_ptr(), fill, ws.data_ptr(), size), "numeric")
        L.check(self.lib.rvsp_cuda_plan_status(self.h, _stream()), "status")

    def close(self):
        self.lib.rvsp_cuda_plan_destroy(self.h)


@pytest.mark.parametrize("fill", [1, 0])
@pytest.mark.parametrize("more", [5, -5])
@pytest.mark.parametrize("b_cols", [3000, 60000])
def test_row_pointers_of_another_length(b_cols, more, fill):
    import torch
    A, B = _operands(b_cols, b_cols + more)
    rp, ci, cv, _ = oracle.spgemm(A, B)
    n = np.diff(rp)
    row = int(np.nonzero(n > 1024)[0][1])
    p = _Plan(A, B)
    assert p.analyse() == ci.size
    # C with the heavy row `more` entries longer, the rows after it moved
    rp2 = rp.copy()
    rp2[row + 1:] += more
    at = np.arange(ci.size) + np.where(np.arange(ci.size) >= rp[row + 1], more, 0)
    other = np.ones(ci.size, bool)
    other[rp[row]:rp[row + 1]] = False
    want_ci = np.full(ci.size + more, 7, np.int32)
    want_cv = np.full(ci.size + more, SENTINEL, np.float32)
    want_ci[at[other]], want_cv[at[other]] = ci[other], cv[other]
    got_ci = torch.full((ci.size + more,), 7, dtype=torch.int32, device="cuda")
    if not fill:
        got_ci.copy_(torch.from_numpy(want_ci))
    got_cv = torch.full((ci.size + more,), SENTINEL, dtype=torch.float32, device="cuda")
    with pytest.raises(RvspError) as e:
        p.numeric(torch.from_numpy(rp2).cuda(), got_ci, got_cv, fill)
    assert e.value.status == L.ERROR_DEVICE
    assert np.array_equal(got_ci.cpu().numpy(), want_ci)
    assert np.array_equal(got_cv.cpu().numpy().view(np.uint32), want_cv.view(np.uint32))
    # the plan goes on with its own row pointers
    c_ci = torch.zeros(ci.size, dtype=torch.int32, device="cuda")
    c_cv = torch.zeros(ci.size, dtype=torch.float32, device="cuda")
    for f in (1, 0):
        p.numeric(p.rp, c_ci, c_cv, f)
        assert np.array_equal(c_ci.cpu().numpy(), ci)
        assert np.array_equal(c_cv.cpu().numpy().view(np.uint32), cv.view(np.uint32))
    p.close()


def test_b_of_more_than_2_30_entries():
    import torch
    rows, cols = 8300, 131072  # 1.09e9 entries
    k = [8200, 8299]
    a = np.array([0.75, -1.25], np.float32)
    p = _Plan(CSR(1, rows, np.array([0, 2]), np.array(k), a), CSR(1, 1, [0, 0], [], []))
    g = torch.Generator(device="cuda").manual_seed(1)
    p.b = DeviceCSR(rows, cols,
                    torch.arange(rows + 1, dtype=torch.int32, device="cuda") * cols,
                    torch.arange(cols, dtype=torch.int32, device="cuda").repeat(rows),
                    torch.rand(rows * cols, generator=g, device="cuda"))
    assert p.analyse() == cols
    ci = torch.zeros(cols, dtype=torch.int32, device="cuda")
    cv = torch.zeros(cols, dtype=torch.float32, device="cuda")
    b = p.b.values.view(rows, cols)
    want = float(a[0]) * b[k[0]] + float(a[1]) * b[k[1]]
    for fill in (1, 0):
        p.numeric(p.rp, ci, cv, fill)
        assert torch.equal(ci, torch.arange(cols, dtype=torch.int32, device="cuda"))
        assert torch.equal(cv, want)
    p.close()
