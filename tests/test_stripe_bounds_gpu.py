"""Stripe rows where C, memory or the index range end (csrc/cuda/k_stripe.cu).

A call whose row pointers do not give a heavy row its analysed length reports
it and leaves that row alone, whether the row grew or shrank, in a fill and in
a numeric-only repeat.  B may have more than 2^30 entries.  All that the rows
keep counts against their memory, and rows without room give the same results
by the block-per-row kernels, on the plain and on the learned path, as do rows
too few for stripes to pay.
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
        L.check(self.lib.rvsp_cuda_plan_set_stripes(self.h, 2), "always")
        self.rp = torch.zeros(A.rows + 1, dtype=torch.int32, device="cuda")

    def learned(self, model, scale=1.0):
        a, b, total = self.a, self.b, C.c_int64()
        L.check(self.lib.rvsp_cuda_learned_symbolic(
            self.h, model.h, _stream(), a.rows, b.rows, b.cols, a.row_ptr.data_ptr(),
            a.col_idx.data_ptr(), a.values.data_ptr(), a.nnz, b.row_ptr.data_ptr(),
            b.col_idx.data_ptr(), b.values.data_ptr(), b.nnz, C.c_float(scale),
            self.rp.data_ptr(), C.byref(total)), "learned")
        return total.value

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


def test_memory_counts_items_and_offsets():
    # 400,000 rows of three B rows of 400 columns each: 56 MB of bitmaps and
    # 270 MB of items and offsets
    import torch
    rng = np.random.default_rng(3)
    n = 400000
    B = _rows(rng, [400] * 50, 1100)
    picks = np.sort(rng.permuted(np.tile(np.arange(50), (n, 1)), axis=1)[:, :3], axis=1)
    A = CSR(n, 50, np.arange(0, 3 * n + 1, 3), picks.reshape(-1), np.ones(3 * n, np.float32))
    p, q = _Plan(A, B), _Plan(A, B)
    for plan in (p, q):  # all else that an analysis takes
        L.check(plan.lib.rvsp_cuda_plan_set_stripe_memory(plan.h, 0), "set_stripe_memory")
        nnz = plan.analyse()

    def grows(plan, limit):
        L.check(plan.lib.rvsp_cuda_plan_set_stripe_memory(plan.h, limit), "set_stripe_memory")
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        assert plan.analyse() == nnz
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]

    assert grows(p, 200 << 20) <= 200 << 20
    assert grows(q, 400 << 20) > 200 << 20
    p.close()
    q.close()


@pytest.mark.parametrize("b_cols", [1100, 40000])
@pytest.mark.parametrize("path", ["plain", "learned"])
def test_rows_without_room(path, b_cols):
    import torch
    from rvsp.learn import RowModel, weights_for
    A, B = _operands(b_cols, b_cols + 1)
    rp, ci, cv, _ = oracle.spgemm(A, B)
    assert (np.diff(rp) > 1024).sum() > 1
    p = _Plan(A, B)
    model = RowModel(path=weights_for("rmat"))
    # (limit, policy): no room, room, no room, never, where it pays (not here)
    for limit, policy in ((0, 2), (1 << 30, 2), (0, 2), (1 << 30, 1), (1 << 30, 0)):
        L.check(p.lib.rvsp_cuda_plan_set_stripes(p.h, policy), "set_stripes")
        L.check(p.lib.rvsp_cuda_plan_set_stripe_memory(p.h, limit), "set_stripe_memory")
        assert (p.learned(model) if path == "learned" else p.analyse()) == ci.size
        assert np.array_equal(p.rp.cpu().numpy(), rp)
        if path == "learned" and policy == 2:
            # without room they are redone by the plain passes
            assert (p.lib.rvsp_cuda_plan_overflow_rows(p.h) >= 2) == (limit == 0)
        c_ci = torch.zeros(ci.size, dtype=torch.int32, device="cuda")
        c_cv = torch.zeros(ci.size, dtype=torch.float32, device="cuda")
        for fill in (1, 0):
            p.numeric(p.rp, c_ci, c_cv, fill)
            assert np.array_equal(c_ci.cpu().numpy(), ci)
            assert np.array_equal(c_cv.cpu().numpy().view(np.uint32), cv.view(np.uint32))
    p.close()


def test_more_parts_of_rows_than_the_count_holds():
    # 600 rows of 63 parts of the count each, of which 520 rows' fit and leave 8
    # places; all rows have one structure and values a power of two apart, so
    # one row gives all
    import torch
    rng = np.random.default_rng(4)
    rows, inner, cols = 600, 4096, 4096
    B = _rows(rng, [1000] * inner, cols)
    one = CSR(1, inner, [0, inner], np.arange(inner),
              rng.uniform(-1, 1, inner).astype(np.float32))
    rp, ci, cv, ops = oracle.spgemm(one, B)
    assert -(-ops[0] // 65536) == 63
    p = _Plan(one, B)
    scale = torch.exp2(torch.randint(-3, 4, (rows, 1), device="cuda").float())
    p.a = DeviceCSR(rows, inner, torch.arange(rows + 1, dtype=torch.int32, device="cuda") * inner,
                    torch.arange(inner, dtype=torch.int32, device="cuda").repeat(rows),
                    (scale * torch.from_numpy(one.values).cuda()).reshape(-1).contiguous())
    p.rp = torch.zeros(rows + 1, dtype=torch.int32, device="cuda")
    assert p.analyse() == rows * ci.size
    c_ci = torch.zeros(rows * ci.size, dtype=torch.int32, device="cuda")
    c_cv = torch.zeros(rows * ci.size, dtype=torch.float32, device="cuda")
    for fill in (1, 0):
        p.numeric(p.rp, c_ci, c_cv, fill)
        assert torch.equal(c_ci.view(rows, -1),
                           torch.from_numpy(ci).cuda().expand(rows, -1))
        assert torch.equal(c_cv.view(rows, -1), scale * torch.from_numpy(cv).cuda())
    p.close()
