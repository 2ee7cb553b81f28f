"""The calls whose time matters to a user of this library.

Each case is one call (or the short sequence of calls) that a program makes
through the public API of `rvsp`, the ctypes mirror of the C API:

  oneshot   rvsp_spgemm_csr on host arrays: the drop-in call, in and out of
            host memory, FP32, FP64 or INT8 -> INT32
  product   a descriptor on device arrays: work_estimation, C allocated, the
            first compute (columns and values)
  repeat    a descriptor that has C's structure: one numeric-only compute
  batch     many uneven products in one batch: one numeric-only compute
  mtx       Matrix Market text to canonical CSR on the device

Matrix families: rows of Poisson or fixed length with uniform columns, the 2D
5-point Laplacian, the 3D 27-point stencil (both on grids that need not be
square) and R-MAT graphs of average degree 16.

listed() names twelve cases, draw(rng) gives others of the same ranges,
prepare / run / work / exact describe one.  The sparsity of a case's operands
is its own; the seed draws their values.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "rv-sparse_b200"))

from rvsp import CSR, Batch, Descriptor, DeviceCSR, read_mtx, spgemm_csr, spgemm_typed  # noqa: E402
from rvsp import _lib as L  # noqa: E402
from rvsp.learn import RowModel, weights_for  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # A small product of a program written for the CPU library: all call
        # overhead and launches.
        {"name": "oneshot_small_f32", "kind": "oneshot", "dtype": "f32", "family": "poisson",
         "rows": 200, "inner": 300, "cols": 250, "mean": 4.0},
        # A double-precision PDE matrix squared, host arrays in and out.
        {"name": "oneshot_laplace_f64", "kind": "oneshot", "dtype": "f64", "family": "laplace",
         "gx": 181, "gy": 181},
        # A quantised rectangular product, host arrays in and out.
        {"name": "oneshot_rect_i8", "kind": "oneshot", "dtype": "i8", "family": "poisson",
         "rows": 20011, "inner": 30011, "cols": 10007, "mean": 11.0},
        # An ordinary product of short uniform rows, once: 4096^2, 16 a row.
        {"name": "product_uniform_4096", "kind": "product", "algo": "plain", "family": "uniform",
         "rows": 4096, "inner": 4096, "cols": 4096, "k": 16},
        # A mesh operator squared, once (multigrid setup): 1024^2 Laplacian.
        {"name": "product_laplace_1024", "kind": "product", "algo": "plain", "family": "laplace",
         "gx": 1024, "gy": 1024},
        # The same in 3D with wide rows, on a grid that is no power of two.
        {"name": "product_stencil_ragged", "kind": "product", "algo": "plain", "family": "stencil",
         "gx": 127, "gy": 90, "gz": 113},
        # A time stepper's repeat: values changed, structure kept, 128^3.
        {"name": "repeat_stencil_128", "kind": "repeat", "algo": "plain", "family": "stencil",
         "gx": 128, "gy": 128, "gz": 128},
        # A graph squared (paths of length two), skewed rows with hubs.
        {"name": "product_rmat_16", "kind": "product", "algo": "plain", "family": "rmat",
         "scale": 16},
        # A smaller graph through the learned algorithm.
        {"name": "product_rmat_14_learned", "kind": "product", "algo": "learned",
         "family": "rmat", "scale": 14},
        # A reweighted graph: values changed, structure kept.
        {"name": "repeat_rmat_15", "kind": "repeat", "algo": "plain", "family": "rmat",
         "scale": 15},
        # Many independent products of uneven sizes, values redrawn.
        {"name": "batch_48", "kind": "batch", "count": 48, "n_lo": 256, "n_hi": 65536},
        # A symmetric matrix file's text, read onto the device.
        {"name": "mtx_text", "kind": "mtx", "gx": 512, "gy": 300},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["oneshot", "oneshot", "product", "product", "product", "product",
                       "repeat", "repeat", "batch", "mtx"])
    if kind == "mtx":
        return {"kind": kind, "gx": _log_int(rng, 16, 512), "gy": _log_int(rng, 16, 300)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 48), "n_lo": 256,
                "n_hi": _log_int(rng, 1024, 65536)}
    case = {"kind": kind}
    if kind == "oneshot":
        case["dtype"] = rng.choice(["f32", "f64", "i8"])
        case["family"] = rng.choice(["poisson", "poisson", "laplace"])
        top = 20000
    else:
        case["algo"] = rng.choice(["plain", "plain", "learned"]) if kind == "product" else "plain"
        case["family"] = rng.choice(["poisson", "uniform", "laplace", "stencil", "rmat", "rmat"])
        top = 100000
    if case["family"] == "poisson":
        case.update(rows=_log_int(rng, 64, top), inner=_log_int(rng, 64, top),
                    cols=_log_int(rng, 64, top), mean=round(rng.uniform(2.0, 16.0), 2))
    elif case["family"] == "uniform":
        case.update(rows=_log_int(rng, 64, top), inner=_log_int(rng, 64, top),
                    cols=_log_int(rng, 64, top), k=rng.randint(1, 24))
    elif case["family"] == "laplace":
        g = 181 if kind == "oneshot" else 1024
        case.update(gx=_log_int(rng, 8, g), gy=_log_int(rng, 8, g))
    elif case["family"] == "stencil":
        case.update(gx=_log_int(rng, 8, 128), gy=_log_int(rng, 8, 120), gz=_log_int(rng, 8, 110))
    else:
        case["scale"] = rng.randint(10, 15)
    return case


# ---- inputs -----------------------------------------------------------------
# A matrix here is (rows, cols, row_ptr, col_idx): int32 tensors on the GPU.

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _row_ptr(lengths):
    rp = torch.zeros(lengths.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lengths, 0, out=rp[1:])
    return rp.to(torch.int32)


def _from_keys(rows, cols, key):
    """CSR of the distinct row * cols + col keys."""
    key = torch.unique(key)
    r = key // cols
    return (rows, cols, _row_ptr(torch.bincount(r, minlength=rows)),
            (key - r * cols).to(torch.int32))


def _poisson(rows, cols, mean, g):
    n = torch.poisson(torch.full((rows,), float(mean), device=DEV), generator=g).to(torch.int64)
    n.clamp_(max=cols)
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), n)
    c = torch.randint(0, cols, (r.numel(),), generator=g, device=DEV)
    return _from_keys(rows, cols, r * cols + c)


def _uniform(rows, cols, k, g):
    """k distinct ascending columns in every row."""
    k = min(k, cols)
    c = torch.randint(0, cols - k + 1, (rows, k), generator=g, device=DEV)
    c = c.sort(dim=1).values + torch.arange(k, device=DEV)
    return rows, cols, _row_ptr(torch.full((rows,), k, device=DEV)), c.reshape(-1).to(torch.int32)


def _grid(dims, reach):
    """Neighbours of every point of a row-major grid: all offsets of {-1, 0,
    1}^d with at most `reach` non-zero parts."""
    n = math.prod(dims)
    strides = [math.prod(dims[i + 1:]) for i in range(len(dims))]
    idx = torch.arange(n, device=DEV)
    coord = [(idx // s) % d for s, d in zip(strides, dims)]
    oks, deltas = [], []
    for m in range(3 ** len(dims)):
        o = [m // 3 ** (len(dims) - 1 - i) % 3 - 1 for i in range(len(dims))]
        if sum(map(abs, o)) > reach:
            continue
        ok = torch.ones(n, dtype=torch.bool, device=DEV)
        for x, d, step in zip(coord, dims, o):
            if step:
                ok &= (x + step >= 0) & (x + step < d)
        oks.append(ok)
        deltas.append(sum(a * b for a, b in zip(o, strides)))
    ok = torch.stack(oks, dim=1)
    col = idx[:, None] + torch.tensor(deltas, device=DEV)
    return n, n, _row_ptr(ok.sum(dim=1)), col[ok].to(torch.int32)


def _rmat(scale, g, degree=16):
    n = 1 << scale
    r = torch.zeros(degree * n, dtype=torch.int64, device=DEV)
    c = torch.zeros_like(r)
    for _ in range(scale):
        u = torch.rand(r.numel(), generator=g, device=DEV)
        r = 2 * r + (u >= 0.76)
        c = 2 * c + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    return _from_keys(n, n, r * n + c)


def _structure(case, g):
    """(A, B) with B None where the product is A * A."""
    f = case["family"]
    if f == "poisson":
        return (_poisson(case["rows"], case["inner"], case["mean"], g),
                _poisson(case["inner"], case["cols"], case["mean"], g))
    if f == "uniform":
        return (_uniform(case["rows"], case["inner"], case["k"], g),
                _uniform(case["inner"], case["cols"], case["k"], g))
    if f == "laplace":
        return _grid((case["gy"], case["gx"]), 1), None
    if f == "stencil":
        return _grid((case["gz"], case["gy"], case["gx"]), 3), None
    return _rmat(case["scale"], g), None


def _values(case, M, g):
    """Mesh operators: a diagonal of 4 or 26 and neighbours of -1, each
    perturbed by U[-0.01, 0.01]; graphs: U(0, 1]; others U[-1, 1]; INT8:
    quantised positive weights, 1 .. 127 (no sum is zero, so C's structure
    does not hang on the values)."""
    n = M[3].numel()
    if case.get("dtype") == "i8":
        return torch.randint(1, 128, (n,), generator=g, device=DEV).to(torch.int8)
    wide = torch.float64 if case.get("dtype") == "f64" else torch.float32
    u = torch.rand(n, generator=g, device=DEV, dtype=wide)
    if case["family"] in ("laplace", "stencil"):
        r = torch.repeat_interleave(torch.arange(M[0], device=DEV), M[2].diff())
        base = torch.where(r == M[3], 4.0 if case["family"] == "laplace" else 26.0, -1.0)
        return (base.to(wide) + (u * 0.02 - 0.01)).contiguous()
    return 1.0 - u if case["family"] == "rmat" else 2.0 * u - 1.0


def _operands(case, seed, structure=1):
    """((A, values), (B, values)); the two are one object where B is A."""
    A, B = _structure(case, _gen(structure))
    g = _gen(seed)
    a = (A, _values(case, A, g))
    return a, a if B is None else (B, _values(case, B, g))


def _batch_cases(case):
    r = np.random.default_rng(7)
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        out.append({"family": "poisson", "rows": n, "inner": n, "cols": n,
                    "mean": float(r.uniform(8.0, 32.0))})
    return out


def _batch_operands(case, seed):
    return [_operands(c, int(seed) * 1009 + i, i) for i, c in enumerate(_batch_cases(case))]


def _mtx_entries(case, seed):
    """The stored lower triangle of a symmetric mesh operator in file order,
    and its values as the text gives them."""
    g = _gen(seed)
    A = _grid((case["gy"], case["gx"]), 1)
    v = _values({"family": "laplace"}, A, g)
    r = torch.repeat_interleave(torch.arange(A[0], device=DEV), A[2].diff())
    keep = r >= A[3]
    text = ["%.6g" % x for x in v[keep].tolist()]
    return A[0], r[keep].cpu().numpy(), A[3][keep].cpu().numpy(), text


# ---- prepare and run ----------------------------------------------------------

def _device_csr(M, v):
    return DeviceCSR(M[0], M[1], M[2], M[3], v)


class _View:
    """Device memory that the library owns, for torch.as_tensor."""

    def __init__(self, ptr, n, keep):
        self.keep = keep
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "version": 3,
                                         "data": (ptr, False)}


def _new_c(d, A, B):
    n = max(d.c_nnz, 1)
    C = DeviceCSR(A.rows, B.cols, torch.empty(A.rows + 1, dtype=torch.int32, device=DEV),
                  torch.empty(n, dtype=torch.int32, device=DEV),
                  torch.empty(n, dtype=torch.float32, device=DEV))
    return C, torch.empty(max(d.ws_bytes, 1), dtype=torch.uint8, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mtx":
        n, r, c, text = _mtx_entries(case, seed)
        body = "\n".join("%d %d %s" % (i + 1, j + 1, t) for i, j, t in zip(r.tolist(), c.tolist(), text))
        return {"kind": kind, "text": ("%%%%MatrixMarket matrix coordinate real symmetric\n%d %d %d\n%s\n"
                                       % (n, n, r.size, body)).encode()}
    if kind == "batch":
        ops = [(_device_csr(*a), _device_csr(*b)) for a, b in _batch_operands(case, seed)]
        torch.cuda.synchronize()
        # repeats replay a captured graph: a stream of its own, not the legacy one
        stream = torch.cuda.Stream()
        b = Batch(memory=L.MEM_DEVICE, stream=stream, autotune=True)
        for x, y in ops:
            b.add(x, y)
        b.work_estimation()
        b.compute()
        out = []
        for i in range(len(ops)):
            c = b.view(i)
            out.append(torch.as_tensor(_View(c.values, c.nnz, b), device=DEV))
        return {"kind": kind, "batch": b, "stream": stream, "out": out}
    a, b = _operands(case, seed)
    if kind == "oneshot":
        def host(x):
            M, v = x
            return M[0], M[1], M[2].cpu().numpy(), M[3].cpu().numpy(), v.cpu().numpy()
        A = host(a)
        B = A if b is a else host(b)
        if case["dtype"] == "f32":
            A = CSR(*A)
            B = A if b is a else CSR(*B)
        return {"kind": kind, "dtype": case["dtype"], "A": A, "B": B}
    A = _device_csr(*a)
    B = A if b is a else _device_csr(*b)
    learned = case["algo"] == "learned"
    d = Descriptor(algo=L.ALGO_CUDA_LEARNED if learned else L.ALGO_CUDA_PLAIN,
                   memory=L.MEM_DEVICE, stream=torch.cuda.current_stream())
    if learned:
        d.set_model(RowModel(path=weights_for(case["family"])))
    state = {"kind": kind, "A": A, "B": B, "d": d}
    if kind == "repeat":
        d.work_estimation(A, B)
        state["C"], state["ws"] = _new_c(d, A, B)
        d.compute(A, B, state["C"], state["ws"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "mtx":
        M = read_mtx(state["text"], device=True)
        return M.row_ptr, M.col_idx, M.values
    if kind == "batch":
        state["batch"].compute()
        return state["out"]
    A, B = state["A"], state["B"]
    if kind == "oneshot":
        if state["dtype"] == "f32":
            C = spgemm_csr(A, B)
            return C.row_ptr, C.col_idx, C.values
        return spgemm_typed(A, B, state["dtype"])
    d = state["d"]
    if kind == "product":
        d.work_estimation(A, B)
        C, ws = _new_c(d, A, B)
        d.compute(A, B, C, ws)
    else:
        C = state["C"]
        d.compute(A, B, C, state["ws"])
    return C.row_ptr, C.col_idx[:d.c_nnz], C.values[:d.c_nnz]


# ---- the same in 64 bits, and what a pass cannot do without -------------------

def _multiply(a, b, values=True, chunk=1 << 25):
    """(row_ptr, col_idx, float64 values, products) of A * B by expanding,
    sorting and summing the products of runs of rows; with values=False only
    C's entries are counted: (None, count, None, products)."""
    (rows, _, arp, aci), av = a
    (_, cols, brp, bci), bv = b
    arp, brp = arp.to(torch.int64), brp.to(torch.int64)
    blen = brp.diff()
    per = blen[aci.to(torch.int64)]
    cum = torch.zeros(per.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(per, 0, out=cum[1:])
    row_end = cum[arp].cpu().numpy()
    arow = torch.repeat_interleave(torch.arange(rows, device=DEV), arp.diff())
    counts, cis, vs, total, r0 = [], [], [], 0, 0
    while r0 < rows:
        r1 = int(np.searchsorted(row_end, row_end[r0] + chunk, side="right")) - 1
        r1 = min(max(r1, r0 + 1), rows)
        p0, p1 = int(arp[r0]), int(arp[r1])
        n = per[p0:p1]
        which = torch.repeat_interleave(torch.arange(p0, p1, device=DEV), n)
        m = which.numel()
        e = torch.arange(m, device=DEV) - (cum[which] - cum[p0]) + brp[aci[which].to(torch.int64)]
        key = (arow[which] - r0) * cols + bci[e].to(torch.int64)
        if values:
            prod = av[which].to(torch.float64) * bv[e].to(torch.float64)
            uniq, inv = torch.unique(key, return_inverse=True)
            out = torch.zeros(uniq.numel(), dtype=torch.float64, device=DEV)
            out.scatter_add_(0, inv, prod)
            r = uniq // cols
            cis.append((uniq - r * cols).to(torch.int32))
            vs.append(out)
            counts.append(torch.bincount(r, minlength=r1 - r0))
        else:
            total += int(torch.unique(key).numel())
        r0 = r1
    products = int(row_end[-1])
    if not values:
        return None, total, None, products
    return _row_ptr(torch.cat(counts)), torch.cat(cis), torch.cat(vs), products


def _without_zeros(rp, ci, v):
    """The FP64 and INT8 products do not store sums of zero."""
    keep = v != 0
    before = torch.zeros(v.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(keep, 0, out=before[1:])
    return before[rp.to(torch.int64)].to(torch.int32), ci[keep], v[keep]


def exact(case, seed):
    kind = case["kind"]
    if kind == "mtx":
        n, r, c, text = _mtx_entries(case, seed)
        v = np.array([float(t) for t in text])
        off = r != c
        key = np.concatenate([r * n + c, c[off].astype(np.int64) * n + r[off]])
        v = np.concatenate([v, v[off]])
        order = np.argsort(key, kind="stable")
        key = key[order]
        rp = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))])
        return rp.astype(np.int32), (key % n).astype(np.int32), v[order]
    if kind == "batch":
        return [_multiply(a, b)[2] for a, b in _batch_operands(case, seed)]
    rp, ci, v, _ = _multiply(*_operands(case, seed))
    if kind == "oneshot" and case["dtype"] != "f32":
        rp, ci, v = _without_zeros(rp, ci, v)
        if case["dtype"] == "i8":
            v = v.to(torch.int32)
    return rp, ci, v


def work(case):
    kind = case["kind"]
    if kind == "mtx":
        n, r, c, text = _mtx_entries(case, 0)
        # the text in, CSR out (every off-diagonal entry twice)
        chars = sum(len("%d %d %s\n" % (i + 1, j + 1, t)) for i, j, t in zip(r.tolist(), c.tolist(), text))
        return {"bytes": chars + 4 * (n + 1) + 8 * (2 * r.size - n), "flops": 0}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for a, b in _batch_operands(case, 0):
            _, nc, _, products = _multiply(a, b, values=False)
            na, nb = a[1].numel(), b[1].numel()
            total["bytes"] += 4 * (a[0][0] + b[0][0] + 2) + 8 * (na + nb) + 4 * nc
            total["flops"] += 2 * products
        return total
    a, b = _operands(case, 0)
    if case["family"] == "stencil":
        dims = (case["gx"], case["gy"], case["gz"])
        nc, products = math.prod(5 * d - 6 for d in dims), math.prod(9 * d - 10 for d in dims)
    else:
        _, nc, _, products = _multiply(a, b, values=False)
    dtype = case.get("dtype", "f32")
    vin, vout = {"f32": (4, 4), "f64": (8, 8), "i8": (1, 4)}[dtype]
    read = 4 * (a[0][0] + 1) + (4 + vin) * a[1].numel()
    if b is not a:
        read += 4 * (b[0][0] + 1) + (4 + vin) * b[1].numel()
    # a repeat writes C's values alone, the others its structure too
    write = vout * nc if kind == "repeat" else 4 * (a[0][0] + 1) + (4 + vout) * nc
    return {"bytes": read + write, "flops": 2 * products}
