"""Rows on either side of the merge classes' bounds (csrc/cuda/kernels.cuh,
k_merge.cu) in a matrix large enough for them: A rows of up to 16 nonzeros with
128 to 272 products, in consecutive columns or apart (where the bound is 256
or 128); warps of rows of at most four lists, of eight, and of both; rows of C
that follow one another in a warp and rows that do not."""
import numpy as np
import pytest

from oracle import oracle
from rvsp import CSR, Descriptor, DeviceCSR
from rvsp import _lib as L

pytestmark = pytest.mark.gpu

ZONE = 512                      # rows of B of one length
LENGTHS = [0, 1, 8, 9, 16, 17]
B_COLS = 4096


def _b(rng):
    """Rows of each zone's length, in a window of 60 columns that moves along."""
    cols = []
    for z, n in enumerate(LENGTHS):
        for i in range(ZONE):
            cols.append(np.sort(rng.choice(60, n, replace=False)) + 7 * i % (B_COLS - 60))
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])])
    ci = np.concatenate(cols).astype(np.int32)
    return CSR(len(cols), B_COLS, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))


def _row(rng, zone, n, near):
    at = int(rng.integers(ZONE - 16))
    c = np.arange(n) if near else np.arange(n) * 31 - at
    return zone * ZONE + at + c


def _matrix(pick, rows, seed):
    """A with pick(i) = (zone, nonzeros, near) for row i."""
    rng = np.random.default_rng(seed)
    out = [_row(rng, *pick(i)) for i in range(rows)]
    rp = np.concatenate([[0], np.cumsum([c.size for c in out])])
    ci = np.concatenate(out).astype(np.int32)
    A = CSR(rows, ZONE * len(LENGTHS), rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))
    return A, _b(rng)


EDGES = [(2, 16, False), (2, 16, True), (3, 15, False), (3, 15, True), (3, 16, True),
         (4, 16, True), (4, 16, False), (5, 15, True), (5, 16, True), (0, 3, True)]

PICKS = {
    # every bound, side by side
    "edges": lambda i: EDGES[i % len(EDGES)],
    "edges apart": lambda i: EDGES[i % len(EDGES)][:2] + (False,),
    # whole warps of at most four lists, of eight, and mixed lanes
    "lists": lambda i: (2, (3 if i // 32 % 3 == 0 else 7 if i // 32 % 3 == 1 else 2 + 6 * (i % 2)),
                        i % 2 == 0),
    # runs of merge rows broken by single rows of another class
    "broken runs": lambda i: (5, 16, False) if i % 101 == 50 else (1, 4, True),
    # no rows but merge rows: one round trip, C in one run
    "merge only": lambda i: (4, 16, True) if i % 2 else (2, 8, False),
}


@pytest.mark.parametrize("algo", [L.ALGO_CUDA_PLAIN, L.ALGO_CUDA_LEARNED])
@pytest.mark.parametrize("kind", sorted(PICKS))
def test_bounds(kind, algo):
    import torch
    from rvsp.learn import RowModel, weights_for
    A, B = _matrix(PICKS[kind], 33003, len(kind))
    rp, ci, cv, _ = oracle.spgemm(A, B)
    a, b = DeviceCSR.from_host(A), DeviceCSR.from_host(B)
    with Descriptor(algo=algo, memory=L.MEM_DEVICE) as d:
        if algo == L.ALGO_CUDA_LEARNED:
            d.set_model(RowModel(path=weights_for("mixed")))
        size, nnz = d.work_estimation(a, b)
        c = DeviceCSR.empty(A.rows, B.cols, nnz)
        ws = torch.zeros(max(size, 1), dtype=torch.uint8, device="cuda")
        for _ in range(3):
            d.compute(a, b, c, ws)
            d.synchronize()
            got = c.to_host(ci.size)
            assert np.array_equal(got.row_ptr, rp)
            assert np.array_equal(got.col_idx, ci)
            assert np.array_equal(got.values.view(np.uint32), cv.view(np.uint32))
        if algo == L.ALGO_CUDA_PLAIN:
            sym, _ = d.class_counts()
            merged = sym["m4"] + sym["m8"] + sym["m16"]
            if kind == "edges":  # many in consecutive columns: to 256 products
                assert merged == sum(i % 10 < 8 for i in range(A.rows))
            elif kind == "edges apart":  # to 128
                assert merged == sum(i % 10 < 2 for i in range(A.rows))
            else:
                assert merged >= A.rows * 0.98
