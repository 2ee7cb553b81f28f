"""Bounds inside the row kernels: the register sorts of the warp fill (output
counts around each length, column counts around 2^22, from which keys are 64
bits wide), the steps of the map walk (B rows around 32 entries, mean lengths
around the six from which rows are stepped), more classes of translates than
one look-up brings to the host or one block's tables hold, and rows around the
64 entries from which a row of A is checked and counted by a warp.  Columns and
values are the oracle's, bit for bit, in the fill and in repeats."""
import numpy as np
import pytest

from oracle import oracle
from rvsp import CSR, Descriptor, DeviceCSR, gen
from rvsp import _lib as L

pytestmark = pytest.mark.gpu


def csr(cols, rows, rng):
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    ci = np.concatenate([np.asarray(r, np.int32) for r in rows])
    return CSR(len(rows), cols, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))


def check(A, B, shift=None, repeats=2):
    """a fill, then repeats with new values of A; the descriptor's reports"""
    import torch
    with Descriptor(algo=L.ALGO_CUDA_PLAIN, memory=L.MEM_DEVICE) as d:
        if shift is not None:
            d.set_shift_classes(shift)
        dA = DeviceCSR.from_host(A)
        dB = dA if B is A else DeviceCSR.from_host(B)
        ws_b, n = d.work_estimation(dA, dB)
        dC = DeviceCSR.empty(A.rows, B.cols, n)
        ws = torch.zeros(max(ws_b, 1), dtype=torch.uint8, device="cuda")
        for k in range(1 + repeats):
            A2 = A.with_values((A.values * np.float32(1 + k)).astype(np.float32))
            dA.values.copy_(torch.from_numpy(A2.values))
            torch.cuda.synchronize()
            d.compute(dA, dB, dC, ws)
            d.synchronize()
            rp, ci, cv, _ = oracle.spgemm(A2, A2 if B is A else B)
            got = dC.to_host(n)
            assert np.array_equal(got.row_ptr, rp), k
            assert np.array_equal(got.col_idx, ci), k
            assert np.array_equal(got.values.view(np.uint32), cv.view(np.uint32)), k
        return d.class_counts()[1], d.shift_rows()


@pytest.mark.parametrize("b_cols", [5000, 1 << 22, (1 << 22) + 1])
def test_warp_fill_sorts(b_cols):
    rng = np.random.default_rng(b_cols)
    # 8 rows of one column, then twice 160 rows of eight: all columns distinct,
    # the second 160 repeating the first
    cols = rng.choice(b_cols, size=8 + 160 * 8, replace=False)
    cols[0], cols[8] = 0, b_cols - 1
    cols = np.concatenate([np.unique(cols[:8]), np.unique(cols[8:])]) \
        if np.unique(cols).size == cols.size else np.unique(rng.choice(b_cols, 1288, False))
    rng.shuffle(cols)
    ones = [[c] for c in cols[:8]]
    eights = [np.sort(cols[8 + 8 * i:16 + 8 * i]) for i in range(160)]
    B = csr(b_cols, ones + eights + eights, rng)
    rows = []
    for m in (127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025):
        for twice in (False, True):
            pick = np.sort(rng.choice(160, m // 8, replace=False))
            a = np.concatenate([np.arange(m % 8), 8 + pick, 168 + pick if twice else []])
            rows.append(a.astype(np.int32))
    A = csr(B.rows, rows, rng)
    classes, _ = check(A, B)
    assert all(classes[f"w{w}"] > 0 for w in (256, 512, 1024)), classes


@pytest.mark.parametrize("lens", [(5,), (6,), (7,), (1, 11), (31, 33), (32,), (33, 64, 65), (3, 40)])
def test_map_walk_lengths(lens):
    rng = np.random.default_rng(sum(lens))
    B = csr(3000, [np.sort(rng.choice(3000, rng.choice(lens), replace=False))
                   for _ in range(1500)], rng)
    A = csr(1500, [np.sort(rng.choice(1500, n, replace=False))
                   for n in rng.integers(9, 21, 700)], rng)
    check(A, B, repeats=3)


@pytest.mark.parametrize("shift", [0, 2])
def test_many_patterns(shift):
    """400 classes of 20 consecutive translates each, of twelve nonzeros"""
    rng = np.random.default_rng(4)
    offs = [np.sort(rng.choice(400, 12, replace=False)) for _ in range(400)]
    n = 8000
    A = csr(n + 500, [i + offs[i // 20] for i in range(n)], rng)
    B = csr(n + 600, [i + np.arange(0, 90, 9) for i in range(n + 500)], rng)
    _, members = check(A, B, shift=shift)
    assert (members >= 400 * 19) == (shift == 2), members


@pytest.mark.parametrize("period", [1, 63, 300])
def test_interleaved_classes(period):
    """classes met in turn by the lanes of a warp and by the blocks"""
    rng = np.random.default_rng(period)
    offs = [np.sort(rng.choice(300, 10, replace=False)) for _ in range(period)]
    n = 9000
    A = csr(n + 300, [i + offs[i % period] for i in range(n)], rng)
    B = csr(n + 400, [i + np.arange(0, 80, 8) for i in range(n + 300)], rng)
    _, members = check(A, B, shift=2)
    assert members == n - period


@pytest.mark.parametrize("n", [31, 63, 64, 65, 257])
def test_rows_around_the_warp_bound(n):
    """A rows of n entries among short ones, four and eight lists a warp"""
    rng = np.random.default_rng(n)
    B = csr(2000, [np.sort(rng.choice(2000, 3, replace=False)) for _ in range(400)], rng)
    A = csr(400, [np.sort(rng.choice(400, n if i % 7 == 0 else i % 9, replace=False))
                  for i in range(500)], rng)
    check(A, B)
    check(A, gen.uniform_rows(400, 90, 1, 3))
