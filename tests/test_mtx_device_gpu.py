"""Matrix Market text parsed on the device: every spelling of an index or a
value must give the bits that strtol / strtof give (the oracle's), whether the
device decides it, lists it for the host, or hands the text back; sizes on
either side of the bound from which the device parses, tokens on every offset
of its 4096-byte chunks."""
import numpy as np
import pytest

from oracle import oracle
from rvsp import read_mtx

pytestmark = pytest.mark.gpu
DEVICE_MIN = 8 << 10


def check(text, device=True):
    rows, cols, rp, ci, cv = oracle.mtx_to_csr(text)
    got = read_mtx(text, device=device)
    got = got.to_host() if device else got
    assert (got.rows, got.cols) == (rows, cols)
    assert np.array_equal(got.row_ptr, rp)
    assert np.array_equal(got.col_idx[:rp[-1]], ci)
    assert np.array_equal(got.values[:rp[-1]].view(np.uint32), cv.view(np.uint32))
    return rp[-1]


def text_of(values, n=5000, field="real", sym="general", sep="\n", declared=None):
    """one entry a value, all at different places"""
    k = np.arange(len(values))
    r, c = 1 + k % n, 1 + (k // n * 7 + k) % n
    return (f"%%MatrixMarket matrix coordinate {field} {sym}\n% x\n"
            f"{n} {n} {declared or len(values)}\n" +
            sep.join(f"{a} {b} {v}" for a, b, v in zip(r, c, values))).encode()


rng = np.random.default_rng(17)
BITS = rng.integers(0, 1 << 32, 40000, dtype=np.uint64).astype(np.uint32).view(np.float32)
BITS = BITS[np.isfinite(BITS)].astype(np.float64)
MID = (BITS + np.nextafter(BITS.astype(np.float32), np.float32(np.inf)).astype(np.float64)) / 2
MID = MID[np.isfinite(MID)]
SPELLINGS = {
    "g7": [f"{x:.7g}" for x in BITS],                  # every exponent, subnormals
    "g17": [f"{x:.17g}" for x in rng.normal(size=20000)],
    "e25": [f"{x:+.25e}" for x in rng.normal(size=20000)],  # past 19 digits
    "f": [f"{x:.3f}" for x in rng.normal(size=30000) * 1e6],
    "cut": [f"{x:.30f}" for x in rng.normal(size=9000) * 1e-4],
    "integers": [str(x) for x in rng.integers(-2**62, 2**62, 20000)],
    "odd": ["1.", ".5", "-.5", "+3", "-0", "-0.0e5", "0e-99", "000.001e+02", "1E3",
            "123456789012345678901234567890"] * 2000,
    "halfway": [repr(float(x)) for x in MID[:100]] +
               ["16777217", "33554435", "0.5000000298023223876953125"] +
               [f"{x:.4g}" for x in BITS[:20000]],
    "listed": ["nan", "inf", "-infinity", "0x1.8p3", "1e-70", "1e60", "1e39",
               "1" * 60, "1e0005"] + ["2.5"] * 20000,
    "many listed": ["inf"] * 300 + ["2.5"] * 20000,     # the text goes back
}


@pytest.mark.parametrize("name", sorted(SPELLINGS))
def test_spelling(name):
    text = text_of(SPELLINGS[name])
    assert len(text) > DEVICE_MIN
    assert check(text) == len(SPELLINGS[name])


@pytest.mark.parametrize("where", [0, 1, 7000, 19999])
@pytest.mark.parametrize("bad", ["x 2 3.0", "2 x 3.0", "2 2 x", "2.5 2 3", "2 2 3.0x", "+4 +5 6",
                                 "00000000003 4 5"])
def test_odd_entry(where, bad):
    """reading stops, shifts or goes on at that entry as fscanf does"""
    head, *lines = text_of(["1.25"] * 20000).rsplit(b"\n", 20000)
    lines[where] = bad.encode()
    check(b"\n".join([head] + lines))


@pytest.mark.parametrize("pad", range(0, 34, 3))
def test_chunk_edges_and_white_space(pad):
    """every kind of token on many offsets of a chunk, a few white spaces"""
    seps = ["\n", " \n", "\r\n", "\t\n\v", "\f\n  "]
    vals = [f"{x:.9g}" + seps[k % 5] for k, x in enumerate(rng.normal(size=6000))]
    text = text_of(vals, sep="").replace(b"% x", b"% " + b"x" * pad)
    check(text)
    check(text + b" ", device=False)


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("sym", ["general", "symmetric"])
def test_size_bound_and_pattern(extra, sym):
    lines = [f"{1 + k % 3000:d} {1 + (k * 7) % 3000:d}" for k in range(3000)]
    body = "\n".join(lines)[:DEVICE_MIN + extra].encode()
    assert len(body) == DEVICE_MIN + extra
    head = f"%%MatrixMarket matrix coordinate pattern {sym}\n3000 3000 %d\n"
    check((head % 3000).encode() + body)  # fewer entries than declared
    check((head % 500).encode() + body)  # and more
