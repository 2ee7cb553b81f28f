"""Entry indices near 2^31 (csrc/cuda/index.cuh), compiled for the host with
overflow checks."""
import subprocess
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parents[1] / "rv-sparse_b200" / "csrc" / "cuda"


def _run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text('#define __host__\n#define __device__\n#include "index.cuh"\n'
                   "using namespace rvsp;\nint main() {\n%s\nreturn 0;\n}\n" % body)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    "-I", str(CUDA), "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)]).returncode


@pytest.mark.parametrize("lo,hi", [(0, 0), (0, 1), (5, 8), (2**30, 2**30 + 1),
                                   (2**30 - 1, 2**30 + 2), (0, 2**31 - 1),
                                   (2**31 - 2, 2**31 - 1)])
def test_middle(tmp_path, lo, hi):
    assert _run(tmp_path, "if (middle(%d, %d) != %d) return 1;" % (lo, hi, (lo + hi) // 2)) == 0


@pytest.mark.parametrize("base,step,end", [(0, 0, 0), (3, 4, 8), (3, 5, 8),
                                           (2**31 - 33, 31, 2**31 - 1),
                                           (2**31 - 33, 32, 2**31 - 1),
                                           (2**31 - 1, 31, 2**31 - 1),
                                           (2**31 + 62, 31, 2**31 - 1)])
def test_before(tmp_path, base, step, end):
    want = int(base + step < end)
    assert _run(tmp_path, "if (before(%dU, %d, %d) != %d) return 1;" % (base, step, end, want)) == 0
