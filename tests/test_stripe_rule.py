"""Where column stripes pay (csrc/cuda/stripe_rule.cuh), on products measured
both ways: (heavy rows, A entries of each, B's mean row, columns)."""
import subprocess
from pathlib import Path

CUDA = Path(__file__).resolve().parents[1] / "rv-sparse_b200" / "csrc" / "cuda"

PAY = [(300, 3000, 8, 10000), (1000, 1000, 8, 10000), (1000, 10000, 8, 10000),
       (1000, 150, 30, 10000), (300, 400, 30, 10000), (1000, 400, 8, 10000), (1, 3000, 30, 10000),
       (1, 10000, 30, 100000), (1000, 400, 30, 100000), (300, 3000, 30, 100000),
       (1982, 40, 40, 2000), (1100, 100, 100, 1100), (19824, 40, 40, 20000)]
NOT = [(0, 0, 0, 5000), (1, 400, 8, 2000), (100, 1000, 8, 2000), (100, 1000, 30, 2000),
       (300, 400, 8, 10000), (100, 3000, 8, 10000), (100, 10000, 8, 10000),
       (100, 150, 30, 10000), (1000, 1000, 8, 100000), (1000, 3000, 8, 100000),
       (1000, 10000, 8, 100000), (300, 150, 30, 100000)]
# rows, products, A entries, longest row, columns of R-MAT 2^11, 2^12 and 2^16
GRAPHS = [(598, 1997270, 22398, 19796, 2048), (1331, 6080724, 48597, 40382, 4096),
          (26861, 397812266, 930177, 652075, 65536)]


def test_measured_products(tmp_path):
    lines = []
    for pay, cases in ((1, PAY), (0, NOT)):
        for rows, entries, mean, cols in cases:
            ops = entries * mean
            lines.append((rows, rows * ops, rows * entries, ops + ops // 20, cols, pay))
    lines += [g + (1,) for g in GRAPHS]
    body = "\n".join("  if (stripes_pay({%dull, %dull, %dull, %dull}, %d, %d) != %d) return %d;"
                     % (r, o, n, m, c, c, pay, i + 1)
                     for i, (r, o, n, m, c, pay) in enumerate(lines))
    src = tmp_path / "t.cpp"
    src.write_text('#define __host__\n#define __device__\n#include "stripe_rule.cuh"\n'
                   "using namespace rvsp;\nint main() {\n%s\n  return 0;\n}\n" % body)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-I", str(CUDA), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)]).returncode
    assert r == 0, lines[r - 1]
