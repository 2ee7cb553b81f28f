"""Shift-class members with row tiles switched off after the first compute
(csrc/cuda/plan.cu): the list of their rows is in place whether the first call
that needs it runs or is only captured.
"""
import numpy as np
import pytest

from oracle import oracle
from rvsp import Descriptor, DeviceCSR, gen
from rvsp import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["dropped", "second graph", "eager"])
def test_rows_listed_before_a_captured_call(first):
    import torch
    A = gen.stencil_3d_27(18)
    A2 = A.with_values((A.values * np.float32(1.5)).astype(np.float32))
    rp, ci, cv, _ = oracle.spgemm(A2, A2)
    dA = DeviceCSR.from_host(A)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s), Descriptor(memory=L.MEM_DEVICE, stream=s) as d:
        d.set_shift_classes(2)
        size, n = d.work_estimation(dA, dA)
        dC = DeviceCSR.empty(A.rows, A.cols, n)
        ws = torch.zeros(max(size, 1), dtype=torch.uint8, device="cuda")
        d.compute(dA, dA, dC, ws)
        d.synchronize()
        assert d.shift_rows() > 0 and d.tiled_rows() > 0
        d.set_row_tiles(False)
        dA.values.copy_(torch.from_numpy(A2.values))
        dC.values.zero_()
        s.synchronize()
        graphs = []
        for _ in range({"dropped": 1, "second graph": 2, "eager": 0}[first]):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1], stream=s):
                d.compute(dA, dA, dC, ws)
        if first == "second graph":
            graphs[1].replay()
        else:
            graphs.clear()
            d.compute(dA, dA, dC, ws)
        d.synchronize()
        got = dC.to_host(n)
    assert np.array_equal(got.row_ptr, rp)
    assert np.array_equal(got.col_idx, ci)
    assert np.array_equal(got.values.view(np.uint32), cv.view(np.uint32))
