"""The cases of test_stripes_gpu.py, most of them too small for stripes to pay,
with stripes for every heavy row, on the plain and on the learned path."""
import pytest

import test_stripes_gpu as cases
from rvsp import Descriptor
from rvsp import _lib as L
from rvsp.learn import RowModel, weights_for
from test_stripes_gpu import (test_columns_of_another_product_are_reported,  # noqa: F401
                              test_hub_rows_and_every_row_heavy,
                              test_values_that_cancel_or_are_not_finite, test_widths)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True, params=[L.ALGO_CUDA_PLAIN, L.ALGO_CUDA_LEARNED])
def always(request, monkeypatch):
    class Always(Descriptor):
        def __init__(self, algo, memory):
            super().__init__(algo=request.param, memory=memory)
            self.set_stripes(2)
            if request.param == L.ALGO_CUDA_LEARNED:
                self.set_model(RowModel(path=weights_for("rmat")))

    monkeypatch.setattr(cases, "Descriptor", Always)
