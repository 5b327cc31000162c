"""The library's scratch pool: a clustered gather of more than 4 GB of records allocates none, a scattered one
keeps at most 8 GB, and ral_trim_scratch gives that back."""
import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu.capi import trim_scratch

pytestmark = pytest.mark.gpu

SLACK = 256 << 20


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("rows", [20_000_000, 70_000_000, 140_000_000])
def test_memory_of_gathers(rows):
    cols = [R.Column(torch.zeros(rows, dtype=torch.int64, device="cuda"), None, D.GDF_INT64, size=rows) for _ in range(8)]
    n_out = rows // 4 + 1
    in_order = R.Column(torch.arange(n_out, dtype=torch.int32, device="cuda"), None, D.GDF_INT32)
    scattered = R.Column(torch.randint(0, rows, (n_out,), dtype=torch.int32, device="cuda"), None, D.GDF_INT32)
    few = R.Column(torch.arange(100, dtype=torch.int32, device="cuda"), None, D.GDF_INT32)
    R.materialize_columns(cols, few, with_valid=[False] * 8)  # the kernels' module
    outs = [torch.empty(n_out, dtype=torch.int64, device="cuda") for _ in range(8)]  # torch's memory for the outputs
    del outs
    trim_scratch()
    before = _free()
    R.materialize_columns(cols, in_order, with_valid=[False] * 8)
    if 64 * rows > 4 << 30:
        assert before - _free() < SLACK
    R.materialize_columns(cols, scattered, with_valid=[False] * 8)
    assert before - _free() <= (8 << 30) + SLACK
    trim_scratch()
    assert before - _free() < SLACK
