"""Gathers whose records are allocated ahead, and those above 4 GB, allocated once the index is known to be
scattered, each with and without a column left over: against torch's indexing."""
import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["scattered", "sorted"])
@pytest.mark.parametrize("rows,columns", [(9_000_001, 8), (9_000_001, 9), (70_000_001, 9), ((1 << 27) + 3, 8)])
def test_large_gathers(rows, columns, order):
    g = torch.Generator(device="cuda").manual_seed(rows + columns)
    n_out = rows // 4 + 5
    idx = torch.randint(0, rows, (n_out,), generator=g, device="cuda", dtype=torch.int32)
    if order == "sorted":
        idx = torch.arange(n_out, device="cuda", dtype=torch.int32) + 3
    idx[::1001] = -1
    row = torch.arange(rows, device="cuda", dtype=torch.int64)
    cols = [R.Column(row * (2 * c + 1) + c, None, D.GDF_INT64, size=rows) for c in range(columns)]
    del row
    got = R.materialize_columns(cols, R.Column(idx, None, D.GDF_INT32), with_valid=[False] * columns)
    ok = idx >= 0
    at = idx.to(torch.int64)[ok]
    for c, out in enumerate(got):
        assert torch.equal(out.data[:n_out][ok], at * (2 * c + 1) + c)
