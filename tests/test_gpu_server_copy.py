"""Copies of served results into buffers of any alignment, at sizes around 16-byte words and mask bytes,
and bytes next to the destination left alone: against the rows that ral_filter_project keeps."""
import ctypes as C

import numpy as np
import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu.capi import _check, _colarray, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 33, 1000, 70_001])
@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_copy_result_alignment(rows, shift):
    rng = np.random.default_rng(rows)
    vals = [rng.integers(-1000, 1000, rows).astype(np.int32), rng.standard_normal(rows)]
    frame = [R.Column.from_numpy(v, t, rng.random(rows) >= 0.1) for v, t in zip(vals, (D.GDF_INT32, D.GDF_FLOAT64))]
    filt, proj = "LogicalFilter(condition=[>=($0, -900)])", "LogicalProject(a=[+($0, 1)], b=[*($1, 2.5)], c=[$0])"
    exp = R.filter_project(frame, filt, proj)
    srv = R.Server(budget_bytes=1 << 30)
    q = srv.add_query(srv.add_table(frame), filt, proj)
    srv.start()
    rid = srv.submit(q, keep=True)
    n, _ = srv.wait(rid)
    outs, bufs = [], []
    for dt, e in zip(srv.query_outputs(q)[0], exp):
        w = D.WIDTH[dt]
        data = torch.full(((n + 8) * w,), 0x5A, dtype=torch.uint8, device="cuda")
        mask = torch.full(((n + 7) // 8 + 16,), 0x5A, dtype=torch.uint8, device="cuda")
        bufs.append((data, mask, w))
        outs.append(R.Column(data[shift:], mask[shift:], dt, size=n))
    arr, structs = _colarray(outs)
    _check(lib().ral_server_copy_result(srv._h, rid, arr, len(outs)))
    for (data, mask, w), e, st in zip(bufs, exp, structs):
        assert st.size == n == e.size and st.null_count == e.null_count
        got = data.cpu().numpy()
        ev = e.valid_bools()
        gv = np.unpackbits(mask.cpu().numpy()[shift:], bitorder="little")[:n].astype(bool)
        np.testing.assert_array_equal(gv, ev)
        ed = e.to_numpy().view(np.uint8).reshape(n, w)
        np.testing.assert_array_equal(got[shift:shift + n * w].reshape(n, w)[ev], ed[ev])
        assert (got[:shift] == 0x5A).all() and (got[shift + n * w:] == 0x5A).all()
        mb = mask.cpu().numpy()
        assert (mb[:shift] == 0x5A).all() and (mb[shift + (n + 7) // 8:] == 0x5A).all()
    srv.release(rid)
    srv.close()
