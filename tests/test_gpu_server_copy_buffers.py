"""Buffers a served result is copied into: a column without data is refused before anything is copied, and
page-locked host memory takes the copy as device memory does."""
import numpy as np
import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu.capi import _check, _colarray, lib

pytestmark = pytest.mark.gpu


@pytest.fixture
def served():
    rows = 5000
    rng = np.random.default_rng(3)
    frame = [R.Column.from_numpy(rng.integers(-1000, 1000, rows).astype(np.int32), D.GDF_INT32, rng.random(rows) >= 0.1),
             R.Column.from_numpy(rng.standard_normal(rows), D.GDF_FLOAT64)]
    filt, proj = "LogicalFilter(condition=[>=($0, -900)])", "LogicalProject(a=[+($0, 1)], b=[*($1, 2.5)])"
    exp = R.filter_project(frame, filt, proj)
    srv = R.Server(budget_bytes=1 << 30)
    q = srv.add_query(srv.add_table(frame), filt, proj)
    srv.start()
    rid = srv.submit(q, keep=True)
    n, _ = srv.wait(rid)
    yield srv, rid, n, exp
    srv.release(rid)
    srv.close()


def _check_outs(outs, structs, exp):
    for o, st, e in zip(outs, structs, exp):
        assert st.size == e.size and st.null_count == e.null_count
        ev = e.valid_bools()
        np.testing.assert_array_equal(np.unpackbits(o.valid.cpu().numpy(), bitorder="little")[:st.size].astype(bool), ev)
        np.testing.assert_array_equal(o.data.cpu().numpy()[:st.size][ev], e.to_numpy()[ev])


@pytest.mark.parametrize("missing", [0, 1])
def test_a_column_without_data_is_refused_and_nothing_is_copied(served, missing):
    srv, rid, n, exp = served
    outs = [R.Column.empty(e.dtype, n) for e in exp]
    for o in outs:
        o.data.fill_(77)
    arr, structs = _colarray(outs)
    kept = structs[missing].data
    structs[missing].data = None
    structs[1 - missing].size = 123
    assert lib().ral_server_copy_result(srv._h, rid, arr, 2) != 0
    torch.cuda.synchronize()
    assert structs[1 - missing].size == 123
    for o in outs:
        assert bool((o.data == 77).all()) and bool((o.valid == 0xFF).all())
    structs[missing].data = kept
    _check(lib().ral_server_copy_result(srv._h, rid, arr, 2))
    _check_outs(outs, structs, exp)


@pytest.mark.parametrize("host", [(0,), (1,), (0, 1)])
def test_page_locked_host_buffers_take_the_copy(served, host):
    srv, rid, n, exp = served
    outs = [R.Column.empty(e.dtype, n, device="cpu" if k in host else "cuda") for k, e in enumerate(exp)]
    for k in host:
        outs[k].data, outs[k].valid = outs[k].data.pin_memory(), outs[k].valid.pin_memory()
    arr, structs = _colarray(outs)
    _check(lib().ral_server_copy_result(srv._h, rid, arr, 2))
    _check_outs(outs, structs, exp)


def test_buffers_of_one_allocation_and_of_several(served):
    """Columns in slices of one allocation, in allocations of their own, and at an allocation's very end."""
    srv, rid, n, exp = served
    one = torch.full((1 << 20,), 0x5A, dtype=torch.uint8, device="cuda")
    at = one.numel()
    outs = []
    for k, e in enumerate(exp):
        w = D.WIDTH[e.dtype]
        at = (at - n * w) // w * w if k else at - n * w
        data = one[at:at + n * w].view(torch.int32 if w == 4 else torch.int64)
        valid = torch.zeros((n + 7) // 8 + 64, dtype=torch.uint8, device="cuda")
        outs.append(R.Column(data, valid, e.dtype, size=n))
    arr, structs = _colarray(outs)
    _check(lib().ral_server_copy_result(srv._h, rid, arr, 2))
    for o, st, e in zip(outs, structs, exp):
        ev = e.valid_bools()
        assert st.size == n and st.null_count == e.null_count
        np.testing.assert_array_equal(np.unpackbits(o.valid.cpu().numpy(), bitorder="little")[:n].astype(bool), ev)
        np.testing.assert_array_equal(o.data.cpu().numpy()[ev], e.to_numpy().view(o.data.cpu().numpy().dtype)[ev])
    assert bool((one[:at] == 0x5A).all())
