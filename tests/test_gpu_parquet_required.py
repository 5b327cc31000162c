"""The ways a required leaf's PLAIN values get written: all by the values kernel (PLAIN leaves only), every fourth
item beside the dictionary indices (PLAIN next to dictionary leaves), beside the levels (an optional leaf in the
batch), read in place and copied in batches that mix them.  Outputs are prefilled: an item that nobody writes shows."""
import ctypes as C

import numpy as np
import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu import workloads as W

pytestmark = pytest.mark.gpu

ITEM = 8192


def _leaf(kind, k, rows, rng):
    if kind == "plain":  # more distinct values than a dictionary takes
        return (f"p{k}", D.GDF_FLOAT64, rng.standard_normal(rows), None) if k % 2 else \
            (f"p{k}", D.GDF_INT32, rng.permutation(rows).astype(np.int32), None)
    if kind == "dict":
        return f"d{k}", D.GDF_INT64, rng.integers(0, 50, rows).astype(np.int64) * 7, None
    return f"o{k}", D.GDF_INT32, rng.integers(0, 40, rows).astype(np.int32), rng.random(rows) >= 0.2


def _check(leaves, rows, page_rows, group_rows, monkeypatch, how):
    rng = np.random.default_rng(rows + len(leaves))
    cols = [_leaf(kind, k, rows, rng) for k, kind in enumerate(leaves)]
    b = W.parquet_bytes(cols, row_group_rows=group_rows, page_rows=page_rows, dictionary="dict" in leaves,
                        dictionary_max=min(100, rows // 3))
    if how == "copied":
        monkeypatch.setenv("RAL_PARQUET_STAGED", "1")
        monkeypatch.setenv("RAL_PARQUET_BATCH_BYTES", "300000")
    file = np.frombuffer(b, np.uint8).copy()
    outs = [R.Column.empty(t, rows, with_valid=True) for _, t, _, _ in cols]
    for o in outs:
        o.data.view(torch.uint8).fill_(0x5A)
        o.valid.fill_(0xA5)
    structs = [o.to_c() for o in outs]
    arr = (C.POINTER(type(structs[0])) * len(outs))(*[C.pointer(s) for s in structs])
    n = C.c_int32(-1)
    pr = (C.c_int32 * len(outs))(*range(len(outs)))
    assert R.lib().ral_parquet_scan_filter(C.c_void_p(file.ctypes.data), len(b), pr, len(outs), None,
                                           C.cast(arr, C.c_void_p), C.byref(n)) == 0
    assert n.value == rows
    for (name, _, v, m), o, s in zip(cols, outs, structs):
        keep = np.ones(rows, bool) if m is None else m
        np.testing.assert_array_equal(np.unpackbits(o.valid.cpu().numpy(), bitorder="little")[:rows].astype(bool), keep, name)
        np.testing.assert_array_equal(o.data.cpu().numpy()[:rows][keep], v[keep], name)
        assert s.null_count == int((~keep).sum())


@pytest.mark.parametrize("how", ["in place", "copied"])
@pytest.mark.parametrize("items", [1, 4, 5, 31, 32, 33])
@pytest.mark.parametrize("leaves", [["plain"], ["plain", "plain"], ["plain", "dict"], ["dict", "plain", "plain", "dict"],
                                    ["plain", "dict", "optional", "plain"]], ids="-".join)
def test_items(leaves, items, how, monkeypatch):
    """A page of these many items, the last one a row short of full, full, or of one row."""
    for rows in (items * ITEM - 1, items * ITEM, (items - 1) * ITEM + 1):
        _check(leaves, rows, rows, rows, monkeypatch, how)


@pytest.mark.parametrize("how", ["in place", "copied"])
@pytest.mark.parametrize("page_rows", [997, 8191, 8193, 30_011])
def test_odd_pages_in_batches_of_all_kinds(page_rows, how, monkeypatch):
    """Row groups of 40,000 rows: batches of 300 KB hold one to three of the leaves' chunks each."""
    leaves = ["plain", "dict", "plain", "optional", "dict", "plain", "plain", "optional"]
    _check(leaves, 150_001, page_rows, 40_000, monkeypatch, how)
    _check(["plain", "dict", "plain", "plain"], 150_001, page_rows, 40_000, monkeypatch, how)
