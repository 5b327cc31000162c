"""The ways a Parquet file's bytes reach the decode kernels: ordinary memory and a mapped file read in place where
the device reads host pages, chunks copied in on request; one mask byte, one item and one copy piece more
or less, dictionary chunks (copied to the device) next to PLAIN ones (read in place), Snappy pages."""
import ctypes as C
import mmap

import numpy as np
import pytest

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu import workloads as W

pytestmark = pytest.mark.gpu


def _columns(rows):
    rng = np.random.default_rng(rows)
    valid = rng.random(rows) >= 0.1
    return [("a", D.GDF_INT32, rng.integers(0, 90, rows).astype(np.int32), valid),
            ("b", D.GDF_FLOAT64, rng.standard_normal(rows), None),  # more values than a dictionary takes
            ("c", D.GDF_INT64, rng.integers(0, 7, rows).astype(np.int64), None),
            ("d", D.GDF_FLOAT64, rng.standard_normal(rows), ~valid)]


def _scan(address, n_bytes, rows, dts):
    outs = [R.Column.empty(t, rows, with_valid=True) for t in dts]
    for o in outs:
        o.valid.fill_(0xA5)
    structs = [o.to_c() for o in outs]
    arr = (C.POINTER(type(structs[0])) * len(outs))(*[C.pointer(s) for s in structs])
    n = C.c_int32(-1)
    pr = (C.c_int32 * len(outs))(*range(len(outs)))
    assert R.lib().ral_parquet_scan_filter(C.c_void_p(address), n_bytes, pr, len(outs), None,
                                           C.cast(arr, C.c_void_p), C.byref(n)) == 0
    assert n.value == rows
    return outs, structs


@pytest.mark.parametrize("how", ["ordinary", "unaligned", "mapped", "copied"])
@pytest.mark.parametrize("dictionary,snappy", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("rows", [1, 7, 8, 8193, 131_072, 150_001])
def test_ways_in(monkeypatch, tmp_path, how, dictionary, snappy, rows):
    cols = _columns(rows)
    b = W.parquet_bytes(cols, row_group_rows=100_000, page_rows=40_000, dictionary=dictionary, snappy=snappy,
                        dictionary_max=1000)
    if how == "copied":
        monkeypatch.setenv("RAL_PARQUET_STAGED", "1")
    if how == "mapped":
        path = tmp_path / "f.parquet"
        path.write_bytes(b)
        with open(path, "rb") as f:
            held = mmap.mmap(f.fileno(), 0, access=mmap.ACCESS_COPY)
        view = np.frombuffer(held, np.uint8)
    else:
        shift = 5 if how == "unaligned" else 0
        view = np.empty(len(b) + shift, np.uint8)[shift:]
        view[:] = np.frombuffer(b, np.uint8)
    outs, structs = _scan(view.ctypes.data, len(b), rows, [t for _, t, _, _ in cols])
    for (name, _, v, m), o, s in zip(cols, outs, structs):
        keep = np.ones(rows, bool) if m is None else m
        mask = o.valid.cpu().numpy()
        bits = np.unpackbits(mask, bitorder="little")
        np.testing.assert_array_equal(bits[:rows].astype(bool), keep, err_msg=name)
        assert not bits[rows:].any(), name  # the bytes after the last row are cleared
        np.testing.assert_array_equal(o.data.cpu().numpy()[:rows][keep], v[keep], err_msg=name)
        assert s.null_count == int((~keep).sum())
