"""Definition levels and dictionary indices in every shape of the RLE / bit-packed hybrid: one packed run,
runs of 63 groups (pyarrow's), RLE runs of any length, mixtures with empty runs and padded varints, streams
that run past the rows, at sizes around items and the levels kernel's windows; and streams that end too
early, which fail the call."""
import numpy as np
import pytest

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu import workloads as W

pytestmark = pytest.mark.gpu


def _varint(v, pad=0):
    out = bytearray()
    while True:
        b = v & 0x7F
        v >>= 7
        if v or pad:
            out.append(b | 0x80)
            if not v:
                return bytes(out) + b"\x80" * (pad - 1) + b"\x00"
        else:
            out.append(b)
            return bytes(out)


def _packed(vals, bw, pad=0):
    groups = (len(vals) + 7) // 8
    v = np.zeros(groups * 8, dtype=np.uint64)
    v[:len(vals)] = vals
    bits = ((v[:, None] >> np.arange(bw, dtype=np.uint64)) & np.uint64(1)).astype(np.uint8)
    return _varint(groups << 1 | 1, pad) + np.packbits(bits.reshape(-1), bitorder="little").tobytes()


def _rle(v, n, bw, pad=0):
    return _varint(n << 1, pad) + int(v).to_bytes((bw + 7) // 8, "little")


def _encode(vals, bw, shape, seed):
    """vals (non-negative, below 2^bw) as one stream of the hybrid."""
    rng = np.random.default_rng(seed)
    n = len(vals)
    if shape == "packed":
        return _packed(vals, bw)
    out = bytearray()
    i = 0
    while i < n:
        same = 1
        if shape != "63 groups":
            while i + same < n and vals[i + same] == vals[i]:
                same += 1
        if shape == "rle" or (shape == "mixed" and (same >= 16 or rng.random() < 0.2)):
            m = same if shape == "rle" or rng.random() < 0.7 else int(rng.integers(1, same + 1))
            out += _rle(vals[i], m + (1000 if i + m == n else 0), bw, int(rng.integers(0, 3)) if shape == "mixed" else 0)
            i += m
        else:
            m = min(n - i, 8 * (63 if shape == "63 groups" else int(rng.integers(1, 40))))
            out += _packed(vals[i:i + m], bw, int(rng.integers(0, 2)) if shape == "mixed" else 0)
            i += m
        if shape == "mixed" and rng.random() < 0.1:
            out += _rle(0, 0, bw) + _varint(1)  # runs of no rows
    return bytes(out)


def _columns(rows, null_rate, seed):
    rng = np.random.default_rng(seed)
    if null_rate == "clusters":  # long runs of both kinds, then short ones
        valid = np.repeat(rng.random(rows // 700 + 1) < 0.5, 700)[:rows].copy()
        tail = rows // 3
        valid[:tail] ^= rng.random(tail) < 0.1
    else:
        valid = rng.random(rows) >= null_rate
    return [("a", D.GDF_INT32, rng.integers(0, 3000, rows).astype(np.int32), valid),
            ("b", D.GDF_INT64, np.repeat(rng.integers(0, 20, rows // 50 + 1), 50)[:rows].astype(np.int64), ~valid),
            ("c", D.GDF_FLOAT64, rng.integers(0, 5, rows) / 4.0, None)]


def _scan(cols, dictionary, page):
    b = W.parquet_bytes(cols, page_rows=page, dictionary=dictionary)
    for locked in (False, True):
        got = R.parquet_scan_filter(b, [0, 1, 2], None, page_locked=locked)
        for (name, _, v, m), g in zip(cols, got):
            keep = np.ones(len(v), bool) if m is None else m
            np.testing.assert_array_equal(g.valid_bools(), keep, err_msg=name)
            np.testing.assert_array_equal(g.to_numpy()[keep], v[keep], err_msg=name)
            assert g.null_count == int((~keep).sum())


@pytest.mark.parametrize("shape", ["packed", "63 groups", "rle", "mixed"])
@pytest.mark.parametrize("rows,page", [(1, 1), (31, 31), (8191, 8191), (8193, 8193), (70_001, 70_001), (70_001, 12_345)])
@pytest.mark.parametrize("null_rate", [0.0, 0.03, 0.5, 1.0, "clusters"])
def test_level_streams(monkeypatch, shape, rows, page, null_rate):
    def levels(valid):
        s = _encode(valid.astype(np.int64), 1, shape, rows)
        return len(s).to_bytes(4, "little") + s
    monkeypatch.setattr(W, "_def_levels", levels)
    _scan(_columns(rows, null_rate, rows), False, page)


@pytest.mark.parametrize("shape", ["63 groups", "rle", "mixed"])
@pytest.mark.parametrize("rows,page", [(1, 1), (33, 33), (70_001, 70_001), (70_001, 12_345)])
def test_index_streams(monkeypatch, shape, rows, page):
    one_entry = W._bit_packed  # indices of no bits
    monkeypatch.setattr(W, "_bit_packed", lambda idx, bw: _encode(idx, bw, shape, rows) if bw else one_entry(idx, bw))
    _scan(_columns(rows, 0.2, rows), True, page)


@pytest.mark.parametrize("rows", [300_007, 1_000_000])
def test_large_pages(monkeypatch, rows):
    """Pages of several batches of indices, many items and many windows of levels."""
    _scan(_columns(rows, "clusters", 4), True, rows)


@pytest.mark.parametrize("shape", ["packed", "63 groups", "rle"])
@pytest.mark.parametrize("rows", [5, 8192, 70_001])
def test_streams_that_end_too_early(monkeypatch, shape, rows):
    def levels(valid):
        s = _encode(valid.astype(np.int64), 1, shape, rows)[:-1]
        if shape == "rle":
            s = s[:-2]
        return len(s).to_bytes(4, "little") + s
    monkeypatch.setattr(W, "_def_levels", levels)
    b = W.parquet_bytes(_columns(rows, 0.3, rows), page_rows=rows)
    for locked in (False, True):
        with pytest.raises(R.RalError):
            R.parquet_scan_filter(b, [0, 1, 2], None, page_locked=locked)
    monkeypatch.undo()
    _scan(_columns(100, 0.3, 1), False, 100)  # the context stays usable
