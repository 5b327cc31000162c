"""Several columns of a scattered index gathered by way of row records (RAL_GATHER_RECORDS_BYTES lowers the
table size from which they are): against numpy's indexing at sizes around the kernels' steps and mask
words, records of 16, 32 and 64 bytes and groups of columns, every element and index width, indices
outside the input, and a clustered index, which keeps the direct kernel."""
import numpy as np
import pytest

import ralgpu as R
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu

MIXED = [D.GDF_INT8, D.GDF_INT16, D.GDF_INT32, D.GDF_INT64, D.GDF_FLOAT64]
IDX = {4: D.GDF_INT32, 8: D.GDF_INT64, 2: D.GDF_INT16}


@pytest.fixture(autouse=True)
def _always(monkeypatch):
    monkeypatch.setenv("RAL_GATHER_RECORDS_BYTES", "1")


def _check(n_in, idx, width, dtypes=MIXED, null_rate=0.1, masked=lambda k: k % 2 == 0, out_masked=lambda k: True):
    rng = np.random.default_rng(n_in + len(idx) + len(dtypes))
    n = len(idx)
    vals = [rng.integers(-(1 << 62), 1 << 62, n_in).astype(D.NP[t]) if t != D.GDF_FLOAT64 else rng.standard_normal(n_in)
            for t in dtypes]
    valid = [rng.random(n_in) >= null_rate if masked(k) else None for k in range(len(dtypes))]
    cols = [R.Column.from_numpy(v, t, m) for v, t, m in zip(vals, dtypes, valid)]
    ok = (idx >= 0) & (idx < n_in)
    at = np.where(ok, idx, 0)
    got = R.materialize_columns(cols, R.Column.from_numpy(idx, IDX[width]),
                                with_valid=[out_masked(k) for k in range(len(cols))])
    for v, m, g in zip(vals, valid, got):
        np.testing.assert_array_equal(g.to_numpy()[ok], v[at][ok])
        if g.valid is not None:
            bits = ok & (m[at] if m is not None else True)
            np.testing.assert_array_equal(g.valid_bools(), bits)
            assert g.null_count == n - bits.sum()


@pytest.mark.parametrize("n_in,n_out", [(100_003, 30_000), (70_000, 65_535), (70_000, 65_536), (70_001, 65_537),
                                        (2048, 2048), (127, 2049), (129, 5000), (1, 2049), (300_017, 100_000)])
def test_sizes(n_in, n_out):
    rng = np.random.default_rng(7)
    idx = rng.integers(0, n_in, n_out).astype(np.int32)
    _check(n_in, idx, 4)
    out = idx.astype(np.int64)
    out[rng.random(n_out) < 0.2] = rng.choice([-1, n_in, 1 << 40, -(1 << 40)], 1)
    _check(n_in, out, 8)


@pytest.mark.parametrize("dtypes", [
    [D.GDF_INT8] * 2, [D.GDF_INT8] * 8, [D.GDF_INT64, D.GDF_INT32, D.GDF_INT16, D.GDF_INT8], [D.GDF_FLOAT64] * 2, [D.GDF_INT64] * 4,
    [D.GDF_INT16] * 15 + [D.GDF_INT8] * 3, [D.GDF_INT64] * 7 + [D.GDF_INT16, D.GDF_INT8], [D.GDF_INT64] * 8, [D.GDF_INT64] * 9,
    [D.GDF_INT8] * 64, MIXED * 12], ids=lambda d: f"{len(d)}x{sum(D.WIDTH[t] for t in d)}")
@pytest.mark.parametrize("masks", ["none", "all", "in only", "some"])
def test_records(dtypes, masks):
    rng = np.random.default_rng(8)
    n = 70_001
    idx = rng.permutation(n).astype(np.int32)
    _check(n, idx, 4, dtypes, 0.3, masked=lambda k: masks in ("all", "in only") or (masks == "some" and k % 3 != 1),
           out_masked=lambda k: masks == "all" or (masks == "some" and k % 2 == 0))


@pytest.mark.parametrize("pattern", ["sorted", "one row", "all outside", "int16"])
def test_patterns(pattern):
    rng = np.random.default_rng(8)
    n = 400_000
    if pattern == "sorted":
        _check(n, np.sort(rng.integers(0, n, n)).astype(np.int32), 4)
    elif pattern == "one row":  # every sample scattered, most rows read one row
        idx = rng.integers(0, n, n).astype(np.int32)
        idx[rng.random(n) < 0.9] = 123_456
        _check(n, idx, 4)
    elif pattern == "all outside":
        idx = np.full(n, -1, dtype=np.int32)
        idx[::2] = n
        idx[::31] = rng.integers(0, n, len(idx[::31]))
        _check(n, idx, 4)
    else:
        _check(n, rng.integers(-(1 << 15), 1 << 15, n).astype(np.int16), 2)
