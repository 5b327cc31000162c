"""Dictionary-encoded pages whose definition levels end too early, alone and next to whole pages: the scan is refused
(what such a page's rows would read of the indices stays within the page's own), and the next scan is right."""
import numpy as np
import pytest

import ralgpu as R
from ralgpu import dtypes as D
from ralgpu import workloads as W

pytestmark = pytest.mark.gpu


def _columns(rows):
    rng = np.random.default_rng(rows)
    valid = rng.random(rows) >= 0.05
    return [("a", D.GDF_INT32, rng.integers(0, 9, rows).astype(np.int32), valid),
            ("b", D.GDF_FLOAT64, rng.integers(0, 50, rows) / 8.0, rng.random(rows) >= 0.5)]


@pytest.mark.parametrize("locked", [False, True])
@pytest.mark.parametrize("rows,page", [(5, 5), (31, 31), (8192, 8192), (8193, 8193), (70_001, 70_001), (70_001, 20_000)])
@pytest.mark.parametrize("broken", ["all", "last"])
def test_broken_levels_of_dictionary_pages(monkeypatch, rows, page, locked, broken):
    levels, calls = W._def_levels, [0]
    pages = -(-rows // page) * 2

    def short(valid):
        s = levels(valid)
        calls[0] += 1
        if broken == "last" and calls[0] < pages:
            return s
        cut = s[4:-1] if len(s) < 40 else s[4:len(s) // 2]  # the stream's last byte, or its second half
        return len(cut).to_bytes(4, "little") + cut

    monkeypatch.setattr(W, "_def_levels", short)
    b = W.parquet_bytes(_columns(rows), page_rows=page, dictionary=True)
    assert calls[0] == pages
    monkeypatch.undo()
    with pytest.raises(R.RalError, match="malformed"):
        R.parquet_scan_filter(b, [0, 1], None, page_locked=locked)
    cols = _columns(1000)
    got = R.parquet_scan_filter(W.parquet_bytes(cols, dictionary=True), [0, 1], None, page_locked=locked)
    for (_, _, v, m), g in zip(cols, got):
        np.testing.assert_array_equal(g.valid_bools(), m)
        np.testing.assert_array_equal(g.to_numpy()[m], v[m])
