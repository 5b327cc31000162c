"""Which columns of a scattered gather travel in row records, on both sides of every condition, and that the
records never take more device memory than they may."""
import pytest

from ralgpu.capi import debug_gather_plan

KEPT = 8 << 30


@pytest.fixture(autouse=True)
def _default(monkeypatch):
    monkeypatch.delenv("RAL_GATHER_RECORDS_BYTES", raising=False)


def _plan(widths, rows_in, rows_out=None, masked=False, most=KEPT):
    return debug_gather_plan(widths, [int(masked)] * len(widths), rows_in, rows_in if rows_out is None else rows_out, most)


def test_table_size():
    least = (24 << 20) // 16
    assert _plan([8, 8], least) == ([16, 16], 16 * least)
    assert _plan([8, 8], least - 1) == ([0, 0], 0)


def test_rows_gathered(monkeypatch):
    assert _plan([8, 8], 2_000_003, 500_000)[0] == [16, 16]
    assert _plan([8, 8], 2_000_003, 499_999)[0] == [0, 0]
    monkeypatch.setenv("RAL_GATHER_RECORDS_BYTES", "1")
    assert _plan([8, 8], 3000, 2048)[0] == [16, 16]
    assert _plan([8, 8], 3000, 2047)[0] == [0, 0]


def test_columns_and_row_bytes():
    n = 40_000_000
    assert _plan([8], n)[0] == [0]
    assert _plan([4, 2, 1], n)[0] == [0, 0, 0]
    assert _plan([4, 2, 1, 1], n)[0] == [16] * 4
    assert _plan([4, 4, 4, 4], n, masked=True)[0] == [32] * 4
    assert _plan([1] * 64, n)[0] == [64] * 64


@pytest.mark.parametrize("left", [[8], [1, 1], [4, 2]])
def test_leftover_columns_go_straight(left):
    """Eight 8-byte columns fill a record; what is left fills less than half of another, or is one column."""
    assert _plan([8] * 8 + left, 10_000_000) == ([64] * 8 + [0] * len(left), 640_000_000)


@pytest.mark.parametrize("widths", [[8] * 8, [8, 8, 4, 4, 4, 1], [8, 4], [1] * 64, [8] * 9, [2] * 40 + [8] * 24])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("rows", [1 << 27, (1 << 27) + 1, 1 << 28, (1 << 28) + 1, 300_000_000, 1 << 29, (1 << 29) + 1, (1 << 31) - 1])
@pytest.mark.parametrize("most", [KEPT, 1 << 36, 1 << 20])
def test_scratch_is_bounded(widths, masked, rows, most):
    records, scratch = _plan(widths, rows, masked=masked, most=most)
    assert scratch == rows * max(records) <= most


def test_narrower_records_where_wider_ones_do_not_fit():
    assert _plan([8] * 8, 1 << 27) == ([64] * 8, KEPT)
    assert _plan([8] * 8, (1 << 27) + 1)[0] == [32] * 8
    assert _plan([8] * 8, (1 << 28) + 1)[0] == [16] * 8
    assert _plan([8] * 8, (1 << 29) + 1) == ([0] * 8, 0)
    assert _plan([8, 8], (1 << 28) + 1, masked=True) == ([0, 0], 0)  # a mask's bits leave room for one column only
