"""The text scan's ranges, ring and line slots at the sizes where they can go wrong, against the oracle's
scan (oracle/textscan.py): lines that cross range ends, lines longer than a slot, the delimiter window and
the ring, ranges that keep more lines than wait in shared memory, dense blank lines, texts that start at
any byte, and skipped lines by both searches."""
import random

import pytest
import torch

import helpers as H
import oracle as O
import ralgpu as R
from oracle import textscan as T
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu

DTYPES = [D.GDF_INT64, D.GDF_FLOAT64, D.GDF_DATE64, D.GDF_INT32]
FILTER = "LogicalFilter(condition=[AND(>=($0, 100), <($1, 50.5))])"


def _check(text, proj=(0, 1, 2, 3), fq=FILTER, offset=0, **kw):
    exp = T.scan_filter(text, DTYPES, list(proj), fq, **kw)
    for e in exp:
        O.update_null_count(e)
    buf = torch.frombuffer(bytearray(b"\n" * offset + text + b"|7\n"), dtype=torch.uint8).to("cuda")
    got = R.text_scan_filter(buf[offset:offset + len(text)], DTYPES, list(proj), fq, **kw)
    for k, (g, e) in enumerate(zip(got, exp)):
        H.assert_columns_equal(g, e, what=f"column {k} (offset {offset}, {kw})")


def _line(rng, pad=0):
    f = [str(rng.randint(-999, 10 ** rng.randint(3, 12))),
         rng.choice([f"{rng.randint(0, 99999)}.{rng.randint(0, 99):02d}", f"{rng.random() * 99:.9f}", "1e2", f"{rng.randint(0, 60)}"]),
         f"{rng.randint(1, 9999):04d}-{rng.randint(1, 12):02d}-{rng.randint(1, 29):02d}", str(rng.randint(-50, 50))]
    if pad:
        f[rng.randrange(4)] = " " * pad + f[0]
    return "|".join(f[:rng.randint(1, 4)] if rng.random() < 0.1 else f)


@pytest.mark.parametrize("offset", [0, 1, 7, 15, 16])
def test_texts_at_any_address(offset):
    rng = random.Random(offset)
    for n in (1, 2, 31, 33, 300):
        text = "\n".join(_line(rng) for _ in range(n)).encode()
        _check(text, offset=offset)
        _check(text + b"\n", offset=offset, fq=None)
    for n in (1022, 1023, 1024, 1025, 2047, 2049):  # the text ends next to a range's end
        _check((b"123456|1.5|2001-01-01|5\n" * 90)[:n], offset=offset)


@pytest.mark.parametrize("pad", [80, 100, 235, 250, 1010, 4000, 4200, 9000, 70000])
def test_long_lines(pad):
    """Beyond the delimiter window, a line's slot, a step, the ring and 16-bit positions and lengths."""
    rng = random.Random(pad)
    lines = [_line(rng, pad if rng.random() < 0.3 else 0) + ("\r" if rng.random() < 0.1 else "") for _ in range(60)]
    _check("\n".join(lines).encode())
    _check(("\n".join(lines) + "\n").encode(), fq=None)
    _check(("\n".join(lines[::-1])).encode(), proj=(3, 0), fq="LogicalFilter(condition=[<($0, 10)])")


@pytest.mark.parametrize("blank", [b"\n", b"\r\n"])
def test_dense_blank_lines(blank):
    rng = random.Random(3)
    text = b"".join(blank * rng.choice([0, 1, 5, 600, 3000]) + _line(rng).encode() + b"\n" for _ in range(80))
    _check(text)
    _check(blank * 5000, fq=None)


@pytest.mark.parametrize("tail", [0, 1])
def test_ranges_with_more_kept_lines_than_wait(tail):
    """Long lines first (they set the range size), then two-byte lines: over 512 kept lines a range."""
    rng = random.Random(5)
    lines = [_line(rng, 230) for _ in range(17000)] + ["7"] * 60000 + [_line(rng) for _ in range(500)]
    text = "\n".join(lines).encode() + b"\n" * tail
    _check(text, proj=(0, 3), fq=None)
    _check(text, proj=(0,), fq="LogicalFilter(condition=[>($0, 6)])")


@pytest.mark.parametrize("skip", [0, 1, 16, 17, 4000, 9999, 10000, 10001, 20000])
def test_skipped_lines(skip):
    rng = random.Random(9)
    text = "\n".join(_line(rng) if rng.random() < 0.9 else "" for _ in range(10000)).encode()
    _check(text, skip_rows=skip, offset=skip % 16)
