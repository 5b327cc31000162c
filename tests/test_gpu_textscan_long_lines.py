"""Lines of megabytes: what a scan reads of one ends with the last field it needs, and line ends with a
carriage return, also as the delimiter, agree with the oracle's on both sides of the line slots' sizes."""
import random
import time

import pytest
import torch

import ralgpu as R
from oracle import textscan as T
from test_gpu_textscan_ranges import DTYPES, FILTER, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fq", [None, FILTER])
def test_a_line_of_64_mb_costs_its_fields(fq):
    """By one lane a byte at a time, or by one warp 512 bytes at a time, 64 MB take over 50 ms of latency alone
    (2^26 bytes of at least 10 ns, 2^17 steps of at least 400 ns); the whole text is read in 0.1 ms."""
    lines = [b"123456|1.5|2001-01-01|5", b"777|2.25|1999-12-31|-3|" + b"x" * (64 << 20), b"100|0.5|2000-02-29|9"]
    short = b"\n".join(line[:60] for line in lines)
    text = torch.frombuffer(bytearray(b"\n".join(lines)), dtype=torch.uint8).to("cuda")
    exp = T.scan_filter(short, DTYPES, [0, 1, 2, 3], fq)
    best = 1e9
    for _ in range(3):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        got = R.text_scan_filter(text, DTYPES, [0, 1, 2, 3], fq, capacity=3)
        best = min(best, time.perf_counter() - t0)
    for g, e in zip(got, exp):
        assert g.size == e.size == 3
        assert g.to_numpy().tolist() == e.data.tolist() and g.valid_bools().all()
    assert best < 0.025


@pytest.mark.parametrize("delim", [b"|", b"\r"])
@pytest.mark.parametrize("pad", [0, 100, 245, 4200, 70000])
def test_carriage_returns_at_line_ends(delim, pad):
    rng = random.Random(pad)
    lines = []
    for _ in range(40):
        f = [b"%d" % rng.randint(100, 999), b"%d.5" % rng.randint(0, 40), b"2001-02-%02d" % rng.randint(1, 28), b"%d" % rng.randint(0, 9)]
        k = rng.randrange(4)
        f[k] = b" " * (pad if rng.random() < 0.5 else 0) + f[k]
        lines.append(delim.join(f[:rng.randint(1, 4)]) + b"\r" * rng.choice([0, 1, 1, 2, 3]))
    for text in (b"\n".join(lines), b"\n".join(lines) + b"\n", b"\r\n".join(lines) + b"\r"):
        _check(text, delimiter=delim)
        _check(text, delimiter=delim, fq=None, proj=(3, 1))
