"""The scan kernels' word-wise field functions (csrc/textscan.cuh), built for the host: wherever one gives
a value it is the byte-wise function's (which test_textscan_cpu.py compares with the oracle), bit for
bit, and the common shapes of a field are among those it gives."""
import os
import random
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

OK = 1


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    out = str(tmp_path_factory.mktemp("textwords") / "textwords_check")
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"),
                           os.path.join(ROOT, "tests", "textscan", "textwords_check.cpp"), "-o", out])
    return out


def _fields(kind, rng):
    """(field, whether the word-wise function must take it)."""
    if kind == "d":
        for _ in range(40000):
            y, m, d = rng.randint(0, 9999), rng.randint(0, 13), rng.randint(0, 32)
            yield f"{y:04d}-{m:02d}-{d:02d}".encode(), False
        for y in (1, 4, 100, 400, 1900, 1970, 2000, 2024, 9999):
            for m in range(1, 13):
                for d in (1, 28):
                    yield f"{y:04d}-{m:02d}-{d:02d}".encode(), True
    else:
        for n in range(1, 18):
            for _ in range(1500):
                s = "".join(rng.choice("0123456789") for _ in range(n))
                neg = rng.choice(["", "-"])
                if kind == "i":
                    yield (neg + s).encode(), n + len(neg) <= 16
                    continue
                p = rng.randint(0, n)
                f = (neg + s[:p] + "." + s[p:]).encode()
                yield f, len(f) <= 16 and n <= 15
                yield (neg + s).encode(), n + len(neg) <= 16 and n <= 15
        for _ in range(20000 if kind == "f" else 0):  # quotients next to a midpoint of two doubles are the hard ones to round
            f = rng.randint(1, 15)
            q = rng.uniform(1, 10) * 10.0 ** rng.randint(-1, 14 - f) if f < 14 else rng.uniform(0, 4)
            m = int(q * 10 ** f)
            if 0 < m < 1 << 52 and len(str(m)) <= 14 and f < len(str(m)):
                s = str(m)
                yield (s[:-f] + "." + s[-f:]).encode(), True
    chars = b"0123456789.-+ eE:|\r\xff\x00/"
    for _ in range(40000):  # anything at all, and one wrong byte in a good field
        yield bytes(rng.choice(chars) for _ in range(rng.randint(0, 18))), False
        f = bytearray(b"1995-03-17" if kind == "d" else str(rng.randint(0, 10 ** rng.randint(1, 16))).encode())
        f[rng.randrange(len(f))] = rng.randrange(256)
        yield bytes(f), False


@pytest.mark.parametrize("kind", ["i", "f", "d"])
def test_word_wise_fields_match_the_byte_wise_ones(checker, kind):
    cases = list(_fields(kind, random.Random(ord(kind))))
    inp = "".join(f"{kind} {f.hex()}\n" for f, _ in cases)
    out = subprocess.run([checker], input=inp, capture_output=True, text=True, check=True).stdout.split("\n")
    for (f, must), line in zip(cases, out):
        fast, fv, slow, sv = (int(x) for x in line.split())
        assert not fast or (slow == OK and fv == sv), (f, line)
        assert fast or not must, (f, line)
