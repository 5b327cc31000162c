"""The error of the integer-pipe sin / cos (csrc/softfp.cuh), built for the host: below 0.52 ulp of the exact value
for every kind of finite argument below 2^52 (0.51 is what the functions state; the reference adds 2^-11)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT


def test_error_against_long_double(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    out = str(tmp_path / "trig_check")
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"),
                           os.path.join(ROOT, "tests", "softfp", "trig_check.cpp"), "-o", out])
    lines = subprocess.run([out, "400000"], capture_output=True, text=True, check=True).stdout.split("\n")
    rows = {f[0]: (int(f[1]), float(f[2]), f[3]) for f in (line.split() for line in lines if line)}
    assert set(rows) == {"bounds", "quarters", "spread", "small", "plain"}
    for name, (n, err, at) in rows.items():
        assert n >= 200_000 and err < 0.52, f"{name}: {err} ulp at {at}"
