"""RAL_SCAN_TUNE: every accepted value gives text scan kernels that compile within a plain launch's shared memory."""
import re

import pytest

import ralgpu as R
from ralgpu import workloads as W


@pytest.mark.parametrize("tune", ["T=128", "T=256", "T=512", "J=4,B=2", "B=16"])
def test_tuned_scan_kernels_compile(tmp_path, monkeypatch, tune):
    monkeypatch.setenv("RAL_JIT_CACHE_DIR", str(tmp_path))
    monkeypatch.setenv("RAL_SCAN_TUNE", tune)
    _, log = R.debug_text_scan_source(W.TEXT_DTYPES, list(range(8)), "LogicalFilter(condition=[<($0, 26)])", compile=True)
    smem = [int(b) for b in re.findall(r"(\d+) bytes smem", log)]
    assert smem and max(smem) <= 48 * 1024
