"""The device memory of a text scan follows the text's lines, not the room in the caller's outputs."""
import ctypes as C

import pytest
import torch

import ralgpu as R
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu

_USED, _USED_HIGH = 7, 8  # CUmemPool_attribute


def _pool():
    cu, pool = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), C.c_int(torch.cuda.current_device())) == 0
    return cu, pool


@pytest.mark.parametrize("from_host", [False, True])
@pytest.mark.parametrize("room", ["counted", "roomy"])
def test_scan_memory(room, from_host):
    line = b"12|" + b"x" * 58 + b"\n"  # 62 bytes
    rows = 4 << 20
    text = torch.frombuffer(bytearray(line), dtype=torch.uint8).repeat(rows)
    n = text.numel()
    text = text.pin_memory() if from_host else text.to("cuda")
    torch.cuda.synchronize()
    cu, pool = _pool()
    zero, before, high = C.c_uint64(0), C.c_uint64(0), C.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, C.c_int(_USED_HIGH), C.byref(zero)) == 0
    assert cu.cuMemPoolGetAttribute(pool, C.c_int(_USED), C.byref(before)) == 0
    got = R.text_scan_filter(text, [D.GDF_INT8], [0], None, capacity=rows if room == "counted" else n // 2, from_host=from_host)
    torch.cuda.synchronize()
    assert cu.cuMemPoolGetAttribute(pool, C.c_int(_USED_HIGH), C.byref(high)) == 0
    assert got[0].size == rows and bool((got[0].data[:rows] == 12).all()) and got[0].null_count == 0
    # the list at no more than the text, the ranges' words, and for host text three pieces of 64 MB (and a line)
    pieces = 3 * ((64 << 20) + 4096) if from_host else 0
    assert 0 < high.value - before.value <= n + (8 << 20) + pieces
