"""Filters and text scans clear their scratch and every output mask in one launch: nothing of what the masks held
before shows, at mask sizes around one and several 16-byte words and with more outputs than one launch
takes."""
import numpy as np
import pytest

import helpers as H
import oracle as O
import ralgpu as R
from ralgpu import dtypes as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ncols", [(1, 3), (31, 1), (129, 4), (4097, 2), (1000, 75), (70_001, 5)])
@pytest.mark.parametrize("tune", ["R=0", ""])
def test_masks_are_cleared(monkeypatch, n, ncols, tune):
    if tune:
        monkeypatch.setenv("RAL_FILTER_TUNE", tune)
    rng = np.random.default_rng(n)
    spec = [(D.GDF_INT32, rng.integers(-5, 5, n).astype(np.int32), rng.random(n) >= 0.3) for _ in range(ncols)]
    query = "LogicalFilter(condition=[>($0, 0)])"
    frame = H.to_device(spec)
    for _ in range(2):  # the second call's scratch and masks hold the first one's
        got = R.process_filter(frame, query)
        exp = O.process_filter(H.to_oracle(spec), query)
        for g, e in zip(got, exp):
            O.update_null_count(e)
            H.assert_columns_equal(g, e)


def test_text_masks_are_cleared():
    import ctypes as C
    import torch
    rows = 1000
    text = "".join(f"{i}|{'' if i % 3 else i}\n" for i in range(rows)).encode()
    dev = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    outs = [R.Column.empty(D.GDF_INT32, rows, with_valid=True) for _ in range(2)]
    for o in outs:
        o.valid.fill_(0xFF)
    structs = [o.to_c() for o in outs]
    arr = (C.POINTER(type(structs[0])) * 2)(*[C.pointer(s) for s in structs])
    fd, pr, n = (C.c_int32 * 2)(D.GDF_INT32, D.GDF_INT32), (C.c_int32 * 2)(0, 1), C.c_int32(0)
    q = b"LogicalFilter(condition=[<($0, 500)])"
    assert R.lib().ral_text_scan_filter(dev.data_ptr(), dev.numel(), b"|", b"\n", 0, fd, 2, pr, 2, q,
                                        C.cast(arr, C.c_void_p), C.byref(n)) == 0
    assert n.value == 500
    bits = np.unpackbits(outs[1].valid.cpu().numpy(), bitorder="little")
    np.testing.assert_array_equal(bits[:500], (np.arange(500) % 3 == 0).astype(np.uint8))
    assert not bits[500:rows].any()
