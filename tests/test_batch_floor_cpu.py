"""The table that the batched floor is computed from is the one of this mix, with plausible counts, and gives the
floor that the profile summary states."""
import json
import os

import bench as B
from ralgpu import workloads as W


def test_floor_of_the_table_that_is_read():
    table = json.load(open(os.path.join(B.ROOT, "profiles", "batch_mix_counters.json")))
    meta = B.batch_mix_meta(256, W.SEED)
    assert [(p["rows"], p["bytes_per_row"]) for p in table["programs"]] == [(m["rows"], round(m["bytes_per_row"], 4)) for m in meta]
    assert all(0 <= p["fp64_per_row"] < p["inst_per_row"] for p in table["programs"])
    f = B.batch_floor(table, 2070.0, 6782.4)
    assert f["floor_ms"] == f["fp64_ms"] and 13.4 < f["fp64_ms"] < 13.8
    assert f["source"] == "profiles/batch_mix_counters.json"
    assert 6.3 < f["hbm_ms"] < 6.6 and f["floor_ms"] < f["per_program_floor_ms"] < 15.0
