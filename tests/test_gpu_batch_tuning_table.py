"""The batch tuning table: an entry that the autotuner of this build wrote is used by later processes."""
import json

import pytest

import ralgpu as R
from ralgpu import workloads as W
from test_batch_tuning_table_cpu import _item

pytestmark = pytest.mark.gpu


def test_a_recorded_entry_is_used(tmp_path, monkeypatch):
    default, key = _item(tmp_path)
    monkeypatch.setenv("RAL_JIT_CACHE_DIR", str(tmp_path))
    t = W.batched_mix(1, seed=3)[0]
    pp = R.parse_project_plan(t.dtypes, t.project)
    ins = [R.Column.empty(t.dtypes[c], 1000) for c in pp["input_columns"]]
    for c in ins:
        c.data.fill_(1)
        c.null_count = 1
    outs = [R.Column.empty(dt, 1000) for dt in pp["evaluated_dtypes"]]
    R.autotune_program(outs, ins, pp["left"], pp["right"], pp["outputs"], pp["final_output_positions"], pp["operators"],
                       pp["unary_operators"], pp["left_scalars"], pp["right_scalars"])
    with open(tmp_path / "autotune.json") as f:
        table = json.load(f)
    mine = [k for k in table if k.startswith(key + "@")]
    assert mine
    with open(tmp_path / "autotune.json", "w") as f:
        json.dump({k: [16, 2, 0.1, 1] for k in mine}, f)
    assert _item(tmp_path)[0] != default
