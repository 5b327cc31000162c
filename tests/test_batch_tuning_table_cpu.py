"""The batch tuning table: an entry that names no version of the items' code, or another one, is not used."""
import json
import os
import subprocess
import sys

import pytest

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# prints the names of the item function generated for one program, and the program's table key
_SCRIPT = """
import re, sys
sys.path[:0] = [%r, %r]
import ralgpu
from ralgpu import workloads as W
t = W.batched_mix(1, seed=3)[0]
pp = ralgpu.parse_project_plan(t.dtypes, t.project)
ins = [ralgpu.Column.empty(t.dtypes[c], 100, device="cpu") for c in pp["input_columns"]]
for c in ins:
    c.null_count = 1
outs = [ralgpu.Column.empty(dt, 100, device="cpu") for dt in pp["evaluated_dtypes"]]
args = (pp["left"], pp["right"], pp["outputs"], pp["final_output_positions"], pp["operators"], pp["unary_operators"],
        pp["left_scalars"], pp["right_scalars"])
b = ralgpu.Batch()
b.add(outs, ins, *args)
print(re.search(r"void (ral_item_\\w+)\\(", b.debug_source(compile=False)[0]).group(1), ralgpu.batch_tune_key(outs, ins, *args))
""" % (_ROOT, os.path.join(_ROOT, "blazingdb-ral_gb300"))


def _item(cache_dir):
    out = subprocess.run([sys.executable, "-c", _SCRIPT], env=dict(os.environ, RAL_JIT_CACHE_DIR=str(cache_dir)),
                         capture_output=True, text=True, check=True)
    return out.stdout.split()


@pytest.mark.parametrize("suffix", ["", "@0123456789abcdef"])
def test_entries_of_other_code_are_not_used(tmp_path, suffix):
    default, key = _item(tmp_path)
    with open(tmp_path / "autotune.json", "w") as f:
        json.dump({key + suffix: [16, 2, 0.1, 1]}, f)
    assert _item(tmp_path)[0] == default
