"""The packaged tuning table is what the autotuner writes: a bucket for each of its sets of batches, and no bucket whose
configuration its own figures put behind the library's default, which is always among the candidates."""
import json
import os

from kolmo_gb300 import autotune, codec

TABLE = os.path.join(os.path.dirname(codec.__file__), "tuning_gb300.json")


def test_packaged_table_is_the_tuners():
    with open(TABLE) as f:
        t = json.load(f)
    assert t["generated_by"] == "kolmo_gb300/autotune.py"
    assert [b["workload"] for b in t["buckets"]] == [name for name, _ in autotune.BUCKETS]
    grid = autotune.candidate_grid()
    for b in t["buckets"]:
        assert {k: b[k] for k in autotune.CANDIDATES} in grid
        assert b["fwd_ms"] <= b["default_fwd_ms"], b["workload"]
