"""The benchmark's reference arm times the reference's own sorter or says that it is unavailable: never the restatement of
this repository under the reference's name."""
import json
import sys

import bench
import oracle as O


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(O, "ref_lib", lambda: None)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0", "--block-mib", "1"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
