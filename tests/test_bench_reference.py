"""bench.py where the reference's library was not built: both arms still print
their line."""

import json
import sys

import bench
import oracle.oracle


def test_lines_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(oracle.oracle, "ref_available", lambda *a: False)
    assert "not built" in bench.cpu_baseline(1.0, 64)["unavailable"]
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
