"""Without the reference's sources `bench.py --impl reference` says so, and
gives no figure of something else in their place."""
import json

import pytest


def test_reference_arm_without_sources(monkeypatch, capsys):
    bench = pytest.importorskip("bench")
    from oracle import oracle as o
    monkeypatch.setattr(o, "build_ref", lambda *a, **k: None)
    monkeypatch.setattr(bench, "time_cpu_oracle", lambda *a, **k: pytest.fail("timed the oracle"))
    assert bench.run_reference(bench.parse_args(["--impl", "reference"])) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
