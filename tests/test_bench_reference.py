"""The bench's reference arm where the reference pipeline is not built: one line
that says so, and no other program timed in its place."""
import json
import sys

from conftest import ROOT


def test_without_the_reference_the_arm_is_unavailable(monkeypatch, capsys):
    sys.path.insert(0, ROOT)
    import bench
    from oracle import binding as orc
    monkeypatch.setattr(orc, "ref_available", lambda: False)
    monkeypatch.setattr(bench, "port_sample", lambda *a, **k: (1.0, 1.0))
    bench.run_reference(type("A", (), {"ref_scale": 0.001, "warmup": 0, "steps": 1, "gpus": 1})(), 0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "oracle/_ref" in line["unavailable"]
    assert "value" not in line
