"""The reference arm of bench.py where the reference's build is missing: one JSON
line that says why there is no number, and no error."""
import argparse
import json

import bench_reference


def test_reference_arm_without_the_reference_build(tmp_path, monkeypatch, capsys):
    monkeypatch.setattr(bench_reference, "HARNESS", str(tmp_path / "ref_harness"))
    bench_reference.run(argparse.Namespace(n=32, order=3, steps=20))
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    r = json.loads(lines[0])
    assert r["impl"] == "reference" and r["unavailable"] and "\n" not in r["unavailable"]
