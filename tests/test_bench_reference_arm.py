"""The benchmark's reference arm without an installed reference: it says so, and times nothing in its place."""

import argparse
import json


def test_reference_arm_without_the_reference(monkeypatch, tmp_path, capsys):
    import bench

    monkeypatch.setattr(bench, "REFERENCE_DIR", tmp_path / "_ref")
    assert bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=1), 1, 0) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not installed" in line["unavailable"] and set(line) == {"impl", "unavailable"}
