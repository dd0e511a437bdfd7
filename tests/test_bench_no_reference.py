"""Where the reference's sources are absent the benchmark says so, on one line, instead of failing."""
import argparse
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402
from oracle import oracle  # noqa: E402


def test_reference_arm_without_its_library(monkeypatch, capsys):
    monkeypatch.setattr(oracle, "REF_SO", os.path.join(ROOT, "oracle", "_ref", "absent.so"))
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference_arm(argparse.Namespace(gpus=1, steps=3, warmup=3, procs=1))
    lines = capsys.readouterr().out.strip().splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and "absent.so" in line["unavailable"]


def test_nothing_missing_with_the_library(monkeypatch):
    monkeypatch.setattr(oracle, "REF_SO", os.path.abspath(__file__))
    assert bench.reference_missing() is None
