"""The benchmark's reference arm where the reference's code is not built: one
line that says so, and no failure."""
from __future__ import annotations

import argparse
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402
from oracle import oracle as O  # noqa: E402


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(O, "ref_available", lambda: False)
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference(argparse.Namespace(gpus=1, steps=1, warmup=3, gaussians=1000))
    lines = capsys.readouterr().out.splitlines()
    assert len(lines) == 1
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["unavailable"]
