"""bench.py where the reference's own program is not built: the reference arm says so
in its line, and the product's line has a null baseline."""
import json
from argparse import Namespace

import bench
from oracle import ref_inputs as RI

ARGS = Namespace(steps=5, warmup=3, ref_seconds=1.0, ref_single_steps=1, gpus=1, scene="dam_small")


def test_reference_arm_without_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(RI, "ref_available", lambda dim: False)
    bench.run_reference_arm(ARGS, 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "ref_mph3d" in line["unavailable"] and "value" not in line


def test_baseline_without_the_reference(monkeypatch):
    monkeypatch.setattr(RI, "ref_available", lambda dim: False)
    assert bench.cpu_baseline_sample(ARGS) is None
