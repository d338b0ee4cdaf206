"""The benchmark's reference arm reports the reference's own code or nothing."""
import argparse
import json
import os
import sys

import pytest

from conftest import ROOT


@pytest.mark.parametrize("workload", ["multishot", "square"])
def test_without_the_references_code_the_arm_is_unavailable(workload, monkeypatch, capsys):
    monkeypatch.syspath_prepend(ROOT)
    monkeypatch.syspath_prepend(os.path.join(ROOT, "oracle"))
    import bench
    import refrun
    assert workload in bench.WORKLOADS
    monkeypatch.setattr(refrun, "available", lambda w, fast=False: False)
    monkeypatch.setattr(sys, "argv", ["bench.py"])
    args = argparse.Namespace(impl="reference", gpus=1, steps=3, warmup=3, workload=workload)
    assert bench.run_reference_arm(args) in (0, None)
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
