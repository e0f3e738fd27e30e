"""bench.py's reference arm where the reference's core is not there to run: it says
so in one line and times nothing in its place."""
import argparse
import json

import pytest

import bench


@pytest.mark.parametrize("workload,why", [("fe15648_1024x1024", "not built here"),
                                          ("fe6173_4096x4096", "no instrument filter")])
def test_reference_arm_without_the_reference(monkeypatch, capsys, workload, why):
    monkeypatch.setattr(bench, "cpu_kind", lambda name: "port")
    monkeypatch.setattr(bench, "CpuPool", None)  # nothing may run
    args = argparse.Namespace(workload=workload, steps=1, warmup=1, npix=0, sample=16,
                              bounds="auto")
    assert bench.reference_arm(args) == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and why in line["unavailable"] and "value" not in line
