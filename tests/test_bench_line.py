"""The bench line keeps its measurements where a CPU leg cannot run."""
import argparse
import json
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


@pytest.mark.parametrize("failing", [(), ("cpu_baseline_sample",), ("hc_error_vs_reference",)])
def test_a_missing_cpu_leg_costs_its_field(monkeypatch, failing):
    import bench

    def refuse(*args, **kwargs):
        raise RuntimeError("no generated C:\n run the generator")

    monkeypatch.setattr(bench, "cpu_baseline_sample", lambda args: ({"value": 1.0}, {}))
    monkeypatch.setattr(bench, "hc_error_vs_reference", lambda keep, precision: {"hc_bg_max_rel": 0.0})
    for name in failing:
        monkeypatch.setattr(bench, name, refuse)
    cpu, hc_error = bench.cpu_fields(argparse.Namespace(precision="fp64"))
    gone = {"unavailable": "RuntimeError: no generated C: run the generator"}
    assert cpu == (gone if "cpu_baseline_sample" in failing else {"value": 1.0})
    assert hc_error == (None if "cpu_baseline_sample" in failing else gone if failing else {"hc_bg_max_rel": 0.0})
    json.dumps([cpu, hc_error])
