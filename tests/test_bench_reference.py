"""bench.py where the reference has not been built: the reference arm says so in
one line and exits 0, and the framework's own line goes out without a CPU
baseline instead of being lost after its measurement."""
import json
import sys

import pytest

import bench


@pytest.fixture
def no_reference(monkeypatch):
    from oracle import pyoracle

    def absent(self, kind="3d"):
        raise FileNotFoundError(bench.ROOT + "/oracle/_ref/libref3d.so")
    monkeypatch.setattr(pyoracle.Reference, "__init__", absent)


def test_reference_arm_is_unavailable(no_reference, monkeypatch, capsys):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--l0", "0.05"])
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "absent" in line["unavailable"]


def test_own_line_has_no_cpu_baseline(no_reference, monkeypatch):
    args = type("A", (), dict(workload="c2", cpu_steps=1, l0=0.05, restart=True, no_cpu=False))
    assert bench.cpu_baseline(args) is None
    monkeypatch.setattr(bench, "reference_cpu_steps",
                        lambda *a, **k: (2.0, 0.5, dict(cores=4, kind="reference", sample="one step")))
    assert bench.cpu_baseline(args)["value"] == 2.0
    args.no_cpu = True
    assert bench.cpu_baseline(args) is None
