"""bench.py where the reference build is absent (it is made only where the reference's sources are): the
reference arm says so in its one line and ends normally, and the own arm still gives its figures."""
import json
import sys

import pytest

import bench


@pytest.fixture
def no_reference(monkeypatch):
    from oracle import oracle as O
    monkeypatch.setattr(O, "REF_BIN", "/nonexistent/cfdv_ref")


@pytest.mark.parametrize("workload", ["plate", "ramp"])
def test_reference_arm_prints_unavailable(no_reference, monkeypatch, capsys, workload):
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0", "--workload",
                                      workload])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "reference build missing" in line["unavailable"]


def test_own_arm_reports_no_cpu_baseline(no_reference):
    assert "reference build missing" in bench.cpu_baseline("plate")["unavailable"]
