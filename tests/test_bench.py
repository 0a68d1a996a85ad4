"""bench.py on a machine without the compiled reference: the CPU figure comes
from the restatement, and the reference arm says why it has none."""
import argparse
import json

import pytest

import bench
from oracle import oracle as O


@pytest.fixture
def no_reference(monkeypatch):
    have = O.available
    monkeypatch.setattr(O, "available", lambda kind: kind != "ref" and have(kind))


def test_cpu_baseline_without_the_reference(no_reference):
    r = bench.cpu_baseline(6000, procs=1, ns=3)
    assert r["kind"] == "port" and r["cores"] == 1 and r["value"] > 0


def test_reference_arm_without_the_reference(no_reference, capsys):
    bench.reference_arm(argparse.Namespace(nt=None, warmup=1, steps=1, gpus=1))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libifosref" in line["unavailable"] and "value" not in line
