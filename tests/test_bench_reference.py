"""bench.py's reference arm runs the reference's own code or says that it cannot:
a line with figures is never the restated oracle's."""
import argparse
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("workload", [2, 3])
def test_without_the_reference(monkeypatch, capsys, workload):
    monkeypatch.syspath_prepend(os.path.join(ROOT, "myers-gpu_b200"))
    monkeypatch.syspath_prepend(os.path.join(ROOT, "oracle"))
    monkeypatch.syspath_prepend(ROOT)
    monkeypatch.delenv("RANK", raising=False)
    import bench
    import oracle as orc
    monkeypatch.setattr(orc, "have_reference", lambda: False)
    monkeypatch.setattr(orc, "verify", lambda *a, **k: pytest.fail("the oracle in the reference's place"))
    bench.run_reference(argparse.Namespace(workload=workload, scale=1e-4, steps=2, warmup=1))
    line = json.loads(capsys.readouterr().out.splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
