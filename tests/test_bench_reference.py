"""bench.py --impl reference without the reference's sources: one line that says
so, not a traceback."""
import argparse
import json

import pytest

import bench
import pyoracle


@pytest.mark.parametrize("workload", ["config4", "ragged8"])
def test_unavailable_line(workload, tmp_path, monkeypatch, capsys):
    monkeypatch.setattr(pyoracle, "REF_SRC", str(tmp_path / "absent"))
    monkeypatch.setattr(pyoracle, "ref_binary", lambda cfg: str(tmp_path / cfg))
    args = argparse.Namespace(workload=workload, steps=2, warmup=3, gpus=1, c4_nz=128)
    bench.run_reference(args, 1, 0)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "absent" in line["unavailable"]
