"""bench.py --impl reference times the reference itself or nothing."""
import argparse
import json

import bench


def test_restatement_is_not_passed_off_as_the_reference(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_binary", lambda: ("oracle/_build/psst_oracle", "port"))
    monkeypatch.setattr(bench, "cpu_run", lambda *a: (_ for _ in ()).throw(AssertionError("ran the restatement")))
    bench.run_reference_arm(argparse.Namespace(workload="wedge3d_6M_tets", gpus=1, steps=3, warmup=3))
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
