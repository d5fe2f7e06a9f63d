"""The reference arm of the benchmark never times anything but the reference."""
import argparse
import importlib.util
import json
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_without_the_reference_the_arm_says_so(monkeypatch, capsys, oracle):
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    monkeypatch.setenv("RANK", "0")
    assert bench.run_reference_arm(argparse.Namespace(n=10_000, steps=1, warmup=0, gpus=1)) == 0
    line = json.loads(capsys.readouterr().out)
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference" and line["unavailable"]
