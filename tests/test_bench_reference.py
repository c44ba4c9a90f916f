"""The benchmark's reference arm without a reference library: one line that says
so."""

import importlib
import sys

from oracle import oracle


def test_missing_reference_is_one_line(sf, monkeypatch, tmp_path):
    bench = importlib.import_module("bench")
    monkeypatch.setattr(oracle, "REF_LIB_PATH", tmp_path / "lib.so")
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--steps", "20", "--warmup", "5"])
    args = bench.parse()
    line = bench.reference_arm(sf, args, sf.scenes.config1(n=args.size), 1, 0, 0)
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference"
    assert "\n" not in line["unavailable"]
