"""bench.py's host side."""
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench
from oracle import oracle


def test_reference_arm_without_the_compiled_reference(monkeypatch, capsys):
    """Where the reference has not been compiled, its arm says so in one line and ends well."""
    monkeypatch.setattr(oracle, "REF_SO", os.path.join(os.sep, "nonexistent", "libnextref.so"))
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--gpus", "1", "--steps", "2", "--warmup", "3"])
    assert bench.main() == 0
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libnextref.so" in line["unavailable"]


def test_own_arm_without_the_compiled_reference(monkeypatch):
    monkeypatch.setattr(oracle, "REF_SO", os.path.join(os.sep, "nonexistent", "libnextref.so"))
    reference, why = bench.compiled_reference()
    assert reference is None and "libnextref.so" in why


def test_sort_traffic_is_the_passes():
    """The sort stage reads and writes a 12-byte pair per pass; its digits come counted from the kernel of the keys."""
    assert bench.sort_bytes_per_body(bench.sort_passes(10, 1)) == 4 * 24
    assert bench.sort_bytes_per_body(bench.sort_passes(21, 1)) == 8 * 24
