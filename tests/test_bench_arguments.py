"""Every command-line value that bench.py reads is one that it defines."""
import os
import re
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402


def test_arguments_are_defined(monkeypatch):
    monkeypatch.setattr(sys, "argv", ["bench.py"])
    read = set(re.findall(r"\bargs\.(\w+)", open(bench.__file__).read()))
    assert read <= set(vars(bench.parse())), read - set(vars(bench.parse()))
