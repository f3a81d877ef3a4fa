"""bench.py's reference arm is the reference or nothing."""
from __future__ import annotations

import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_reference_arm_without_the_reference(bind_mod):
    if os.path.exists(bind_mod.REF_LIB):
        pytest.skip("oracle/_ref is built")
    out = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                         capture_output=True, text=True, check=True, timeout=300).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"]
    assert "value" not in line
