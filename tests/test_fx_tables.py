"""The committed integer tables of csrc/fx64.cuh (exp and log on the integer
pipes) are what their generator writes."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dennou-ccm_gb300", "csrc")


def test_tables_match_generator():
    pytest.importorskip("mpmath")
    out = subprocess.run([sys.executable, os.path.join(CSRC, "gen_fx_tables.py")], check=True,
                         capture_output=True, text=True, cwd=CSRC).stdout
    with open(os.path.join(CSRC, "fx_tables.cuh")) as f:
        assert f.read() == out
