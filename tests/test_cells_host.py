"""The carry-chained field multiplies (csrc/fr.cuh, csrc/fq.cuh) compiled for
the host against the row forms, on random and all-ones / all-zero limbs."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT


def test_cells_match_rows(tmp_path):
    exe = str(tmp_path / "cells_host_check")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "cells_host_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, "100000"], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr
