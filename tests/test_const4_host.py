"""The canonical four-part constant multiply (csrc/fr.cuh) compiled for the host, and the
division's replay over it: raw words near 0 and near r, shifts that leave the lazy form
at r and above."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT


def test_canonical_product_and_replay(tmp_path):
    exe = str(tmp_path / "const4_host_check")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "const4_host_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, "50000"], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr
