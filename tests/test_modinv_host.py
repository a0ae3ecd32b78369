"""The divstep inversion (csrc/modinv.cuh) compiled for the host: batches against single
divsteps, and inverses at both limb widths against the binary GCD."""
from __future__ import annotations

import os
import subprocess

from conftest import ROOT


def test_batches_and_inverses(tmp_path):
    exe = str(tmp_path / "modinv_host_check")
    subprocess.run(["g++", "-O2", "-std=c++17", os.path.join(ROOT, "tests", "modinv_host_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr
