"""Fq arithmetic spread over lanes (csrc/fq_lanes.cuh) against the whole-lane
multiply, on random and edge limbs."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_spread_products(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fq_lanes_check")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a",
                    os.path.join(ROOT, "tests", "fq_lanes_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr
