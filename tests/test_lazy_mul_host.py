"""fr_mul (csrc/fr.cuh) of two factors below 2r, compiled for the host: what the lazy
kernels pass it.  No build option selects another multiply: the row forms are wrong for
such pairs."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT


@pytest.mark.parametrize("variant", [None, 0, 9, 13])
def test_lazy_factors(tmp_path, variant):
    exe = str(tmp_path / "lazy_mul_check")
    define = [] if variant is None else ["-DPP_MUL_VARIANT=%d" % variant]
    subprocess.run(["g++", "-O2", "-std=c++17", *define, os.path.join(ROOT, "tests", "lazy_mul_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr


def test_flags_select_no_multiply():
    code = ("import importlib.util as u; s = u.spec_from_file_location('b', %r); m = u.module_from_spec(s);"
            "s.loader.exec_module(m); print(m.NVCC_FLAGS)" % os.path.join(ROOT, "ppopp26-artifact_gb300", "build.py"))
    flags = [subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, check=True,
                            env={**os.environ, **env}).stdout for env in ({}, {"PP_MUL_VARIANT": "9"})]
    assert flags[0] == flags[1]
