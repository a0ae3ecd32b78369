"""The MSM workspace that is allocated lies within the bound that include/pp_ops.h states,
for the shortest lists (runs of four entries), ordinary ones and ones with rounds of pair
sums, plain and fixed-base."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# a process of its own: workspaces live as long as it, and each size needs a larger one
CODE = r"""
import ctypes, sys
sys.path.insert(0, %r)
import __graft_entry__ as g
import torch
pp = g.load_package()
L = pp.ppfr.lib()
L.pp_device_alloc_bytes.restype = ctypes.c_uint64
L.pp_msm_g1_window_bits.argtypes = [ctypes.c_uint64]

def bound(n, c, sets):
    w = 256 // c + 1
    entries, buckets = w * n, (w if sets is None else sets) << (c - 1)
    least = min(131 * entries, 16 * entries + 30e6) + 400 * buckets + 32 * 1024
    return least + 72 * entries + 128 * buckets if entries >= 1 << 20 else least

top = 1 << 20
points, scalars = pp.ppfr.g1_mul_gen(pp.random_fr(top, 1)), pp.random_fr(top, 2)
plain, fixed = torch.cuda.Stream(), torch.cuda.Stream()
seen = 0
for n in (1, 2, 129, 300, 512, 1000, 4096, 8192, 1 << 14, 1 << 15, 70000, 200003, top):
    p, s = points[:n].contiguous(), scalars[:n].contiguous()
    key = pp.ppfr.MsmBases(p)
    torch.cuda.synchronize()
    for stream, call, most in ((plain, lambda: pp.ppfr.msm_g1(p, s), bound(n, L.pp_msm_g1_window_bits(n), None)),
                               (fixed, lambda: key.msm(s), bound(n, key.window_bits, 1))):
        before = L.pp_device_alloc_bytes()
        with torch.cuda.stream(stream):
            call()
        stream.synchronize()
        used = L.pp_device_alloc_bytes() - before
        assert used <= most, (n, used, most)
        seen += used > 0
    key.close()
assert seen >= 16, seen
print("ok")
"""


def test_stated_bound(cuda):
    r = subprocess.run([sys.executable, "-c", CODE % ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
