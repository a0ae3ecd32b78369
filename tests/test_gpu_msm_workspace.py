"""The MSM's optional workspace (rounds of pair sums): without room for it on the device a
call does with the smaller one and does not ask again; a buffer that a capture took is not
replaced by a larger one."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

N = 200003  # one round of pair sums: about 313 MB of workspace with it, 117 without

HEAD = r"""
import ctypes, sys
sys.path.insert(0, %r)
import __graft_entry__ as g
import torch
pp = g.load_package()
L = pp.ppfr.lib()
for f in (L.pp_device_alloc_count, L.pp_device_alloc_bytes):
    f.restype = ctypes.c_uint64
n = %d
points, scalars = pp.ppfr.g1_mul_gen(pp.random_fr(n, 1)), pp.random_fr(n, 2)
want = pp.ppfr.msm_g1(points, scalars).clone()
most = L.pp_device_alloc_bytes()
torch.cuda.synchronize()
s = torch.cuda.Stream()

def run(out=None):
    c, b = L.pp_device_alloc_count(), L.pp_device_alloc_bytes()
    with torch.cuda.stream(s):
        r = pp.ppfr.msm_g1(points, scalars, out=out)
    s.synchronize()
    assert torch.equal(r, want)
    return L.pp_device_alloc_count() - c, L.pp_device_alloc_bytes() - b
"""

# free memory in quarters of the larger size: too little for it, and too little beside it
FULL = HEAD + r"""
count, full = run()
assert count == 1, count
for quarters in (3, 5):
    s = torch.cuda.Stream()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    fill = torch.empty(free - full * quarters // 4, dtype=torch.uint8, device="cuda")
    count, less = run()
    assert count == 1 and less < full, (quarters, count, less, full)
    assert run() == (0, 0) and run() == (0, 0), quarters
    del fill
    torch.cuda.empty_cache()
    assert run() == (0, 0), quarters
print("ok")
"""

CAPTURE = HEAD + r"""
assert L.pp_msm_g1_set_window_bits(18, 16) == 0
count, between = run()
assert L.pp_msm_g1_set_window_bits(18, 0) == 0
out = torch.empty((3, 6), dtype=torch.int64, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=s):
    pp.ppfr.msm_g1(points, scalars, out=out)
assert run() == (0, 0), "the captured buffer was replaced"
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, want)
s = torch.cuda.Stream()
count, full = run()
assert between < full, (between, full)  # else the case shows nothing
print("ok")
"""


@pytest.mark.parametrize("code", [FULL, CAPTURE], ids=["no_room", "captured"])
def test_optional_workspace(cuda, code):
    r = subprocess.run([sys.executable, "-c", code % (ROOT, N)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
