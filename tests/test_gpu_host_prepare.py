"""After pp_ntt_prepare a host-endpoint transform has its tables: the first call allocates
nothing (its workspace comes from a device call of the same size), and a capture takes the
same passes as a direct call.  2^19, 2^20 and 2^22 have stored splits that host endpoints
leave, 2^18 has one that they keep."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# a process of its own: this one may hold the tables already
CODE = r"""
import ctypes, sys
sys.path.insert(0, %r)
import __graft_entry__ as g
import torch
pp = g.load_package()
L = pp.ppfr.lib()
L.pp_device_alloc_count.restype = ctypes.c_uint64
lg, inverse = int(sys.argv[1]), sys.argv[2] == "inverse"
n = 1 << lg
pp.ppfr.prepare(lg, inverse)
s = torch.cuda.Stream()
x = pp.random_fr(n, 7)
torch.cuda.synchronize()
with torch.cuda.stream(s):
    want = pp.ntt(x, inverse)
    s.synchronize()
    h, o, o2 = (pp.ppfr.empty_pinned(n) for _ in range(3))
    h.copy_(x)
    allocs, launches = L.pp_device_alloc_count(), pp.launch_count()
    pp.ppfr.ntt_host(h, inverse, out=o)
    s.synchronize()
    assert L.pp_device_alloc_count() == allocs, "allocated"
    passes = pp.launch_count() - launches
    assert torch.equal(o, want.cpu())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        launches = pp.launch_count()
        pp.ppfr.ntt_host(h, inverse, out=o2)
        captured = pp.launch_count() - launches
    graph.replay()
    torch.cuda.synchronize()
    assert captured == passes, (captured, passes)
    assert L.pp_device_alloc_count() == allocs
    assert torch.equal(o2, want.cpu())
print("ok", passes)
"""


@pytest.mark.parametrize("lg", [18, 19, 20, 22])
@pytest.mark.parametrize("direction", ["forward", "inverse"])
def test_first_host_call_has_its_tables(cuda, lg, direction):
    r = subprocess.run([sys.executable, "-c", CODE % ROOT, str(lg), direction], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
