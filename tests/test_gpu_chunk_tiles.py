"""The scans' shared-memory chunk tiles (two elements per lane and tile): odd
chunk lengths, ragged last chunks and lanes past the vector, for every output
form of the grand product, and the same sizes for evaluation and division."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,short", [(4, 1), (5, 0), (5, 1), (5, 4), (7, 3), (8, 2)])
def test_tiles(pp, O, cuda, k, short):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    n = sms * 2 * 256 * k - short  # k elements per thread, the last thread `short` fewer
    x = pp.random_fr(n + 1, 40 + k)
    hx = host(x)
    want = O.gp_prefix(hx)  # want[i] = prod_{j<i}
    excl, incl = want[:n], want[1:]
    fn = pp.ppfr.lib().pp_gp_scan
    fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_uint64, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    xin = x[:n].contiguous()
    for form in ("excl", "incl", "both", "excl in place", "incl in place"):
        src = xin.clone()
        a, b = pp.ppfr.empty(n), pp.ppfr.empty(n)
        e = a if form in ("excl", "both") else src if form == "excl in place" else None
        i = b if form in ("incl", "both") else src if form == "incl in place" else None
        ptr = [None if t is None else t.data_ptr() for t in (src, e, i)]
        pp.ppfr.check(fn(ptr[0], ptr[1], ptr[2], n, None))
        cuda.cuda.synchronize()
        if e is not None:
            assert O.first_diff(host(e), excl) == -1, form
        if i is not None:
            assert O.first_diff(host(i), incl) == -1, form
        if "in place" not in form:
            assert np.array_equal(host(src), hx[:n]), form
    z = pp.random_fr(1, 41)
    y = pp.evaluate(xin, z)
    assert (host(y)[0] == O.evaluate(hx[:n], host(z)[0])).all()
    q = O.div_xplusc(hx[:n], host(z)[0])
    pp.div_xplusc_(xin, z)
    assert O.first_diff(host(xin), q) == -1
