"""The server reserves each slot's workspace for what a bundle's calls take: a bundle
allocates nothing but its own memory, also at the smallest sizes, and a slot holds no more
beside the transform's buffer than the scans' chunk sums."""
from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


def counters(pp):
    L = pp.ppfr.lib()
    for f in (L.pp_device_alloc_count, L.pp_device_alloc_bytes):
        f.restype = ctypes.c_uint64
    return L.pp_device_alloc_count(), L.pp_device_alloc_bytes()


@pytest.mark.parametrize("min_lg,max_lg", [(3, 3), (3, 5), (5, 9), (10, 17), (18, 20)])
def test_reserved(pp, cuda, min_lg, max_lg):
    P, lam = pp.ppfr, 2
    make = lambda: P.Server(budget_bytes=4 << 30, slots=2, min_lg=min_lg, max_lg=max_lg, lam=lam)  # noqa: E731
    make().close()  # builds the tables
    count, total = counters(pp)
    srv = make()
    # two slots' buffers and nothing else
    after, reserved = counters(pp)
    assert after - count == 4
    n = 1 << max_lg
    scans = (reserved - total) // 2 - 32 * (n << lam)
    assert 0 < scans <= 32 * (n // 3 + 200), scans
    for lg in (min_lg, max_lg):
        before = counters(pp)[0]
        t = srv.submit(lg, seed=5)
        srv.wait(t)
        srv.release(t)
        assert counters(pp)[0] - before == 1, lg  # the bundle's own memory
    srv.close()
