"""The tile kernel's rounds: every radix 2^3 .. 2^11 as a first, a middle and a
last pass (one to four rounds, radix-4 and radix-2 ends), forward and inverse,
with plain, zero-padded and coset inputs.  2^18 points under each split equal
the same call under the default split bit for bit; the default split is held
against the oracle here and in test_gpu_ntt.py."""
from __future__ import annotations

import pytest

from conftest import host

pytestmark = pytest.mark.gpu

LG = 18
SPLITS = [(3, 4, 11), (11, 3, 4), (4, 11, 3), (5, 8, 5), (8, 5, 5), (6, 7, 5), (7, 5, 6), (5, 6, 7), (10, 8),
          (8, 10), (7, 11), (11, 7), (3, 5, 5, 5), (6, 3, 3, 6), (4, 4, 4, 6)]


@pytest.fixture(scope="module")
def expected(pp, O, cuda):
    pp.ppfr.set_split(LG)
    x = pp.random_fr(1 << LG, 77)
    want = {"ntt": pp.ntt(x), "intt": pp.intt(x)}
    assert O.first_diff(host(want["ntt"]), O.ntt(host(x))) == -1
    assert O.first_diff(host(want["intt"]), O.ntt(host(x), inverse=True)) == -1
    for lam in (1, 2, 3):
        want["lde", lam] = pp.lde(x[:1 << (LG - lam)].contiguous(), lam, pp.LDE_COEFFS)
        assert O.first_diff(host(want["lde", lam]), O.lde_coeffs(host(x)[:1 << (LG - lam)], lam)) == -1
    return x, want


@pytest.mark.parametrize("split", SPLITS)
def test_radices(pp, cuda, expected, split):
    x, want = expected
    try:
        pp.ppfr.set_split(LG, split)
        assert (pp.ntt(x) == want["ntt"]).all()
        assert (pp.intt(x) == want["intt"]).all()
        y = x.clone()
        assert (pp.ntt(y, out=y) == want["ntt"]).all()  # in place
        for lam in (1, 2, 3):
            got = pp.lde(x[:1 << (LG - lam)].contiguous(), lam, pp.LDE_COEFFS)
            assert (got == want["lde", lam]).all(), lam
    finally:
        pp.ppfr.set_split(LG, [9, 9])


@pytest.mark.parametrize("lg,split", [(6, (3, 3)), (7, (4, 3)), (8, (3, 5)), (9, (9,)), (10, (5, 5)), (11, (4, 7))])
def test_splits_of_small_sizes(pp, O, cuda, lg, split):
    """Single calls below 2^9 points follow a split that is set for them."""
    x = pp.random_fr(1 << lg, 5)
    try:
        pp.ppfr.set_split(lg, split)
        for inverse in (False, True):
            assert O.first_diff(host(pp.ntt(x, inverse)), O.ntt(host(x), inverse=inverse)) == -1
    finally:
        pp.ppfr.set_split(lg)


@pytest.mark.parametrize("split", [(11, 7), (7, 11), (8, 10), (9, 9)])
def test_host_endpoints_under_any_split(pp, cuda, expected, split):
    """Host endpoints leave splits with short row segments for the default one."""
    x, want = expected
    hx, ho = pp.ppfr.empty_pinned(1 << LG), pp.ppfr.empty_pinned(1 << LG)
    hx.copy_(x)
    try:
        pp.ppfr.set_split(LG, split)
        for key, inverse in (("ntt", False), ("intt", True)):
            pp.ppfr.ntt_host(hx, inverse, out=ho)
            cuda.cuda.synchronize()
            assert (ho == want[key].cpu()).all()
        lo = pp.ppfr.lde_host(hx[:1 << (LG - 2)].contiguous().pin_memory(), 2, pp.LDE_COEFFS)
        cuda.cuda.synchronize()
        assert (lo == want["lde", 2].cpu()).all()
    finally:
        pp.ppfr.set_split(LG, [9, 9])
