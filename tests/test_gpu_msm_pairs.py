"""Rounds of affine pair sums: one round (200003 points), two and three (2^20), with
points and scalars that make every kind of pair: distinct, equal, opposite and
infinite points, odd and empty buckets, one bucket with nearly everything.  The points
are known multiples a_i G, so the answer is (sum s_i a_i mod r) G."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
FEW = [0, 1, R - 1, 7, R - 7, 1 << 200]  # infinity, a point and its negative, another


def ints(t):
    a = t.cpu().numpy().view(np.uint64).astype(object)
    return a[:, 0] + (a[:, 1] << 64) + (a[:, 2] << 128) + (a[:, 3] << 192)


def words(vals):
    return dev(np.array([[(v >> (64 * j)) & (2**64 - 1) for j in range(4)] for v in vals], dtype=np.uint64))


def pick(values, n, seed):
    i = np.random.default_rng(seed).integers(0, len(values), n)
    return np.array(values, dtype=object)[i]


@pytest.mark.parametrize(
    "n, points, scalars",
    [(200003, "random", "random"), (200003, "few", "random"), (200003, "random", "few"),
     (200003, "few", "few"), (200003, "few", "bits"), (1 << 20, "random", "random"), (1 << 20, "few", "few")],
)
def test_pairs(pp, cuda, n, points, scalars):
    a = ints(pp.random_fr(n, 21)) if points == "random" else pick(FEW, n, 1)
    s = ints(pp.random_fr(n, 22)) if scalars == "random" else pick([0, 1] if scalars == "bits" else FEW, n, 2)
    base = pp.ppfr.g1_mul_gen(words(a))
    want = pp.ppfr.g1_mul_gen(words([int((a * s).sum()) % R]))[0]
    sd = words(s)
    key = pp.ppfr.MsmBases(base)
    for got in (pp.ppfr.msm_g1(base, sd), key.msm(sd)):
        assert (got[:2].reshape(-1) == want).all()
    key.close()
