"""Bucket sums over equal runs of the sorted list: buckets inside a run, shared
by a few runs, by more than one thread joins and by more than one block joins,
runs that end exactly at a bucket, and hardly any entries.  The points are
known multiples a_i G, so the answer is (sum s_i a_i mod r) G."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev

pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001


def ints(t):
    a = t.cpu().numpy().view(np.uint64)
    return [sum(int(a[i, j]) << (64 * j) for j in range(4)) for i in range(a.shape[0])]


def words(vals):
    return dev(np.array([[(v >> (64 * j)) & (2**64 - 1) for j in range(4)] for v in vals], dtype=np.uint64))


def scalars(kind, n, rnd):
    if kind == "random":
        return rnd
    if kind == "equal":
        return [rnd[0]] * n
    if kind == "two values":
        return [rnd[i % 7 == 0] for i in range(n)]
    if kind == "bits":  # 0 and 1: one bucket holds every entry
        return [v & 1 for v in rnd]
    if kind == "sparse":
        return [v if i % 97 == 0 else 0 for i, v in enumerate(rnd)]
    if kind == "zero":
        return [0] * n
    return [(1 << 256) - 1 - (v & 0xFFFF) for v in rnd]  # above r: every window carries


@pytest.mark.parametrize("n", [1, 9, 1000, 25000])
@pytest.mark.parametrize("kind", ["random", "equal", "two values", "bits", "sparse", "zero", "high"])
def test_known_multiples(pp, cuda, n, kind):
    a = pp.random_fr(n, 11)
    points = pp.ppfr.g1_mul_gen(a)
    s = scalars(kind, n, ints(pp.random_fr(max(n, 2), 12))[:max(n, 2)])[:n]
    total = sum(x * y for x, y in zip(s, ints(a))) % R
    want = pp.ppfr.g1_mul_gen(words([total]))[0]
    sd = words(s)
    key = pp.ppfr.MsmBases(points)
    for got in (pp.ppfr.msm_g1(points, sd), key.msm(sd)):
        assert (got[:2].reshape(-1) == want).all()
    key.close()
