"""Division by (X + c) at raw words near 0 and near r, whose replayed sums meet r and 2r:
every word equals the oracle's, so every quotient is canonical.  Coefficients of the sort
lie around each chunk, warp and block edge, and shifts are small integers, halves and one
whose four-part products end just above r."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import dev, host

pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
MONT = (1 << 256) % R
FOUND = 0x6B3587F04D011E3CEDD0F9684DF03793FB947FC7FD27B6A39740630C7C31DB70  # raw words
SHIFTS = [(-k * MONT) % R for k in range(1, 9)] + [(k * MONT) % R for k in (1, 2)] + \
         [(-MONT * pow(2, -1, R)) % R, FOUND, (R - FOUND) % R]


def words(vals):
    return np.array([[(v >> (64 * j)) & (2**64 - 1) for j in range(4)] for v in vals], dtype=np.uint64)


def check(pp, O, p, c):
    d = dev(p)
    pp.div_xplusc_(d, dev(words([c])))
    assert O.first_diff(host(d), O.div_xplusc(p, words([c])[0])) == -1, hex(c)


@pytest.mark.parametrize("top", [R - 1, R - 5])
def test_found_examples(pp, O, cuda, top):
    check(pp, O, words([0, 0, 0, top, 5, 0, 0, 0]), (-MONT) % R)
    check(pp, O, words([0, 0, 0, R - 1, 1 << 63]), FOUND)


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 128, 129, 1024, 1025, 5000, 311297, 1000003])
def test_edge_words(pp, O, cuda, n):
    rng = np.random.default_rng(n)
    near = [0, 0, 0, 1, 2, 5, 1 << 63, 1 << 160, R - 1, R - 2, R - 5, R - (1 << 63), R - (1 << 160)]
    for c in SHIFTS:
        p = words(near)[rng.integers(0, len(near), n)]
        check(pp, O, p, c)
