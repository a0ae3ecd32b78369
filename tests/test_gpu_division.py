"""Division by (X + c) against its recurrence q_(i-1) = p_i - c q_i, q_(n-1) = 0, checked
with the elementwise kernels: sizes at the edges of chunks, warps and blocks, and
shifts whose powers vanish or repeat."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import dev

pytestmark = pytest.mark.gpu

R = 0x73EDA753299D7D483339D80809A1D80553BDA402FFFE5BFEFFFFFFFF00000001
MONT = (1 << 256) % R


def element(v):
    v = v * MONT % R
    return dev(np.array([[(v >> (64 * j)) & (2**64 - 1) for j in range(4)]], dtype=np.uint64))


@pytest.mark.parametrize("c", [0, 1, R - 1, 12345678901234567890123])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 127, 128, 129, 1023, 1024, 1025, 311295, 311296, 311297, 1000003, 1 << 22])
def test_recurrence(pp, cuda, n, c):
    p = pp.random_fr(n, 31)
    q = p.clone()
    pp.ppfr.div_xplusc_(q, element(c))
    assert not q[-1].any()
    if n > 1:
        cq = pp.ppfr.fr_binary(pp.ppfr.FR_MUL, q[1:].contiguous(), element(c))
        want = pp.ppfr.fr_binary(pp.ppfr.FR_SUB, p[1:].contiguous(), cq)
        assert torch.equal(q[:-1], want)
