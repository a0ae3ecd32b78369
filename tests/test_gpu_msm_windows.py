"""Window sums: two lanes to a segment or one, one or two launches of chunk
sums, ragged chunk blocks, for the smallest and the largest bucket sets.  The
points are known multiples a_i G, so the answer is (sum s_i a_i mod r) G."""
from __future__ import annotations

import pytest

from conftest import dev  # noqa: F401  (skips without a GPU)
from test_gpu_msm_runs import R, ints, scalars, words

pytestmark = pytest.mark.gpu


# buckets 2^(c-1); segments of four on two lanes up to c = 16, of four on one lane
# at 17, of eight at 19 and of sixteen at 20
@pytest.mark.parametrize("c", [6, 8, 10, 11, 12, 14, 16, 17, 19, 20])
@pytest.mark.parametrize("kind", ["random", "equal", "zero", "high"])
def test_fixed_and_plain(pp, cuda, c, kind):
    n = 700
    # equal points too: sums of equal and of opposite points in the trees
    ai = [v if i % 3 else 5 for i, v in enumerate(ints(pp.random_fr(n, 21)))]
    points = pp.ppfr.g1_mul_gen(words(ai))
    s = scalars(kind, n, ints(pp.random_fr(n, 22)))
    total = sum(x * y for x, y in zip(s, ai)) % R
    want = pp.ppfr.g1_mul_gen(words([total]))[0]
    key = pp.ppfr.MsmBases(points, window_bits=c)
    assert (key.msm(words(s))[:2].reshape(-1) == want).all()
    key.close()
    L = pp.ppfr.lib()
    assert L.pp_msm_g1_set_window_bits(10, c) == 0
    try:
        got = pp.ppfr.msm_g1(points, words(s))
    finally:
        L.pp_msm_g1_set_window_bits(10, 0)
    assert (got[:2].reshape(-1) == want).all()
