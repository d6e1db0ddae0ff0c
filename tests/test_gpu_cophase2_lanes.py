"""Phase 2 on both sides of the limits where the number of lanes an output
changes (block length, 2^14 and 2^16 outputs): whole folds against exact
integers, which fit Python's for a few outputs and numpy's sums for all."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


def fold(v, L, j):
    re = im = 0
    for k in range(len(L)):
        (a, b), (c, d) = (int(x) for x in v[j * len(L) + k]), (int(x) for x in L[k])
        re, im = re + a * c - b * d, im + a * d + b * c
    return re % P, im % P


@pytest.mark.parametrize("logout", [0, 1, 13, 14, 15, 16, 17])
@pytest.mark.parametrize("logd", [0, 1, 2, 3, 4, 5, 6])
def test_lanes(ctx, logd, logout):
    rng = np.random.default_rng(logd * 32 + logout)
    v, L = rand_fe(rng, 1 << (logd + logout)), rand_fe(rng, 1 << logd)
    v[:1 << logd] = P - 1  # the largest words
    out = ctx.coSumcheck_phase2(v, L)
    picks = {0, (1 << logout) - 1, *(int(x) for x in rng.integers(0, 1 << logout, size=64))}
    for j in picks:
        assert tuple(int(x) for x in out[j]) == fold(v, L, j), j
    # the sum of all outputs is the fold of the sums: every output takes part
    sums = [[sum(int(x) for x in v[k::1 << logd, c]) % P for c in (0, 1)] for k in range(1 << logd)]
    want = fold(np.array(sums, dtype=np.uint64), L, 0)
    assert tuple(sum(int(x) for x in out[:, c]) % P for c in (0, 1)) == want
