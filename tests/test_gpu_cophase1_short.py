"""Block sums of blocks of 1, 2 and 4 entries (extended blocks of 2 to 16), in
launches of few and of many transforms, against the oracle."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logn", [2, 7, 13, 14, 15, 18])
@pytest.mark.parametrize("logd", [0, 1, 2])
def test_block_sums(ctx, oracle, logn, logd):
    rng = np.random.default_rng(logn * 4 + logd)
    p1, p2, p3, b1 = (rand_fe(rng, 1 << logn) for _ in range(4))
    p1[: 1 << logd] = 0
    H, H4 = oracle.cophase1(p1, p2, p3, b1, logd)
    assert np.array_equal(ctx.coSumcheck_phase1(p1, p2, logd), H)
    assert np.array_equal(ctx.coSumcheck_phase1(p1, p2, logd, p3, b1), H4)
