"""Set shapes against the library's own passes: balanced two-pass shapes that
stage as much as a CTA holds, with and without the tables of the first pass."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


def balanced(logn):
    k1 = (logn + 1) // 2
    k2 = logn - k1
    return k1, min(k1, max(1 if k2 < 13 else 0, min(13, logn - 8) - k2)), min(k2, max(0, min(12, logn - 8) - k1))


@pytest.mark.parametrize("tables", [1, 0])
@pytest.mark.parametrize("logn", [14, 18, 21, 23, 24])
def test_balanced_shape(gbz, ctx, logn, tables):
    x = rand_fe(np.random.default_rng(logn), 1 << logn)
    assert gbz.ntt_get_shape(logn)[0] == -1
    want = [ctx.fft(x.copy(), logn, inv) for inv in (False, True)]
    try:
        gbz.ntt_set_shape(logn, *balanced(logn))
        assert gbz.ntt_get_shape(logn) == balanced(logn)
        gbz.lib.gbz_ntt_full_twiddles(tables)
        got = [ctx.fft(x.copy(), logn, inv) for inv in (False, True)]
    finally:
        gbz.lib.gbz_ntt_full_twiddles(1)
        gbz.ntt_set_shape(logn, -1, -1, -1)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_autotune_long(gbz, ctx):
    try:
        shape, own, best = ctx.ntt_autotune(22, reps=2)
        assert gbz.ntt_get_shape(22) == shape and 0 < best <= own
        x = rand_fe(np.random.default_rng(22), 1 << 22)
        tuned = ctx.fft(x.copy(), 22, False)
    finally:
        gbz.ntt_set_shape(22, -1, -1, -1)
    assert np.array_equal(tuned, ctx.fft(x.copy(), 22, False))
