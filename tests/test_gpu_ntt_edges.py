"""Transforms of extreme inputs at every length around the pass boundaries:
words at p - 1 and 0 in the patterns that drive the butterflies' sums to the
ends of their windows, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


def patterns(n, rng):
    top = np.full((n, 2), P - 1, dtype=np.uint64)
    alt = top.copy()
    alt[n // 2:] = 0                                     # first-stage differences at +-(p - 1)
    comb = np.where(rng.integers(0, 2, size=(n, 2)) == 1, np.uint64(P - 1), np.uint64(0))
    imp = np.zeros((n, 2), dtype=np.uint64)
    imp[n // 3] = (P - 1, P - 1)
    return [top, alt, comb, imp]


@pytest.mark.parametrize("logn", list(range(1, 21)))
def test_extreme_inputs(ctx, gbz, oracle, logn):
    rng = np.random.default_rng(logn)
    for x in patterns(1 << logn, rng):
        for inv in (False, True):
            assert np.array_equal(ctx.fft(x.copy(), logn, inv), oracle.fft(x.copy(), inv)), (logn, inv)


@pytest.mark.parametrize("logn", [21, 22, 23, 24])
def test_three_passes_equal_two(ctx, gbz, logn):
    """The default schedule of the long lengths against a two-pass shape."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(logn)
    x = torch.randint(0, P, (1 << logn, 2), dtype=torch.int64, device="cuda", generator=g)
    saved = gbz.ntt_get_shape(logn)
    got = []
    try:
        for shape in (saved, (logn // 2, 0, 1)):
            gbz.ntt_set_shape(logn, *shape)
            f, i = x.clone(), x.clone()
            torch.cuda.synchronize()
            ctx.fft(f, logn, False)
            ctx.fft(i, logn, True)
            ctx.synchronize()
            got.append((f, i))
    finally:
        gbz.ntt_set_shape(logn, *saved)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("rows", [1, 3])
def test_three_passes_of_padded_rows(ctx, gbz, rows):
    """Rows of 2^19 encoded at rate 4 (zero-padded transforms of 2^21) against
    one row at a time."""
    rng = np.random.default_rng(rows)
    x = rng.integers(0, P, size=(rows, 1 << 19, 2), dtype=np.uint64)
    got = ctx.Encode(x, 4, 1)
    for r in range(rows):
        assert np.array_equal(got[r], ctx.Encode(x[r:r + 1], 4, 1)[0])
