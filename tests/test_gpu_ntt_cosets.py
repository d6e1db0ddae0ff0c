"""Padded transforms taken as cosets of a short one, on both sides of the
lengths (2^10) and rates (8) where that form begins, against the oracle."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


@pytest.mark.parametrize("logn", [1, 2, 3, 4, 5, 6, 7, 9, 10, 11])
@pytest.mark.parametrize("lograte", [1, 2, 3, 4, 7, 12])
def test_padded(ctx, oracle, logn, lograte):
    n, rng = 1 << logn, np.random.default_rng(100 * logn + lograte)
    for x in (rand_fe(rng, n), np.full((n, 2), P - 1, dtype=np.uint64)):
        pad = np.zeros((n << lograte, 2), dtype=np.uint64)
        pad[:n] = x
        assert np.array_equal(ctx.rs_encode(x, 1 << lograte), oracle.fft(pad, False))


@pytest.mark.parametrize("logn,lograte", [(3, 3), (9, 5), (10, 4)])
def test_padded_in_place(ctx, gbz, oracle, logn, lograte):
    """Input and output in one buffer keep to the form that allows it."""
    import torch
    n, L = 1 << logn, 1 << (logn + lograte)
    x = rand_fe(np.random.default_rng(logn), n)
    pad = np.zeros((L, 2), dtype=np.uint64)
    pad[:n] = x
    buf = torch.from_numpy(pad.view(np.int64).copy()).cuda()
    ctx.check(gbz.lib.gbz_rs_encode(ctx.h, buf.data_ptr(), n, 1 << lograte, buf.data_ptr(), gbz.MEM_DEVICE))
    ctx.synchronize()
    assert np.array_equal(buf.cpu().numpy().view(np.uint64), oracle.fft(pad, False))
