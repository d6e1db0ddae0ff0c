"""Codewords stored in the parties' layout by the transform's last pass, at
lengths of one, two and three passes, against a plain transform of each row."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,logS,rate,batch", [(8, 0, 8, 4), (8, 1, 4, 4), (8, 7, 2, 4), (64, 4, 4, 4), (8, 9, 4, 8),
                                               (16, 7, 4, 4), (16, 15, 4, 4), (64, 13, 4, 4)])
def test_layout(ctx, gbz, N, logS, rate, batch):
    S, L = 1 << logS, rate << logS
    rng = np.random.default_rng(N + logS)
    arr = rand_fe(rng, N * batch * S).reshape(N, batch * S, 2)
    cw = gbz.dpcs_batch_commit(ctx, arr, arr, rate, batch)[1]
    for k in range(batch):
        g = np.zeros((N * L, 2), dtype=np.uint64)
        g[: N * S] = arr[:, k * S:(k + 1) * S].transpose(1, 0, 2).reshape(N * S, 2)
        X = ctx.fft(g, (N * L).bit_length() - 1, False).reshape(N, N, L // N, 2)  # [m][r][j]
        assert np.array_equal(cw[:, k], X.transpose(1, 0, 2, 3).reshape(N, L, 2))


def test_short_codewords_are_refused(ctx, gbz):
    a = np.zeros((16, 4, 2), dtype=np.uint64)
    with pytest.raises(gbz.GbzError):
        gbz.dpcs_batch_commit(ctx, a, a, 4, 4)
