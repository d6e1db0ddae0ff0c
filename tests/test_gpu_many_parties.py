"""Whole openings of 32 and 64 parties: the leader's tail passes its checks (the
one that the reference fails on every input aside), begins with the parties'
own opening, and a second opening in the same buffers gives the same bytes."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

RATES = [(4,), (4,), (4, 4), (4, 4)]
STEP3 = 32  # "Error in verification step 3", printed by the reference for every input


@pytest.mark.parametrize("N,logM", [(32, 17), (64, 18)])
def test_opening(gbz, ctx, oracle, N, logM):
    _, _, rnd = gbz.pcs_schedule(N, 1 << logM, RATES)
    shares, random, _ = oracle.copcs_party_shares(N, 1 << logM, rnd * N // 4, state=True)
    com, roots, _ = gbz.pcs_commit(ctx, N, 1 << logM, RATES, shares, random)
    rng = np.random.default_rng(N)
    r = rand_fe(rng, (N // 4).bit_length() - 1 + 5 + com.row_len.bit_length() - 1)
    K, fs = com.claim(r), rand_fe(rng, 1)[0]
    part, _ = com.open(r, K, fs)
    full, after, flags = com.open_full(r, K, fs, gbz.Prng(9))
    assert flags == STEP3 and full[: len(part)] == part
    again = com.open_full(r, K, fs, gbz.Prng(9))
    assert again[0] == full and np.array_equal(again[1], after) and again[2] == flags
    wrong = K.copy()
    wrong[0] ^= np.uint64(1)  # a claim that the parties' first message does not match
    with pytest.raises(gbz.GbzError):
        com.open(r, wrong, fs)
    com.free()
