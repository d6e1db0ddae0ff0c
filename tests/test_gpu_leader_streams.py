"""The leader's delegations on streams beside the parties' rounds: with fewer
rounds than streams, as many, and more (a stream takes a second round), an
opening repeats byte for byte, begins with the parties' own opening and passes
the leader's checks; another opening right behind it in the same buffers changes nothing."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

N, LOGM = 4, 14


@pytest.mark.parametrize("rounds", [4, 5, 6, 7])
def test_opening_repeats(gbz, ctx, oracle, rounds):
    rates = [(4,), (4,)] + [(4, 4)] * (rounds - 2)
    rng = np.random.default_rng(rounds)
    _, _, rnd = gbz.pcs_schedule(N, 1 << LOGM, rates)
    shares, random, _ = oracle.copcs_party_shares(N, 1 << LOGM, rnd * N // 4, state=True)
    com, _, _ = gbz.pcs_commit(ctx, N, 1 << LOGM, rates, shares, random)
    r, r2 = (rand_fe(rng, 5 + com.row_len.bit_length() - 1) for _ in range(2))
    K, K2, fs = com.claim(r), com.claim(r2), rand_fe(rng, 1)[0]
    part, _ = com.open(r, K, fs)

    def full(point, claim):
        g = gbz.Prng(9)
        tr, after, flags = com.open_full(point, claim, fs, g)
        return tr, after.tobytes(), flags, bytes(g)

    want = full(r, K)
    assert want[0][: len(part)] == part
    for _ in range(3):
        full(r2, K2)
        assert full(r, K) == want
    com.free()
