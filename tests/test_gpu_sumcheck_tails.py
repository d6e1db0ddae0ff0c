"""The party sumcheck at the lengths around the one that its one-CTA tail
begins at (2^12 entries in all), Fiat-Shamir rounds and drawn rounds on either
side, against the oracle."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("fill", ["random", "largest"])
@pytest.mark.parametrize("N,logM,offset", [(1, 2, 0), (1, 3, 4), (2, 10, 4), (4, 10, 0), (4, 10, 10), (4, 11, 2), (2, 13, 4)])
def test_party_lengths(ctx, oracle, form, fill, N, logM, offset):
    rng = np.random.default_rng(10 * logM + N)
    n = N << logM
    vecs = [rand_fe(rng, n) if fill == "random" else np.full((n, 2), P - 1, np.uint64) for _ in range(2 + form)]
    w = rand_fe(rng, N) if form else None
    fs = rand_fe(rng, 1)[0]
    first = oracle.party_sumcheck(form, vecs, N, w=w, offset=offset, fs=fs, y=[0, 0])["polys"][0].astype(object)
    y = np.array([(first[:, c].sum() + first[-1, c]) % P for c in range(2)], dtype=np.uint64)  # H(0) + H(1)
    got = ctx.party_sumcheck(form, vecs, N, w=w, offset=offset, fs=fs, y=y)
    ref = oracle.party_sumcheck(form, vecs, N, w=w, offset=offset, fs=fs, y=y)
    for k in ("polys", "challenges", "fin", "fs", "y"):
        assert np.array_equal(got[k], ref[k]), k
    assert got["prng"].next() == ref["prng"].next()
