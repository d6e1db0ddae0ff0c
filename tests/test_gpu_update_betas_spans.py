"""The direct beta update where the entries of a lane change (1, 2 and 8, from
2^13 and 2^15 entries on) and at ragged ends of a block, against the oracle."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 31, 33, (1 << 13) - 1, 1 << 13, (1 << 13) + 65, (1 << 15) - 1, 1 << 15,
                                (1 << 15) + 257])
@pytest.mark.parametrize("l", [1, 7, 9, 256])
def test_spans(ctx, oracle, nb, l):
    rng = np.random.default_rng(nb + l)
    logN = 23  # long enough that no size here takes the sparse transform
    b, r = rand_fe(rng, nb), rand_fe(rng, 1)[0]
    q = rng.integers(0, 1 << logN, size=l).astype(np.int32)
    out, ch = ctx.update_betas(b, q, 1 << logN, r)
    ob, och = oracle.update_betas(b, q, 1 << logN, r)
    assert np.array_equal(out, ob) and np.array_equal(ch, och)
