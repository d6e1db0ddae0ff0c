"""Sums of products that are reduced once at the end: inputs whose words are
all at the ends of their range, so that every term is as large as it can be,
at the lengths where the split of the work changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


def vectors(fill, count, n):
    if fill == "largest":
        return [np.full((n, 2), P - 1, dtype=np.uint64) for _ in range(count)]
    ends = np.array([0, 1, P - 1, P - 2], dtype=np.uint64)
    rng = np.random.default_rng(count * n)
    return [ends[rng.integers(0, 4, (n, 2))] for _ in range(count)]


@pytest.mark.parametrize("fill", ["largest", "ends"])
@pytest.mark.parametrize("form", [0, 1, 2, 3])
@pytest.mark.parametrize("logm", [1, 9, 17])
def test_round_sums(ctx, oracle, fill, form, logm):
    vecs = vectors(fill, oracle.FORM_VECTORS[form], 1 << logm)
    b, r = vectors(fill, 2, 2)[0][0], vectors(fill, 1, 2)[0][1]
    bb = b if form >= 2 else None
    assert np.array_equal(ctx.sumcheck_round(form, [v.copy() for v in vecs], bb), oracle.sumcheck_round(form, vecs, bb))
    got = [v.copy() for v in vecs]
    ctx.sumcheck_round(form, got, bb, r)
    for g, f in zip(got, oracle.sumcheck_fold_many(vecs, r)):
        assert np.array_equal(g[: len(f)], f)


# the lanes of an output: one below 2^3 entries, eight, a warp from 2^5
# entries where there are fewer than 2^14 outputs
@pytest.mark.parametrize("fill", ["largest", "ends"])
@pytest.mark.parametrize("logd,lognout", [(0, 3), (2, 9), (3, 0), (3, 14), (4, 2), (4, 13), (5, 0), (5, 13), (5, 14),
                                          (10, 3), (10, 14)])
def test_cophase2_lanes(ctx, oracle, fill, logd, lognout):
    v, L = vectors(fill, 1, 1 << (logd + lognout))[0], vectors(fill, 1, 1 << logd)[0]
    assert np.array_equal(ctx.coSumcheck_phase2(v, L), oracle.cophase2(v, L))


@pytest.mark.parametrize("fill", ["largest", "ends"])
@pytest.mark.parametrize("N,length", [(4, 33), (1024, 3)])
def test_party_aggregate_sums(ctx, oracle, fill, N, length):
    msgs = np.stack(vectors(fill, N, length))
    b = vectors(fill, 1, N // 4)[0]
    assert np.array_equal(ctx.sumcheck_aggr(msgs, b), oracle.party_aggregate(msgs, b))
