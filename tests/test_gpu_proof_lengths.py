"""Proofs of every length at which the sumcheck's split into two-round passes
and the one-CTA tail changes, against the oracle's transcript; and the
generator's seeding for seeds at the ends of their range."""
import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


def witness(logn, fill):
    n = 1 << logn
    if fill == "general":
        return rand_fe(np.random.default_rng(logn), n)
    w = np.zeros((n, 2), dtype=np.uint64)
    w[:, 0] = P - 1 if fill == "largest" else np.random.default_rng(logn).integers(0, P, n)
    return w


@pytest.mark.parametrize("fill", ["base", "general", "largest"])
@pytest.mark.parametrize("logn", [3, 4, 5, 6, 11, 12, 13, 14, 15, 16, 17])
def test_lengths(ctx, oracle, logn, fill):
    w = witness(logn, fill)
    want = oracle.prove(w, logn, 2, 7)
    assert ctx.prove(w, logn, 2, 7).tobytes() == bytes(want)


@pytest.mark.parametrize("seed", [0, 1, 2, 127773, 2147483646, 2147483647, 2147483648, 2147483649, 4294967295])
def test_seeds(ctx, oracle, seed):
    w = witness(5, "base")
    assert ctx.prove(w, 5, 4, seed).tobytes() == bytes(oracle.prove(w, 5, 4, seed))


@pytest.mark.parametrize("logn,rate", [(3, 2), (12, 4), (21, 2), (21, 4)])
def test_graphs_on_both_sides_of_the_split(gbz, logn, rate):
    c = gbz.Context(0)
    w = witness(logn, "base")
    c.set_graphs(False)
    want = [c.prove(w, logn, rate, s).tobytes() for s in (1, 2)]
    c.set_graphs(True)
    assert [c.prove(w, logn, rate, s).tobytes() for s in (1, 2, 1)] == want + want[:1]
    c.close()
