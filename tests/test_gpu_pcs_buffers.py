"""The device buffers that a context keeps from a freed commitment for the next
one: the next commitment's data and roots are those of a context that keeps
nothing, whatever happened to the first, and the buffers are given back."""
import threading

import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu

N, RATES = 4, [(4,), (4,), (4, 4), (4, 4)]  # 1024-entry rows at 2^14


def commit(gbz, c, logM, seed):
    rng = np.random.default_rng(seed)
    _, _, rnd = gbz.pcs_schedule(N, 1 << logM, RATES)
    return gbz.pcs_commit(c, N, 1 << logM, RATES, rand_fe(rng, 4 << logM), rand_fe(rng, rnd * N))


def contents(gbz, c, logM, seed):
    com, roots, leader = commit(gbz, c, logM, seed)
    out = [roots, leader] + [x for p in range(N) for x in com.data(p)]
    com.free()
    return out


@pytest.mark.parametrize("between", ["same", "other_size", "two_live", "other_context", "thread", "stream"])
def test_next_commitment(gbz, between):
    fresh = gbz.Context(0)
    want = contents(gbz, fresh, 14, 2)
    fresh.close()
    c = gbz.Context(0)
    com, _, _ = commit(gbz, c, 15 if between == "other_size" else 14, 1)
    other = None
    if between == "two_live":
        other, _, _ = commit(gbz, c, 14, 3)
    if between == "other_context":  # buffers another context worked on are not kept
        other = gbz.Context(0)
        r = rand_fe(np.random.default_rng(4), 64)[: 5 + (com.row_len.bit_length() - 1)]
        K = np.zeros(2, dtype=np.uint64)
        other.check(gbz.lib.gbz_pcs_claim(other.h, com.h, r.ctypes.data, r.shape[0], K.ctypes.data, gbz.MEM_HOST))
    if between == "stream":
        torch = pytest.importorskip("torch")
        s = torch.cuda.Stream()
        c.set_stream(s.cuda_stream)
    if between == "thread":
        t = threading.Thread(target=com.free)
        t.start()
        t.join()
    com.free()
    if between == "two_live":
        other.free()
    got = contents(gbz, c, 14, 2)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert c.sched_release() >= N * 32 * (2 * 4096 - 1)  # the column trees alone
    assert c.sched_release() == 0
    if between == "other_context":
        other.close()
    c.close()


def test_handle_freed_after_its_context(gbz, ctx):
    c = gbz.Context(0)
    com, _, _ = commit(gbz, c, 14, 1)
    c.close()
    com.free()
    assert np.array_equal(contents(gbz, ctx, 14, 2)[0], contents(gbz, ctx, 14, 2)[0])
