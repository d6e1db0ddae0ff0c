"""Block sums of coSumcheck: the new evaluations of every block in one pass
(blocks of 2^3 to 2^10 entries, at least 2^11 entries in all) against the
oracle, on both sides of those limits and with words at the ends of their
range; inputs in device memory stay as they were."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = (1 << 61) - 1


@pytest.mark.parametrize("fill", ["largest", "ends"])
@pytest.mark.parametrize("logn,logd", [(11, 2), (10, 3), (11, 3), (12, 4), (14, 5), (13, 6), (15, 7), (12, 8), (13, 9),
                                       (10, 10), (11, 10), (13, 10), (12, 11)])
def test_block_sums(ctx, oracle, fill, logn, logd):
    n, d = 1 << logn, 1 << logd
    if fill == "largest":
        vs = [np.full((n, 2), P - 1, dtype=np.uint64) for _ in range(4)]
    else:
        ends = np.array([0, 1, P - 1, P - 2], dtype=np.uint64)
        vs = [ends[np.random.default_rng(logn * 16 + logd + v).integers(0, 4, (n, 2))] for v in range(4)]
    p1, p2, p3, b1 = vs
    # blocks that the cubic form skips; a last one with one entry set
    for blk in range(0, n // d, 4):
        p1[blk * d:(blk + 1) * d] = 0
    p1[n - d:] = 0
    p1[n - 1, 1] = 1
    H, H4 = oracle.cophase1(p1, p2, p3, b1, logd)
    assert np.array_equal(ctx.coSumcheck_phase1(p1, p2, logd), H)
    assert np.array_equal(ctx.coSumcheck_phase1(p1, p2, logd, p3, b1), H4)


def test_device_inputs_stay(gbz, ctx):
    torch = pytest.importorskip("torch")
    N, n, degs = 4, 1 << 12, [16, 8]
    rng = np.random.default_rng(77)
    draw = lambda *shape: rng.integers(0, P, shape + (2,), dtype=np.uint64)
    p1, p2, p3, R = draw(N, n), draw(N, n), draw(N, n), draw(N, 4 * sum(degs))
    r1, r2, K = draw(12), draw(0), draw(2)
    want = gbz.cosumcheck(ctx, gbz.SC_CUBIC, N, p1, p2, R, K[0], K[1], degs, p3=p3, r1=r1, r2=r2)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in (p1, p2, p3, R)]
    deg = np.array(degs, dtype=np.int32)
    fs, cl, flags = np.zeros(2, dtype=np.uint64), np.zeros((4, 4, 2), dtype=np.uint64), ctypes.c_uint32(0)
    ptr = lambda x: ctypes.c_void_p(x.data_ptr() if hasattr(x, "data_ptr") else x.ctypes.data)
    nb = gbz.lib.gbz_cosumcheck_transcript_bytes(gbz.SC_CUBIC, N, ptr(deg), len(degs))
    tr = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.check(gbz.lib.gbz_cosumcheck(ctx.h, gbz.SC_CUBIC, N, n, ptr(dev[0]), ptr(dev[1]), ptr(dev[2]), ptr(dev[3]),
                                     ptr(r1), 12, ptr(r2), ptr(K[0]), ptr(K[1]), ptr(deg), len(degs), ptr(fs),
                                     ptr(cl), ctypes.byref(flags), ptr(tr), nb, gbz.MEM_DEVICE))
    assert tr.cpu().numpy().tobytes() == want[2] and flags.value == want[1]
    for got, x in zip(dev, (p1, p2, p3, R)):
        assert np.array_equal(got.cpu().numpy().view(np.uint64), x)
