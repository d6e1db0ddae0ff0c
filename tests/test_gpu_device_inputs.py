"""Party inputs in device memory, on a 16-byte boundary and a word off it (a
tensor's slice): the same commitments, claims and transcripts as from the host."""
import ctypes

import numpy as np
import pytest

from conftest import rand_fe

pytestmark = pytest.mark.gpu


def device(torch, a, shift):
    """Device address of a's words, `shift` words behind a boundary, and what keeps it."""
    w = torch.from_numpy(np.ascontiguousarray(a).view(np.int64).reshape(-1).copy()).cuda()
    t = torch.zeros(w.numel() + 2, dtype=torch.int64, device="cuda")
    t[shift:shift + w.numel()] = w
    return t.data_ptr() + 8 * shift, t


@pytest.mark.parametrize("shifts", [(0, 0, 0), (1, 1, 1), (0, 1, 0), (1, 0, 1)])
@pytest.mark.parametrize("form", ["quadratic", "cubic"])
def test_cosumcheck(gbz, ctx, form, shifts):
    torch = pytest.importorskip("torch")
    cubic, N, n, deg = form == "cubic", 8, 1 << 12, [64, 16]
    rng = np.random.default_rng(7)
    p = [rand_fe(rng, N * n) for _ in range(3 if cubic else 2)]
    R = rand_fe(rng, N * (4 if cubic else 2) * sum(deg))
    r1, r2 = (rand_fe(rng, 12), rand_fe(rng, 1)) if cubic else (None, None)
    K, Kr, fs = (rand_fe(rng, 1)[0] for _ in range(3))
    f = gbz.SC_CUBIC if cubic else gbz.SC_QUADRATIC
    _, flags, want, _ = gbz.cosumcheck(ctx, f, N, p[0], p[1], R, K, Kr, deg, p3=p[2] if cubic else None, r1=r1, r2=r2,
                                       fs=fs)
    dp = [device(torch, x, s) for x, s in zip(p, shifts)]
    rest = [device(torch, x, 0) if x is not None else (None, None) for x in (R, r1, r2, K, Kr, fs)]
    d = np.array(deg, dtype=np.int32)
    tr = torch.zeros(len(want), dtype=torch.uint8, device="cuda")
    cl = torch.zeros(5 * 2 * (len(deg) + 2), dtype=torch.int64, device="cuda")
    got_flags = ctypes.c_uint32()
    torch.cuda.synchronize()
    (R_, r1_, r2_, K_, Kr_, fs_) = (x[0] for x in rest)
    for _ in range(2):
        rest[5][1][:2] = torch.from_numpy(fs.view(np.int64)).cuda()
        torch.cuda.synchronize()
        ctx.check(gbz.lib.gbz_cosumcheck(ctx.h, f, N, n, dp[0][0], dp[1][0], dp[2][0] if cubic else None, R_, r1_,
                                         12 if cubic else 0, r2_, K_, Kr_, d.ctypes.data, len(deg), fs_,
                                         cl.data_ptr(), ctypes.byref(got_flags), tr.data_ptr(), len(want),
                                         gbz.MEM_DEVICE))
        ctx.synchronize()
        assert tr.cpu().numpy().tobytes() == want and got_flags.value == flags


@pytest.mark.parametrize("shifts", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_commit(gbz, ctx, shifts):
    torch = pytest.importorskip("torch")
    N, M, rates = 4, 1 << 14, [(4,), (4,), (4, 4), (4, 4)]
    rng = np.random.default_rng(3)
    _, _, rnd = gbz.pcs_schedule(N, M, rates)
    shares, random = rand_fe(rng, 4 * M), rand_fe(rng, N * rnd)
    com, want, leader = gbz.pcs_commit(ctx, N, M, rates, shares, random)
    data = com.data(N - 1)
    com.free()
    (s, _s), (r, _r) = device(torch, shares, shifts[0]), device(torch, random, shifts[1])
    torch.cuda.synchronize()
    r0, r1 = gbz._rates(rates)
    h = ctypes.c_void_p()
    roots = torch.zeros((N, 32), dtype=torch.uint8, device="cuda")
    ctx.check(gbz.lib.gbz_pcs_commit(ctx.h, N, M, len(rates), r0.ctypes.data, r1.ctypes.data, s, r, gbz.MEM_DEVICE,
                                     ctypes.byref(h), roots.data_ptr(), None))
    com = gbz.PcsCommitment(ctx, h, N, M, rates)
    assert np.array_equal(roots.cpu().numpy(), want)
    assert all(np.array_equal(a, b) for a, b in zip(com.data(N - 1), data))
    com.free()
