"""Performance cases: calls that a program makes of this framework, as a measuring harness runs them.

Every case goes through the public surface (gbz.py or the C ABI it loads)
on one long-lived context, as a proving service holds one.  Inputs are
device-resident unless the case says otherwise.  Sizes follow the
configurations of the benchmark and of the tests: the plain prover from
2^10 to 2^24 witnesses, mixed batches, the N-party commitment scheme, the
R1CS front end, the distributed commitments, and the encode, Merkle and
sumcheck calls a program makes by themselves.

All outputs are field elements, hashes or transcript bytes: whole numbers
that are the same on every correct run.
"""
import ctypes
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "shorter-and-faster-post-quantum-secure-scalable-collaborative-snarks_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gbz  # noqa: E402

P = gbz.P
DEV = gbz.MEM_DEVICE
PCS_RATES = [[4], [4], [4, 4], [4, 4]]  # the reference's coPCS test (main.cpp:54)
MASK_L = 333                            # mask length of the R1CS front end (coPIOP.cpp:1392-1393)
FMUL_OPS = 8                            # one F_{p^2} multiply: four products, four additions

_held = {}


def _context():
    """The process's context, on a stream that torch work can be queued on too."""
    if not _held:
        _held["stream"] = torch.cuda.Stream()
        _held["ctx"] = gbz.Context(0)
        _held["ctx"].set_stream(_held["stream"].cuda_stream)
    return _held["ctx"], _held["stream"]


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest proof the tests make: a serving system's floor of latency
        {"name": "prove_2e10_r4", "do": "prove", "logn": 10, "rate": 4},
        # benchmark configuration 1, one ordinary proof
        {"name": "prove_2e18_r4", "do": "prove", "logn": 18, "rate": 4},
        # benchmark configuration 2, the headline proof
        {"name": "prove_2e24_r2", "do": "prove", "logn": 24, "rate": 2},
        # benchmark configuration 3: 64 mixed proofs from pinned host memory
        {"name": "batch_64_mixed", "do": "batch", "count": 64, "lo": 12, "hi": 20, "rate": 4, "mix": 3},
        # benchmark configuration 4: the coPCS test of 16 parties (commit, claim, whole opening)
        {"name": "copcs_16x2e24", "do": "copcs", "N": 16, "logM": 24},
        # the same protocol at a size of the tests, where rounds and launches count
        {"name": "copcs_8x2e16", "do": "copcs", "N": 8, "logM": 16},
        # the R1CS front end's two sumcheck phases for 2^20 gates
        {"name": "piop_16x2e20", "do": "piop", "N": 16, "logM": 20},
        # the distributed commitment of the witness and its opening
        {"name": "dpcs_16x2e20", "do": "dpcs", "N": 16, "logA": 20, "batch": 16, "rate": 4},
        # Whir_Commit_initial for a caller that keeps codeword and whole tree
        {"name": "whir_commit_2e20_r4", "do": "commit", "logm": 20, "rate": 4},
        # decoding direction: an inverse transform of an odd log length
        {"name": "ifft_2e21", "do": "fft", "logn": 21, "inverse": True},
        # the distributed cubic sumcheck alone
        {"name": "party_sumcheck_16x2e20", "do": "sumcheck", "N": 16, "logM": 20, "cubic": True},
        # aggregation of an odd number of claims before a shared WHIR opening
        {"name": "aggregate_3x3_2e21", "do": "aggregate", "k": 3, "c": 3, "logn": 21},
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        c = _draw_one(rng)
        if c not in known:
            return c


def _draw_one(rng):
    do = rng.choice(["prove", "prove", "batch", "copcs", "piop", "dpcs", "commit", "fft", "sumcheck", "aggregate"])
    if do == "prove":
        rate = rng.choice([2, 4, 8])
        return {"do": do, "logn": rng.randint(10, 25 - rate.bit_length() + 1), "rate": rate}
    if do == "batch":
        lo = rng.randint(10, 14)
        return {"do": do, "count": int(round(2 ** rng.uniform(1.5, 6))), "lo": lo, "hi": rng.randint(lo, 20),
                "rate": rng.choice([2, 4]), "mix": rng.randint(0, 10 ** 6)}
    if do == "copcs":
        N = rng.choice([4, 8, 16])
        return {"do": do, "N": N, "logM": rng.randint({4: 14, 8: 16, 16: 16}[N], {4: 21, 8: 23, 16: 24}[N])}
    if do == "piop":
        N, logM = rng.choice([(8, 16), (8, 17), (8, 18), (8, 19), (16, 16), (16, 17), (16, 18), (16, 19), (16, 20)])
        return {"do": do, "N": N, "logM": logM}
    if do == "dpcs":
        return {"do": do, "N": rng.choice([8, 16]), "logA": rng.randint(13, 20), "batch": rng.choice([4, 8, 16]),
                "rate": rng.choice([2, 4])}
    if do == "commit":
        rate = rng.choice([2, 4, 8])
        return {"do": do, "logm": rng.randint(8, 25 - rate.bit_length()), "rate": rate}
    if do == "fft":
        return {"do": do, "logn": rng.randint(8, 25), "inverse": rng.random() < 0.5}
    if do == "sumcheck":
        N = rng.choice([4, 8, 16, 32])
        return {"do": do, "N": N, "logM": rng.randint(8, 25 - N.bit_length()), "cubic": rng.random() < 0.6}
    return {"do": do, "k": rng.randint(2, 6), "c": rng.randint(1, 5), "logn": rng.randint(10, 22)}


# ----------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(0x5EED0000 + seed)


def _base(g, n):
    """n base-field values (imaginary words zero), as the witnesses are."""
    v = torch.zeros((n, 2), dtype=torch.int64, device="cuda")
    v[:, 0] = torch.randint(0, P, (n,), dtype=torch.int64, device="cuda", generator=g)
    return v


def _ext(g, *shape):
    return torch.randint(0, P, (*shape, 2), dtype=torch.int64, device="cuda", generator=g)


def _host_ext(rng, *shape):
    return rng.integers(0, P, size=(*shape, 2), dtype=np.uint64)


def _bytes(n):
    return torch.zeros(n, dtype=torch.uint8, device="cuda")


def _shares(ctx, v, N):
    """Packed shares of v for N parties (N x 4 |v| / N)."""
    M = v.shape[0]
    out = torch.empty((N, 4 * M // N, 2), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ctx.check(gbz.lib.gbz_secret_shares(ctx.h, v.data_ptr(), M, N, 0, 1, out.data_ptr(), DEV))
    return out


def _fmul(a, b):
    """One F_{p^2} product of host values (pairs of ints)."""
    (x, y), (u, v) = a, b
    return ((x * u - y * v) % P, (x * v + y * u) % P)


def _ints(v):
    return tuple(int(t) for t in v)


def _batch_logs(case):
    r = np.random.default_rng(case["mix"])
    return [int(x) for x in r.integers(case["lo"], case["hi"] + 1, size=case["count"])]


def prepare(case, seed):
    ctx, stream = _context()
    s = {"case": case, "seed": seed, "ctx": ctx, "stream": stream}
    _PREPARE[case["do"]](s, case, seed, ctx)
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state["case"]["do"]](state, state["ctx"])


# the plain prover, witness and transcript on the device
def _prepare_prove(s, case, seed, ctx):
    s["w"] = _base(_gen(seed), 1 << case["logn"])
    s["tr"] = _bytes(gbz.transcript_bytes(case["logn"], case["rate"]))


def _run_prove(s, ctx):
    return ctx.prove(s["w"], s["case"]["logn"], s["case"]["rate"], 1 + s["seed"], out=s["tr"])


# independent proofs of mixed sizes, witnesses and transcripts in pinned host memory
def _prepare_batch(s, case, seed, ctx):
    logs = _batch_logs(case)
    rng = np.random.default_rng(seed)
    w = torch.zeros((sum(1 << x for x in logs), 2), dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    w[:, 0] = rng.integers(0, P, size=w.shape[0], dtype=np.uint64)
    sizes = [gbz.transcript_bytes(x, case["rate"]) for x in logs]
    s["tr"] = torch.zeros(sum(sizes), dtype=torch.uint8, pin_memory=True).numpy()
    at = np.cumsum([0] + [1 << x for x in logs])
    to = np.cumsum([0] + sizes)
    s["ws"] = [w[at[i]:at[i + 1]] for i in range(len(logs))]
    s["out"] = [s["tr"][to[i]:to[i + 1]] for i in range(len(logs))]
    s["logs"], s["rates"] = logs, [case["rate"]] * len(logs)
    s["seeds"] = [1 + seed + i for i in range(len(logs))]


def _run_batch(s, ctx):
    ctx.prove_batch(s["ws"], s["logs"], s["rates"], s["seeds"], out=s["out"])
    return s["tr"]


# the N-party commitment, its claim and the whole opening
def _prepare_copcs(s, case, seed, ctx):
    N, M = case["N"], 1 << case["logM"]
    g = _gen(seed)
    _, _, rnd = gbz.pcs_schedule(N, M, PCS_RATES)
    s["shares"] = _shares(ctx, _base(g, M), N)
    s["random"] = _shares(ctx, _base(g, rnd * (N // 4)), N)
    s["r"] = _ext(g, case["logM"] + 1)
    s["K"] = torch.zeros(2, dtype=torch.int64, device="cuda")
    s["fs0"] = _ext(g, 1)[0]
    s["fs"] = torch.zeros_like(s["fs0"])
    s["roots"] = _bytes(32 * N)
    s["root"] = _bytes(32)
    s["rates"] = [np.array([r[k] if len(r) > k else 0 for r in PCS_RATES], dtype=np.int32) for k in (0, 1)]
    h = _copcs_commit(s, ctx)
    n = ctypes.c_uint64(0)
    ctx.check(gbz.lib.gbz_pcs_open_full_bytes(h, ctypes.byref(n)))
    gbz.lib.gbz_pcs_free(h)
    s["tr"] = _bytes(n.value)


def _copcs_commit(s, ctx):
    h = ctypes.c_void_p()
    r0, r1 = s["rates"]
    ctx.check(gbz.lib.gbz_pcs_commit(ctx.h, s["case"]["N"], 1 << s["case"]["logM"], len(PCS_RATES), r0.ctypes.data,
                                     r1.ctypes.data, s["shares"].data_ptr(), s["random"].data_ptr(), DEV,
                                     ctypes.byref(h), s["roots"].data_ptr(), s["root"].data_ptr()))
    return h


def _run_copcs(s, ctx):
    nr = s["r"].shape[0]
    h = _copcs_commit(s, ctx)
    try:
        ctx.check(gbz.lib.gbz_pcs_claim(ctx.h, h, s["r"].data_ptr(), nr, s["K"].data_ptr(), DEV))
        with torch.cuda.stream(s["stream"]):
            s["fs"].copy_(s["fs0"])
        g = gbz.Prng(1 + s["seed"])
        flags = ctypes.c_uint32(0)
        ctx.check(gbz.lib.gbz_pcs_open_full(ctx.h, h, s["r"].data_ptr(), nr, s["K"].data_ptr(), s["fs"].data_ptr(),
                                            ctypes.addressof(g), ctypes.byref(flags), s["tr"].data_ptr(),
                                            s["tr"].numel(), DEV))
    finally:
        gbz.lib.gbz_pcs_free(h)
    return [s["roots"], s["root"], s["K"], s["fs"], s["tr"], flags.value]


# the R1CS front end: both sumcheck phases of N parties
def _piop_shape(case):
    N, logM = case["N"], case["logM"]
    n = (1 << (logM + 1)) // N               # vL, vR, vO share length (2^(logM - 1) constraints)
    nws = (1 << (logM + 2)) // N             # the witness's share length
    lv, lw = n.bit_length() - 1, (2 * nws).bit_length() - 1 - 5
    d1 = [16, 1 << ((lv - 4) // 2), 1 << (lv - 4 - (lv - 4) // 2), 2]
    d2 = [1 << (lw // 2), 1 << (lw - lw // 2), 32]
    rows = (1 << logM) // N
    nw = (N * rows // (N // 4)) + 2 * (d1[0] * d1[1] * d1[2])
    return n, nw, rows, d1, d2


def _prepare_piop(s, case, seed, ctx):
    N, logM = case["N"], case["logM"]
    n, nw, rows, d1, d2 = _piop_shape(case)
    g, rng = _gen(seed), np.random.default_rng(seed)
    s["v"] = [_shares(ctx, _base(g, 1 << (logM - 1)), N) for _ in range(3)]
    s["masks"] = _ext(g, N, 12)
    s["R1"], s["R2"] = _ext(g, N, 4 * sum(d1)), _ext(g, N, 2 * sum(d2))
    s["w"] = _ext(g, N, nw)
    # the circuit: two left wires and one right wire a constraint, its output in a row of its own
    m, total = 1 << (logM - 1), 1 << logM
    ptrs, cols = [], []
    for wires in (2, 1, 0):
        row = rng.integers(0, total, size=wires * m) if wires else np.arange(m) + (total - m)
        con = np.tile(np.arange(m), max(wires, 1))
        order = np.argsort(row, kind="stable")
        cols.append(con[order])
        ptrs.append(np.concatenate([[0], np.cumsum(np.bincount(row, minlength=total))]))
    s["r1cs"] = gbz.R1cs(ctx, N, rows, logM - 1, ptrs, cols)
    s["d1"], s["d2"] = np.array(d1, dtype=np.int32), np.array(d2, dtype=np.int32)
    s["K"], s["fs0"] = _ext(g, 1)[0], _ext(g, 1)[0]
    s["fs"] = torch.zeros_like(s["fs0"])
    i64 = dict(dtype=torch.int64, device="cuda")
    s["cl1"], s["cl2"] = torch.zeros((4, len(d1) + 2, 2), **i64), torch.zeros((5, len(d2) + 2, 2), **i64)
    s["ip1"], s["ip2"] = torch.zeros((N, 4 * sum(d1), 2), **i64), torch.zeros((N, 2 * sum(d2), 2), **i64)
    s["ip3"], s["abc"] = torch.zeros((N, 12, 2), **i64), torch.zeros((3, 2), **i64)
    s["tr1"] = _bytes(gbz.lib.gbz_piop_phase1_bytes(N, n, s["d1"].ctypes.data, len(d1)))
    s["tr2"] = _bytes(gbz.lib.gbz_piop_phase2_bytes(N, s["d2"].ctypes.data, len(d2)))


def _run_piop(s, ctx):
    N = s["case"]["N"]
    n, nw, _, d1, d2 = _piop_shape(s["case"])
    f1, f2 = ctypes.c_uint32(0), ctypes.c_uint32(0)
    vL, vR, vO = s["v"]
    with torch.cuda.stream(s["stream"]):
        s["fs"].copy_(s["fs0"])
        ctx.check(gbz.lib.gbz_piop_phase1(ctx.h, N, n, vL.data_ptr(), vR.data_ptr(), vO.data_ptr(),
                                          s["masks"].data_ptr(), s["R1"].data_ptr(), s["d1"].ctypes.data, len(d1),
                                          s["fs"].data_ptr(), s["cl1"].data_ptr(), s["ip1"].data_ptr(), None, None,
                                          ctypes.byref(f1), s["tr1"].data_ptr(), s["tr1"].numel(), DEV))
        point = s["cl1"][0, 1:].contiguous()
        evals = s["cl1"][:3, 0].contiguous()
        ctx.check(gbz.lib.gbz_piop_phase2(ctx.h, N, nw, s["w"].data_ptr(), s["masks"].data_ptr(), s["r1cs"].h, MASK_L,
                                          s["R2"].data_ptr(), point.data_ptr(), evals.data_ptr(),
                                          s["d1"].ctypes.data, len(d1), s["d2"].ctypes.data, len(d2),
                                          s["K"].data_ptr(), s["fs"].data_ptr(), s["cl2"].data_ptr(),
                                          s["abc"].data_ptr(), s["ip2"].data_ptr(), s["ip3"].data_ptr(), None, None,
                                          ctypes.byref(f2), s["tr2"].data_ptr(), s["tr2"].numel(), DEV))
    return [s[k] for k in ("cl1", "ip1", "tr1", "cl2", "abc", "ip2", "ip3", "tr2", "fs")] + [f1.value, f2.value]


# the distributed commitment of N parties and its opening beside a zero index commitment
def _prepare_dpcs(s, case, seed, ctx):
    N, A, B, rate = case["N"], 1 << case["logA"], case["batch"], case["rate"]
    g = _gen(seed)
    S, L = A // B, A // B * rate
    i64 = dict(dtype=torch.int64, device="cuda")
    s["arr"], s["arr2"] = _base(g, N * A), _base(g, N * A)
    # polynomial 0 is committed by the pass, polynomial 1 is the zero index commitment made here
    s["cd"], s["cw"] = torch.zeros((2, N, B, S, 2), **i64), torch.zeros((2, N, B, L, 2), **i64)
    s["lv"] = _bytes(N * (2 * L - 1) * 32)
    s["roots"], s["root"] = np.zeros((N, 32), dtype=np.uint8), np.zeros(32, dtype=np.uint8)
    zero = torch.zeros_like(s["arr"])
    torch.cuda.synchronize()
    ctx.check(gbz.lib.gbz_dpcs_batch_commit(ctx.h, N, A, s["arr"].data_ptr(), zero.data_ptr(), rate, B,
                                            s["cd"][1].data_ptr(), s["cw"][1].data_ptr(), None, None, None, DEV))
    npt = sum(x.bit_length() - 1 for x in (S, B, N))
    s["pts"], s["ys"] = _ext(g, 2, npt), torch.zeros((2, 2), **i64)
    s["fs0"] = _ext(g, 1)[0]
    s["fs"] = torch.zeros_like(s["fs0"])
    lN = N.bit_length() - 1
    na = N * S // ((1 << (lN - lN // 2)) * (1 << (lN // 2)))
    s["ao"], s["bo"], s["K"] = torch.zeros((na, 2), **i64), torch.zeros((na, 2), **i64), torch.zeros(2, **i64)
    s["wcw"], s["wroot"] = torch.zeros((na * rate, 2), **i64), np.zeros(32, dtype=np.uint8)
    s["tr"] = _bytes(gbz.lib.gbz_dpcs_open_bytes(N, 2, rate))


def _run_dpcs(s, ctx):
    c = s["case"]
    N, A, B, rate = c["N"], 1 << c["logA"], c["batch"], c["rate"]
    flags = ctypes.c_uint32(0)
    ctx.check(gbz.lib.gbz_dpcs_batch_commit(ctx.h, N, A, s["arr"].data_ptr(), s["arr2"].data_ptr(), rate, B,
                                            s["cd"].data_ptr(), s["cw"].data_ptr(), s["lv"].data_ptr(),
                                            s["roots"].ctypes.data, s["root"].ctypes.data, DEV))
    with torch.cuda.stream(s["stream"]):
        s["fs"].copy_(s["fs0"])
    ctx.check(gbz.lib.gbz_dpcs_open(ctx.h, N, 2, B, A // B, rate, s["cd"].data_ptr(), s["cw"].data_ptr(),
                                    s["pts"].data_ptr(), s["ys"].data_ptr(), 0, rate, s["fs"].data_ptr(),
                                    s["ao"].data_ptr(), s["bo"].data_ptr(), s["K"].data_ptr(), s["wcw"].data_ptr(),
                                    s["wroot"].ctypes.data, ctypes.byref(flags), s["tr"].data_ptr(),
                                    s["tr"].numel(), DEV))
    return [s[k] for k in ("cd", "cw", "lv", "roots", "root", "ao", "bo", "K", "wcw", "wroot", "tr", "fs")] + [flags.value]


# RS encoding and the whole Merkle tree
def _prepare_commit(s, case, seed, ctx):
    m, L = 1 << case["logm"], case["rate"] << case["logm"]
    s["arr"] = _base(_gen(seed), m)
    s["cw"] = torch.zeros((L, 2), dtype=torch.int64, device="cuda")
    s["lv"] = _bytes((L // 2 - 1) * 32)


def _run_commit(s, ctx):
    ctx.check(gbz.lib.gbz_whir_commit(ctx.h, s["arr"].data_ptr(), s["arr"].shape[0], s["case"]["rate"],
                                      s["cw"].data_ptr(), s["lv"].data_ptr(), DEV))
    return [s["cw"], s["lv"]]


# one transform in place (each pass transforms what the last one left)
def _prepare_fft(s, case, seed, ctx):
    s["x"] = _ext(_gen(seed), 1 << case["logn"])


def _run_fft(s, ctx):
    return ctx.fft(s["x"], s["case"]["logn"], s["case"]["inverse"])


# the distributed sumcheck of N parties, its claim a true one
def _prepare_sumcheck(s, case, seed, ctx):
    N, M, cubic = case["N"], 1 << case["logM"], case["cubic"]
    g = _gen(seed)
    form = gbz.SC_CUBIC if cubic else gbz.SC_QUADRATIC
    s["form"] = form
    s["v"] = [_ext(g, N * M) for _ in range(3 if cubic else 2)]
    s["wt"] = _host_ext(np.random.default_rng(seed), N) if cubic else None
    torch.cuda.synchronize()
    y = (0, 0)
    for p in range(N):
        h = ctx.sumcheck_round(form, [v[p * M:(p + 1) * M] for v in s["v"]])
        at = [sum(int(x[k]) for x in h) + int(h[-1][k]) for k in (0, 1)]
        t = _fmul(_ints(at), _ints(s["wt"][p]) if cubic else (1, 0))
        y = ((y[0] + t[0]) % P, (y[1] + t[1]) % P)
    s["y"] = y
    s["fs"] = _host_ext(np.random.default_rng(seed + 1), 1)[0]


def _run_sumcheck(s, ctx):
    r = ctx.party_sumcheck(s["form"], s["v"], s["case"]["N"], w=s["wt"], offset=4, fs=s["fs"],
                           prng=1 + s["seed"], y=s["y"])
    return [r[k] for k in ("polys", "challenges", "fin", "y", "fs")]


# aggregate_claims of k arrays at c points
def _prepare_aggregate(s, case, seed, ctx):
    g, n = _gen(seed), 1 << case["logn"]
    s["arrays"] = [_ext(g, n) for _ in range(case["k"])]
    s["ptrs"] = (ctypes.c_void_p * case["k"])(*[a.data_ptr() for a in s["arrays"]])
    s["points"] = _host_ext(np.random.default_rng(seed), case["c"], case["logn"])
    s["arr"], s["b"] = torch.empty_like(s["arrays"][0]), torch.empty_like(s["arrays"][0])
    s["K"], s["ch"] = np.zeros(2, dtype=np.uint64), gbz.fe_array(case["k"] + case["c"])
    s["sums"] = gbz.fe_array(case["k"] * case["c"])


def _run_aggregate(s, ctx):
    g = gbz.Prng(1 + s["seed"])
    ctx.check(gbz.lib.gbz_whir_aggregate_claims(ctx.h, s["case"]["k"], ctypes.cast(s["ptrs"], ctypes.c_void_p),
                                                1 << s["case"]["logn"], s["case"]["c"], s["points"].ctypes.data,
                                                ctypes.addressof(g), s["arr"].data_ptr(), s["b"].data_ptr(),
                                                s["K"].ctypes.data, s["ch"].ctypes.data, s["sums"].ctypes.data, DEV))
    return [s[k] for k in ("arr", "b", "K", "ch", "sums")]


_PREPARE = {"prove": _prepare_prove, "batch": _prepare_batch, "copcs": _prepare_copcs, "piop": _prepare_piop,
            "dpcs": _prepare_dpcs, "commit": _prepare_commit, "fft": _prepare_fft, "sumcheck": _prepare_sumcheck,
            "aggregate": _prepare_aggregate}
_RUN = {"prove": _run_prove, "batch": _run_batch, "copcs": _run_copcs, "piop": _run_piop, "dpcs": _run_dpcs,
        "commit": _run_commit, "fft": _run_fft, "sumcheck": _run_sumcheck, "aggregate": _run_aggregate}


def exact(case, seed):
    """Every output is a whole number (field elements, hashes, transcripts), equal on every correct run."""
    return None


# ------------------------------------------------------------------- work
def _butterflies(L):
    """Radix-2 multiplies of a transform of length L."""
    return L // 2 * (L.bit_length() - 1)


def _prove_work(logn, rate):
    n = 1 << logn
    mults = _butterflies(n * rate) // 2        # a base-field witness packs into half the length
    mults += 4 * n                             # the sumcheck of the witness with the eq table
    m = n
    L = n * rate
    while m > 16:                              # WHIR iterations: fold by 4, encode at twice the rate
        mults += 4 * m
        m, L = m // 4, L // 2
        mults += _butterflies(L)
    return {"bytes": 16 * n + gbz.transcript_bytes(logn, rate), "flops": FMUL_OPS * mults}


def work(case):
    """Bytes: every input read once and every output written once.  flops:
    integer operations of the field multiplies, FMUL_OPS each."""
    do = case["do"]
    if do == "prove":
        return _prove_work(case["logn"], case["rate"])
    if do == "batch":
        each = [_prove_work(x, case["rate"]) for x in _batch_logs(case)]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if do == "copcs":
        N, M = case["N"], 1 << case["logM"]
        S = 4 * M // N
        Bs = S // 16
        # 31 rows a party: inverse transform, coset, transform of 4 Bs; the opening's folds and encodes of one row
        mults = N * 31 * (_butterflies(Bs) + Bs + _butterflies(4 * Bs)) + N * (31 * Bs + 4 * _butterflies(4 * Bs))
        return {"bytes": 16 * N * S, "flops": FMUL_OPS * mults}
    if do == "piop":
        N = case["N"]
        n, nw, _, d1, d2 = _piop_shape(case)
        mults, m = 0, 2 * n
        for d in d1:                           # four vectors a block: inverse of d, transform of 4 d, products, fold
            mults += N * (m // d) * 4 * (_butterflies(max(d, 2)) + _butterflies(4 * d) + 4 * d)
            m //= d
        m = 2 * nw
        for d in d2:
            mults += N * (m // d) * 2 * (_butterflies(max(d, 2)) + _butterflies(2 * d) + 2 * d)
            m //= d
        return {"bytes": 16 * N * (3 * n + nw) + (12 << case["logM"]), "flops": FMUL_OPS * mults}
    if do == "dpcs":
        N, A, B, rate = case["N"], 1 << case["logA"], case["batch"], case["rate"]
        L = A // B * rate
        mults = B * _butterflies(N * L) + 2 * N * B * L
        return {"bytes": 16 * N * A * 3 + 16 * N * B * L + 32 * N * 2 * L, "flops": FMUL_OPS * mults}
    if do == "commit":
        m, L = 1 << case["logm"], case["rate"] << case["logm"]
        return {"bytes": 16 * m + 16 * L + 16 * L, "flops": FMUL_OPS * (_butterflies(L) // 2 + L // 2)}
    if do == "fft":
        n = 1 << case["logn"]
        return {"bytes": 32 * n, "flops": FMUL_OPS * _butterflies(n)}
    if do == "sumcheck":
        n, k = case["N"] << case["logM"], 3 if case["cubic"] else 2
        return {"bytes": 16 * k * n, "flops": FMUL_OPS * n * (12 if case["cubic"] else 4)}
    n, k, c = 1 << case["logn"], case["k"], case["c"]
    return {"bytes": 16 * n * (k + 2), "flops": FMUL_OPS * n * (k * c + 2 * c + k)}
