"""What libgbz hands to its kernels, with the CUDA runtime replaced by
tests/fake_cudart.c in a child process (two devices, launches reported and not
run): pointers of the launching device's memory only, tables only after they
are filled, field elements on 16-byte boundaries, buffers given back.

CPU only.
"""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

PRELUDE = r"""
import ctypes, functools, re, subprocess, sys, threading, time
import numpy as np
sys.path[:0] = [%r]
fake = ctypes.CDLL(%r)
fake.cudaMalloc.argtypes = [ctypes.c_void_p, ctypes.c_size_t]

@functools.lru_cache(None)
def parameters(name):
    text = subprocess.run(["c++filt", name], capture_output=True, text=True, check=True).stdout.strip()
    text = text.replace("(anonymous namespace)", "")
    kernel = re.search(r"(\w+)(<[^(]*>)?\(", text).group(1)
    out, depth, cur = [], 0, ""
    for ch in text[text.index("(") + 1:text.rindex(")")] + ",":
        depth += (ch in "<(") - (ch in ">)")
        if ch == "," and not depth:
            out.append(cur.strip())
            cur = ""
        else:
            cur += ch
    return kernel, out

SCAN = {"PassArgs": 320, "CoVectors": 80}  # bytes of a struct that hold pointers

class Pointer:
    def __init__(self, value, kind):
        dev, freed, filled, size = ctypes.c_int(), ctypes.c_int(), ctypes.c_long(), ctypes.c_uint64()
        self.value, self.kind = value, kind
        self.known = bool(fake.fake_lookup(ctypes.c_void_p(value), ctypes.byref(dev), ctypes.byref(freed),
                                           ctypes.byref(filled), ctypes.byref(size)))
        self.device, self.freed = dev.value, bool(freed.value)

    def filled(self):
        filled = ctypes.c_long()
        x = [ctypes.byref(ctypes.c_int()) for _ in range(2)]
        fake.fake_lookup(ctypes.c_void_p(self.value), x[0], x[1], ctypes.byref(filled), ctypes.byref(ctypes.c_uint64()))
        return filled.value

launches = []  # (kernel, device, sequence number, [Pointer])

@ctypes.CFUNCTYPE(None, ctypes.c_char_p, ctypes.c_int, ctypes.c_long, ctypes.POINTER(ctypes.c_void_p))
def on_launch(name, device, seq, args):
    kernel, params = parameters(name.decode())
    ptrs = []
    for i, p in enumerate(params):
        struct = p.split("::")[-1]
        if p.endswith("*"):
            ptrs.append(Pointer(ctypes.c_uint64.from_address(args[i]).value, p))
        elif struct in SCAN:
            words = (ctypes.c_uint64 * (SCAN[struct] // 8)).from_address(args[i])
            ptrs += [q for q in (Pointer(w, struct) for w in words if w) if q.known]
    launches.append((kernel, device, seq, ptrs))

fake.fake_on_launch(on_launch)
import gbz

def device_array(n, shift=0):
    p = ctypes.c_void_p()
    assert fake.cudaMalloc(ctypes.byref(p), 16 * n + 16) == 0
    return p.value + shift

def check(st, ctx):
    assert st == gbz.OK, gbz.lib.gbz_last_error(ctx.h)
"""


@pytest.fixture(scope="module")
def run(gbz, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-o", so, os.path.join(ROOT, "tests", "fake_cudart.c"),
                    "-lpthread"], check=True)

    def run(script):
        env = dict(os.environ, LD_PRELOAD=so)
        r = subprocess.run([sys.executable, "-c", PRELUDE % (PKG, so) + script], capture_output=True, text=True,
                           env=env, timeout=300)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]

    return run


def test_launches_use_their_own_device(run):
    run(r"""
a, b = gbz.Context(0), gbz.Context(1)
x = np.ones((1 << 15, 2), dtype=np.uint64)
for logn in (4, 8, 13, 15):
    a.fft(x[:1 << logn].copy(), logn, False)
for c in (b, a, b, a):
    for logn in (1, 4, 8, 10, 13, 14, 15):
        for inverse in (False, True):
            c.fft(x[:1 << logn].copy(), logn, inverse)
    c.Encode(x[:64].reshape(2, 32, 2), 16, 0)  # cosets
seen = {k for k, *_ in launches}
assert {"ntt_small_kernel", "ntt_pass_kernel"} <= seen, seen
for kernel, device, _, ptrs in launches:
    known = [p for p in ptrs if p.known]
    assert known and all(p.device == device and not p.freed for p in known), (kernel, device)
""")


def test_tables_are_filled_before_they_are_used(run):
    run(r"""
def slow():
    fake.fake_copy_delay(100000)
    c = gbz.Context(0)
    x = np.ones((256, 2), dtype=np.uint64)
    c.fft(x, 8, False)

t = threading.Thread(target=slow)
t.start()
time.sleep(0.05)
c = gbz.Context(0)
while t.is_alive():
    c.fft(np.ones((256, 2), dtype=np.uint64), 8, False)
    c.fft(np.ones((256, 2), dtype=np.uint64), 8, True)
    time.sleep(0.002)
t.join()
assert launches
for kernel, _, seq, ptrs in launches:
    for p in ptrs:
        if p.known and p.filled():  # filled by a copy: a table
            assert p.filled() < seq, kernel
""")


@pytest.mark.parametrize("shift", [0, 8])
def test_device_inputs_at_any_word(run, shift):
    """Inputs that a call takes from device memory may start at any 64-bit word
    (a tensor's slice): the kernels, which load 16 bytes at a time, get the
    caller's pointer only where it is on such a boundary."""
    run("SHIFT = %d" % shift + r"""
ctx = gbz.Context(0)
lib, N, u64 = gbz.lib, 8, ctypes.c_uint64
for form, step in ((gbz.SC_QUADRATIC, 2), (gbz.SC_CUBIC, 4)):
    n, deg = 4096, np.array([64, 8], dtype=np.int32)
    p = [device_array(N * n, SHIFT) for _ in range(3)]
    R = device_array(N * step * int(deg.sum()), SHIFT)
    cubic = form == gbz.SC_CUBIC
    r1, r2, K, Kr, fs, cl = [device_array(64, SHIFT) for _ in range(6)]
    fl = ctypes.c_uint32()
    check(lib.gbz_cosumcheck(ctx.h, form, N, n, p[0], p[1], p[2] if cubic else None, R, r1 if cubic else None,
                             12 if cubic else 0, r2 if cubic else None, K, Kr, deg.ctypes.data, 2, fs, cl,
                             ctypes.byref(fl), None, 0, gbz.MEM_DEVICE), ctx)
rates = [(4,), (4,), (4, 4), (4, 4)]
_, _, rnd = gbz.pcs_schedule(4, 1 << 14, rates)
r0, r1 = gbz._rates(rates)
h = ctypes.c_void_p()
check(lib.gbz_pcs_commit(ctx.h, 4, 1 << 14, 4, r0.ctypes.data, r1.ctypes.data, device_array(4 << 14, SHIFT),
                         device_array(4 * rnd, SHIFT), gbz.MEM_DEVICE, ctypes.byref(h), None, None), ctx)
names = {k for k, *_ in launches}
assert {"k_prepare", "coset_extend_kernel", "cophase2_kernel"} <= names, names
for kernel, _, _, ptrs in launches:
    for q in ptrs:
        if q.known and ("fe" in q.kind or q.kind in SCAN):
            assert q.value %% 16 == 0, (kernel, q.kind)
""".replace("%%", "%"))


def test_commitment_buffers_are_given_back(run):
    run(r"""
rates = [(4,), (4,), (4, 4), (4, 4)]
_, _, rnd = gbz.pcs_schedule(4, 1 << 14, rates)
shares, random = np.ones((4 << 14, 2), dtype=np.uint64), np.ones((4 * rnd, 2), dtype=np.uint64)

def commit(c):
    return gbz.pcs_commit(c, 4, 1 << 14, rates, shares, random)[0]

c = gbz.Context(0)
commit(c).free()
c.sched_release()
base = fake.fake_live()
com = commit(c)
assert fake.fake_live() == base + 4
com.free()
assert fake.fake_live() == base + 4  # one set is kept
one, two = commit(c), commit(c)
assert fake.fake_live() == base + 8
one.free()
two.free()
assert fake.fake_live() == base + 4
assert c.sched_release() > 0 and fake.fake_live() == base
com = commit(c)
c.close()
live = fake.fake_live()
com.free()  # a handle may outlive its context, and then nothing is kept
assert fake.fake_live() == live - 4
""")


@pytest.mark.parametrize("logn", [14, 20, 21])
def test_every_valid_shape_can_be_set(run, logn):
    """A set shape is installed as given and reported; without one the library
    takes passes of its own, which have a name of their own."""
    run("LOGN = %d" % logn + r"""
c, x = gbz.Context(0), np.ones((1 << LOGN, 2), dtype=np.uint64)

def passes():
    launches.clear()
    c.fft(x, LOGN, False)
    return sum(k == "ntt_pass_kernel" for k, *_ in launches)

own = gbz.ntt_get_shape(LOGN)
assert own[0] == -1, own
assert passes() == (3 if LOGN > 20 else 2)
k1 = (LOGN + 1) // 2
valid = [(k1, a, b) for k1 in range(1, 14) for a in range(4) for b in range(4)
         if 1 <= LOGN - k1 <= 13 and a <= k1 and b <= LOGN - k1 and LOGN - k1 + a <= 13 and k1 + b <= 13]
for shape in [(k1, 1, 1)] + valid[::9]:
    gbz.ntt_set_shape(LOGN, *shape)
    assert gbz.ntt_get_shape(LOGN) == shape
    assert passes() == 2, shape
gbz.ntt_set_shape(LOGN, *own)
assert gbz.ntt_get_shape(LOGN) == own and passes() == (3 if LOGN > 20 else 2)
for bad in ((0, 0, 0), (-2, 0, 0), (14, 0, 0)):
    assert gbz.lib.gbz_ntt_set_shape(LOGN, *bad) == gbz.EINVAL
assert gbz.lib.gbz_ntt_set_shape(13, -1, -1, -1) == gbz.EINVAL
assert gbz.lib.gbz_ntt_set_shape(27, -1, -1, -1) == gbz.EINVAL
for n in (13, 27, -1):
    assert gbz.lib.gbz_ntt_get_shape(n, (ctypes.c_int * 3)()) == gbz.EINVAL
""")


def test_autotuning_frees_the_tables_it_built(run):
    run(r"""
c = gbz.Context(0)
x = np.ones((1 << 18, 2), dtype=np.uint64)
c.fft(x, 18, False)
shape, d, b = c.ntt_autotune(18, 1)  # every launch takes as long: the own passes stay
assert shape[0] == -1 and gbz.ntt_get_shape(18) == shape and d == b
base = fake.fake_live()
gbz.ntt_set_shape(18, 8, 1, 1)
assert fake.fake_live() == base + 2  # both directions
c.fft(x, 18, False)
c.ntt_autotune(18, 1)
assert fake.fake_live() == base + 2  # what was there before may still be in use
gbz.ntt_set_shape(18, 8, 1, 1)
launches.clear()
c.fft(x, 18, False)
c.fft(x, 18, True)
assert launches and not any(p.freed for _, _, _, ptrs in launches for p in ptrs)
""")
