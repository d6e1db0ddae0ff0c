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
