"""Contexts that host threads create at the same time in a new process: the
tables that all of them share are built once, and every thread's short
transforms, the ones that read them, are the oracle's."""
import subprocess
import sys

import pytest

from conftest import ORACLE_DIR, PKG

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys, threading
sys.path[:0] = [%r, %r]
import numpy as np
import gbz, gbz_oracle
LOGS = [1, 4, 7, 8, 10, 11, 14]
rng = np.random.default_rng(1)
x = [rng.integers(0, (1 << 61) - 1, size=(1 << l, 2), dtype=np.uint64) for l in LOGS]
rows = x[4][:64].reshape(2, 32, 2)
want = [[gbz_oracle.fft(a.copy(), inv) for inv in (False, True)] for a in x]
cosets = gbz_oracle.encode_rows(rows, 16, 0)
start, bad = threading.Barrier(4), []

def work(t):
    start.wait()
    c = gbz.Context(0)
    for k in range(len(LOGS)):
        for inv in (0, 1):
            if not np.array_equal(c.fft(x[k].copy(), LOGS[k], bool(inv)), want[k][inv]):
                bad.append((t, LOGS[k], inv))
    if not np.array_equal(c.Encode(rows, 16, 0), cosets):
        bad.append((t, "encode"))
    c.close()

threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not bad, bad
"""


def test_first_tables_from_several_threads(gbz, oracle):
    r = subprocess.run([sys.executable, "-c", SCRIPT % (PKG, ORACLE_DIR)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
