"""The windows of the radix-8 butterfly (csrc/gbz_ntt.cu) in exact integers:
every biased sum of extreme inputs must fit 64 bits unsigned, and the stage
twiddles must keep the margin that bounds a folded product by p + 1."""
import itertools

import numpy as np
import pytest

P = (1 << 61) - 1
TOP = 1 << 64
ROT = 1 << 33  # how far a rotated word may leave [0, p]


def outputs(v0, x, rot):
    """Integer values of the biased outputs for real words only (a component
    of every output is a signed sum of this form): v0 and x[1..7], the rotated
    pair given by its two words rot."""
    a = [v0 + 4 * P + x[4], x[1] + x[5], x[2] + x[6], x[3] + x[7]]
    b0, b2 = v0 + 4 * P - x[4], x[2] - x[6]
    even = [a[0] - a[2] + a[1] - a[3], a[0] - a[2] - (a[1] - a[3]), a[0] + a[2] - (a[1] + a[3])]
    total = a[0] + a[2] + a[1] + a[3] - 4 * P
    s, d = rot[0] + rot[1] - P, rot[0] - rot[1]
    odd = [b0 + sg * b2 + t * e for sg in (1, -1) for t in (1, -1) for e in (s, d)]
    return [total] + even + odd


@pytest.mark.parametrize("top0", [P - 1, P + 7])  # first stage; later stages (x = y - 1 in [0, p])
def test_radix8_sums_fit(top0):
    hi = P - 1 if top0 == P - 1 else P
    for bits in itertools.product((0, 1), repeat=8):
        v0, x = bits[0] * top0, [0] + [b * hi for b in bits[1:]]
        for rot in itertools.product((-ROT, P + ROT), repeat=2):
            assert all(0 <= o < TOP for o in outputs(v0, x, rot)), (bits, rot)


def root(log_order):
    """getRootOfUnity (utils.cpp:706-717) in integers."""
    r = (2147483648, 1033321771269002680)
    for _ in range(62 - log_order):
        r = mul(r, r)
    return r


def mul(a, b):
    return ((a[0] * b[0] - a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P)


@pytest.mark.parametrize("inverse", [False, True])
def test_stage_twiddles_keep_the_margin(inverse):
    for ns in range(1, 11):
        w = root(ns + 3)
        if inverse:
            w = (w[0], (P - w[1]) % P)  # unit norm: the inverse is the conjugate
        wr = w
        for _ in range(1, 8):
            x = (1, 0)
            for _ in range(1 << ns):
                nb = P - x[1]
                assert x[0] + nb <= 2 * P - 64 and x[0] + x[1] <= 2 * P - 64
                x = mul(x, wr)
            wr = mul(wr, w)


def test_folded_product_window():
    """t = wrap(S + 1) folded lies in [1, p + 1] at the extremes of S."""
    wrap = lambda s: (s >> 61) + (s & P)
    fold = lambda t: (t & P) + (t >> 61)
    top = (P + 7) * (2 * P - 64) + 1
    rng = np.random.default_rng(1)
    cases = [1, 2, P, P + 1, top, top - 1, (1 << 122) - 1, 1 << 122, (1 << 123) - 1 - (1 << 64)]
    cases += [int(k) << 61 | P for k in range(0, 8)]
    cases += [((1 << 62) - 60 - int(k)) << 61 | P for k in range(8)]
    cases += [int(a) * int(b) % top + 1 for a, b in rng.integers(0, 1 << 62, size=(1000, 2))]
    for s in cases:
        if s <= top:
            assert 1 <= fold(wrap(s)) <= P + 1 and fold(wrap(s)) % P == s % P
