"""When a decoded error is accepted: words of weight t - 2 .. t + 1 on the first m t positions, with and without the
support element 0 (a locator of length t - 1 has a t-th root there), for a key with an irreducible Goppa polynomial and
one with a square factor, in every Berlekamp-Massey form, against the oracle."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)
PARAMS = {0: (12, 64, 3488), 1: (13, 96, 4608), 2: (13, 128, 6688), 3: (13, 119, 6960), 4: (13, 128, 8192)}


def field(m):
    poly = {12: 0x1009, 13: 0x201B}[m]
    exp, log, v = [0] * (1 << m), [0] * (1 << m), 1
    for i in range((1 << m) - 1):  # powers of x + 1, a generator for both m
        exp[i], log[v] = v, i
        v ^= v << 1
        if v >> m:
            v ^= poly
    return exp, log


def mul(f, a, b):
    exp, log = f
    return exp[(log[a] + log[b]) % (len(exp) - 1)] if a and b else 0


def has_root(f, g, points):
    for a in points:
        v = 0
        for c in reversed(g):
            v = mul(f, v, a) ^ c
        if not v:
            return True
    return False


def square_factor(f, m, t, n, rng):
    """h^2 (times x + a for odd t) without roots on the support 0 .. n - 1 in bit-reversed order."""
    support = [int(format(i, f"0{m}b")[::-1], 2) for i in range(1 << m)]
    while True:
        h = [int(x) for x in rng.integers(0, 1 << m, t // 2)] + [1]
        if not has_root(f, h, support[:n]):
            break
    g = [0] * (2 * (t // 2) + 1)
    for i, c in enumerate(h):
        g[2 * i] = mul(f, c, c)
    if t % 2:
        a = support[n]
        g = [mul(f, a, x) ^ y for x, y in zip(g + [0], [0] + g)]
    return g


@pytest.mark.parametrize("square", (False, True), ids=("irreducible", "square"))
@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_acceptance(keys, sid, square):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    z = O.sizes(sid)
    m, t, n = PARAMS[sid]
    rng = np.random.default_rng(10 * sid + square)
    sk = np.array(keys(sid)[1], np.uint8).copy()
    cond = (2 * m - 1) << (m - 4)
    sk[40 + 2 * t : 40 + 2 * t + cond] = 0  # identity: position i holds the bit-reversed i, position 0 the element 0
    if square:
        g = square_factor(field(m), m, t, n, rng)
        sk[40 : 40 + 2 * t] = np.array(g[:t], "<u2").view(np.uint8)
    cts = []
    for w in (t - 2, t - 1, t, t + 1):
        for zero in (False, True):
            for _ in range(3):
                pos = 1 + rng.choice(z["mt"] - 1, w, replace=False)
                if zero:
                    pos[0] = 0
                bits = np.zeros(8 * z["ct_bytes"], np.uint8)
                bits[pos] = 1
                cts.append(np.packbits(bits, bitorder="little"))
    cts = np.array(cts)
    ref, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
    sec = gmc.SecretKey(sid, sk)
    for on in (False, True):
        gmc.set_dec_constant_time(on)
        try:
            for reps in (1, 1 if on else 65536 // len(cts) + 1):
                k, r = sec.dec_batch(np.tile(cts, (reps, 1)))
                assert (k == np.tile(ref, (reps, 1))).all() and (r == np.tile(rc, reps)).all(), (on, reps)
        finally:
            gmc.set_dec_constant_time(False)
