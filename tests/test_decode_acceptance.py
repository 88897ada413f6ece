"""The acceptance rule of the decoder on codes small enough to try every word: over GF(16), for every binary word, the
locator of length t with t distinct roots on the support is that of an error with the word's syndromes, so comparing the
syndromes as well changes nothing, whatever the Goppa polynomial without roots on the support."""
import itertools

import pytest

M, Q = 4, 16
EXP, LOG = [0] * 15, [0] * 16
_v = 1
for _i in range(15):
    EXP[_i], LOG[_v] = _v, _i
    _v = (_v << 1) ^ (0x13 if _v & 8 else 0)


def mul(a, b):
    return EXP[(LOG[a] + LOG[b]) % 15] if a and b else 0


def inv(a):
    return EXP[-LOG[a] % 15]


def value(p, x):
    v = 0
    for c in reversed(p):
        v = mul(v, x) ^ c
    return v


def berlekamp_massey(s):
    c, b, length, gap, bb = [1], [1], 0, 1, 1
    for i in range(len(s)):
        d = 0
        for k in range(min(len(c), i + 1)):
            d ^= mul(c[k], s[i - k])
        if d:
            f, old = mul(d, inv(bb)), c
            nc = c + [0] * max(0, len(b) + gap - len(c))
            for k, x in enumerate(b):
                nc[k + gap] ^= mul(f, x)
            c = nc
            if 2 * length <= i:
                length, b, bb, gap = i + 1 - length, old, d, 0
        gap += 1
    return c, length


def disagreements(g, support):
    """Words that the rule (length t, t distinct roots on the support) accepts and the syndromes do not; and the
    number of words that both accept."""
    t = len(g) - 1
    cols = [[mul(inv(mul(value(g, a), value(g, a))), EXP[LOG[a] * j % 15] if a else int(j == 0)) for j in range(2 * t)]
            for a in support]
    bad = accepted = 0
    for word in itertools.product((0, 1), repeat=len(support)):
        s = [0] * (2 * t)
        for bit, col in zip(word, cols):
            if bit:
                s = [x ^ y for x, y in zip(s, col)]
        c, length = berlekamp_massey(s)
        sigma = [(c + [0] * (t + 1))[t - d] for d in range(t + 1)]
        roots = [i for i, a in enumerate(support) if not value(sigma, a)]
        if length != t or len(roots) != t:
            continue
        e = [0] * (2 * t)
        for i in roots:
            e = [x ^ y for x, y in zip(e, cols[i])]
        accepted += e == s
        bad += e != s
    return bad, accepted


def product(*ps):
    r = [1]
    for p in ps:
        n = [0] * (len(r) + len(p) - 1)
        for i, x in enumerate(r):
            for j, y in enumerate(p):
                n[i + j] ^= mul(x, y)
        r = n
    return r


IRRED2 = next([c, 1, 1] for c in range(1, 16) if all(value([c, 1, 1], a) for a in range(16)))


@pytest.mark.parametrize("g", [
    IRRED2,
    product([3, 1], [5, 1]),
    product(IRRED2, [3, 1]),
    product([3, 1], [3, 1]),
    product([3, 1], [3, 1], [5, 1]),
], ids=("irreducible", "two factors", "degree 3", "square", "square factor"))
def test_length_and_roots_are_enough(g):
    support = [a for a in range(Q) if value(g, a)][:12]
    assert 0 in support
    bad, accepted = disagreements(g, support)
    assert accepted > 0 and bad == 0
