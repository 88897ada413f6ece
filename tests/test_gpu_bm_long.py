"""Error vectors of sequences whose linear complexity ends above t, which no ciphertext of a real key gives in reach of a
search: the library's rule drops the coefficients above t from its arrays, and every Berlekamp-Massey form follows it.
The key is a real one whose front-end matrix is replaced in its exported string, so that bit i of a ciphertext selects
sequence i. The reference is the rule itself with numpy (tests/decode_model.py's bm, all sequences at once)."""
import hashlib
import struct

import numpy as np
import pytest

from tests.conftest import SETS
from tests.decode_model import host_tables

torch = pytest.importorskip("torch")
SEQS = 96


def sequences(sid):
    """A linear recurrence of length l for n0 terms, then random ones: L jumps from about l to n0 + 1 - l."""
    tb = host_tables(sid)
    q, t = tb["q"], tb["t"]
    g = np.random.default_rng(sid)
    S = g.integers(0, q, (SEQS, 2 * t))
    exp, log = tb["gexp"].astype(np.int64), tb["glog"].astype(np.int64)
    for i in range(SEQS):
        lo = (0, 1, 3, t // 2, t - 8, t - 2)[i % 6]
        n0 = min(2 * t - 2, t + lo + (i // 6) % 8 - 2)  # n0 + 1 - lo from t - 1 to t + 6
        if lo == 0:
            S[i, :n0] = 0
            continue
        c = log[g.integers(1, q, lo)]
        for n in range(lo, n0):
            S[i, n] = np.bitwise_xor.reduce(exp[np.minimum(c + log[S[i, n - lo:n]], 2 * q - 2)])
    return tb, S


def berlekamp_massey(tb, S, ahead=False):
    """(C [N, t+1], L) by the library's rule; ahead: by the looked-ahead discrepancy without its truncation term."""
    q, t, N = tb["q"], tb["t"], len(S)
    exp, log = tb["gexp"].astype(np.int64), tb["glog"].astype(np.int64)

    def mul(a, b):
        return exp[np.minimum(log[a] + log[b], 2 * q - 2)]

    def dot(C, n):
        k = min(n, t)
        return np.bitwise_xor.reduce(mul(C[:, :k + 1], S[:, n - k:n + 1][:, ::-1]), axis=1)

    C, B = np.zeros((2, N, t + 1), np.int64)
    C[:, 0], B[:, 1] = 1, 1
    L, b = np.zeros(N, np.int64), np.ones(N, np.int64)
    d = quo = S[:, 0]
    for n in range(2 * t):
        if not ahead:
            d = dot(C, n)
        lf = log[d] - log[b]
        f = np.where(d == 0, 0, exp[np.clip(np.where(lf < 0, lf + q - 1, lf), 0, 2 * q - 2)])
        upd = (d != 0) & (2 * L <= n)
        e = dot(C, n + 1) if n + 1 < 2 * t else d
        C, T, dn = C ^ mul(f[:, None], B), C, e ^ mul(f, quo)
        L, b, quo = np.where(upd, n + 1 - L, L), np.where(upd, d, b), np.where(upd, e, quo)
        B = np.concatenate([np.zeros((N, 1), np.int64), np.where(upd[:, None], T, B)[:, :-1]], axis=1)
        if ahead:
            d = dn
    return C, L


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_lookahead_without_truncation(sid):
    """The sequences tell the two rules apart, and only where both lengths end above t."""
    tb, S = sequences(sid)
    C, L = berlekamp_massey(tb, S)
    C2, L2 = berlekamp_massey(tb, S, ahead=True)
    differ = (C != C2).any(axis=1)
    assert differ.sum() >= 8
    assert (L[differ] > tb["t"]).all() and (L2[differ] > tb["t"]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_error_vectors_above_t(keys, sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    tb, S = sequences(sid)
    m, t, n = tb["m"], tb["t"], tb["n"]
    blob = bytearray(gmc.SecretKey(sid, keys(sid)[1]).export())
    ldf, frows = struct.unpack_from("<2i", blob, 44)
    assert struct.unpack_from("<Q", blob, 64)[0] == 4 * ldf * frows
    bits = np.zeros((frows, 32 * ldf), np.uint8)
    for i in range(SEQS):
        bits[:2 * t * m, i] = ((S[i][:, None] >> np.arange(m)) & 1).reshape(-1)
    blob[136:136 + 4 * ldf * frows] = np.packbits(bits, axis=1, bitorder="little").tobytes()
    support = np.frombuffer(blob, np.uint16, n, 136 + 4 * ldf * frows).astype(np.int64)
    blob[104:136] = bytes(32)
    blob[104:136] = hashlib.shake_256(bytes(blob)).digest(32)
    sec = gmc.SecretKey.from_export(bytes(blob))

    # sigma(x) = sum_deg C[t - deg] x^deg at the support
    q = tb["q"]
    exp, log = tb["gexp"].astype(np.int64), tb["glog"].astype(np.int64)
    C, L = berlekamp_massey(tb, S)
    v = np.zeros((SEQS, n), np.int64)
    for i in range(t + 1):
        v = exp[np.minimum(log[v] + log[support][None, :], 2 * q - 2)] ^ C[:, i:i + 1]
    want = np.packbits(v == 0, axis=1, bitorder="little")

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lde, lds2 = ((n + 31) // 32 + 3) // 4 * 4, ((2 * t * m + 31) // 32 + 3) // 4 * 4
    cb = sec.sizes["ct_bytes"]
    one = np.zeros((SEQS, cb), np.uint8)
    for i in range(SEQS):
        one[i, i >> 3] = 1 << (i & 7)
    for count in (SEQS, 16 * sms, 16 * sms + 1, 22528 if t <= 64 else 29696):  # looked ahead, latency form, bit-sliced
        pick = np.arange(count) % SEQS
        d_c = torch.from_numpy(one[pick]).cuda()
        s2 = torch.zeros(count, lds2, dtype=torch.int32, device="cuda")
        ev = torch.zeros(count, lde, dtype=torch.int32, device="cuda")
        ok = torch.zeros(count, dtype=torch.int32, device="cuda")
        assert gmc.lib().gmc_dec_stages_dev(sec.handle, d_c.data_ptr(), count, s2.data_ptr(), lds2, ev.data_ptr(), lde,
                                            ok.data_ptr(), None) == 0
        torch.cuda.synchronize()
        got = ev.cpu().numpy().view(np.uint8)[:, :n // 8]
        bad = np.flatnonzero((got != want[pick]).any(axis=1))
        assert bad.size == 0, (count, bad.size, sorted(set(L[pick[bad]] - t)))
        assert not (ok.cpu().numpy()[(L != t)[pick]]).any(), count
