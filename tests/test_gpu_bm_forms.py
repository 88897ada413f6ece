"""Berlekamp-Massey forms at the edges of their launch shapes: the constant-time form (a block per 32 requests, a warp
per 32 coefficients and one for the constant coefficient) and the latency form (a warp per request) on one request,
a group that is not full, one group and a little more, against the oracle; and both against each other on a batch in
which some groups hold only corrupted ciphertexts (length profiles that leave the regular one)."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS, request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_bm_forms_edges(keys, sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, sk = keys(sid)
    z = O.sizes(sid)
    sec = gmc.SecretKey(sid, sk)
    n = 289
    cts, _, _ = gmc.PublicKey(sid, pk).enc_batch(request_seeds(sid, n, b"bm"))
    rng = np.random.default_rng(sid)
    for i in range(0, n, 5):
        cts[i, rng.integers(0, z["mt"] // 8)] ^= 1 << rng.integers(0, 8)
    cts[64:96] = rng.integers(0, 256, size=(32, z["ct_bytes"]), dtype=np.uint8)
    cts[64] = 0  # all syndromes zero: no discrepancy in any iteration
    cts[65] = 0
    cts[65, 0] = 1
    if z["mt"] % 8:
        cts[64:96, -1] &= (1 << (z["mt"] % 8)) - 1
    ref, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
    for on in (False, True):
        gmc.set_dec_constant_time(on)
        try:
            for lo, hi in ((0, 1), (64, 65), (65, 66), (0, 31), (0, 33), (64, 96), (0, n)):
                k, r = sec.dec_batch(cts[lo:hi])
                assert (k == ref[lo:hi]).all() and (r == rc[lo:hi]).all(), (on, lo, hi)
        finally:
            gmc.set_dec_constant_time(False)


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_bm_latency_block_sizes(keys, sid):
    """Both sides of the largest batch with at most eight requests per block (the look-ahead discrepancy)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, sk = keys(sid)
    z = O.sizes(sid)
    base = 61
    cts, _, _ = gmc.PublicKey(sid, pk).enc_batch(request_seeds(sid, base, b"blk"))
    rng = np.random.default_rng(sid)
    for i in range(0, base, 4):
        cts[i, rng.integers(0, z["mt"] // 8)] ^= 1 << rng.integers(0, 8)
    cts[3] = 0
    cts[7] = 0
    cts[7, 0] = 2  # discrepancies that vanish from some iteration on
    ref, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
    sec = gmc.SecretKey(sid, sk)
    edge = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    for n in (edge, edge + 1):
        pick = np.arange(n) % base
        k, r = sec.dec_batch(cts[pick])
        assert (k == ref[pick]).all() and (r == rc[pick]).all(), n


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_bm_split_groups(keys, sid):
    """Blocks of the bit-sliced form with 9, 10, 13 and 14 groups of 32 requests, whose last one or two change warps
    halfway, and with 12, which have none."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, sk = keys(sid)
    z = O.sizes(sid)
    base = 89
    cts, _, _ = gmc.PublicKey(sid, pk).enc_batch(request_seeds(sid, base, b"split"))
    rng = np.random.default_rng(sid)
    for i in range(0, base, 4):
        cts[i, rng.integers(0, z["mt"] // 8)] ^= 1 << rng.integers(0, 8)
    cts[3] = 0
    cts[7] = 0
    cts[7, 0] = 2
    ref, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
    sec = gmc.SecretKey(sid, sk)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for groups in (9, 10, 12, 13, 14):
        n = 32 * groups * sms - 300
        pick = np.arange(n) % base
        k, r = sec.dec_batch(cts[pick])
        assert (k == ref[pick]).all() and (r == rc[pick]).all(), groups
