"""The request-sliced root finder against the oracle: row counts at its first size, with a last tile of 512 requests and
a last group of 32 that are not full, over all sets, with corrupted, random and zero ciphertexts."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS, request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)
FIRST = 14000  # kRootSlicedMinRows


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_sliced_roots(keys, sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, sk = keys(sid)
    z = O.sizes(sid)
    sec = gmc.SecretKey(sid, sk)
    base = 97
    cts, _, _ = gmc.PublicKey(sid, pk).enc_batch(request_seeds(sid, base, b"sliced"))
    rng = np.random.default_rng(sid)
    for i in range(0, base, 4):
        cts[i, rng.integers(0, z["mt"] // 8)] ^= 1 << rng.integers(0, 8)
    cts[50:60] = rng.integers(0, 256, size=(10, z["ct_bytes"]), dtype=np.uint8)
    cts[60] = 0
    if z["mt"] % 8:
        cts[50:60, -1] &= (1 << (z["mt"] % 8)) - 1
    ref, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
    for n in (FIRST, FIRST + 335, FIRST + 337, FIRST + 337 + 255):
        pick = np.arange(n) % base
        k, r = sec.dec_batch(cts[pick])
        assert (k == ref[pick]).all() and (r == rc[pick]).all(), n
