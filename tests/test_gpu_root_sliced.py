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


def test_sliced_roots_stage_rows_at_any_word(keys):
    """Error-vector rows of the caller that start between 16-byte boundaries (the stage outputs take any word)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    sid = 0
    pk, sk = keys(sid)
    z = O.sizes(sid)
    cts, _, _ = gmc.PublicKey(sid, pk).enc_batch(request_seeds(sid, 50, b"rows"))
    n = FIRST + 1
    d_c = torch.from_numpy(cts[np.arange(n) % 50]).cuda()
    lds2 = ((2 * z["t"] * z["m"] + 31) // 32 + 3) // 4 * 4
    lde = ((z["n"] + 31) // 32 + 3) // 4 * 4
    sec = gmc.SecretKey(sid, sk)
    rows = []
    for off in (0, 1):
        s2 = torch.zeros(n * lds2 + 1, dtype=torch.int32, device="cuda")
        e = torch.zeros(n * lde + 1, dtype=torch.int32, device="cuda")
        ok = torch.zeros(n, dtype=torch.int32, device="cuda")
        assert gmc.lib().gmc_dec_stages_dev(sec.handle, d_c.data_ptr(), n, s2.data_ptr() + 4 * off, lds2,
                                            e.data_ptr() + 4 * off, lde, ok.data_ptr(), 0) == 0
        torch.cuda.synchronize()
        assert int(ok.sum()) == n
        words = (z["n"] + 31) // 32
        rows.append(e[off : off + n * lde].view(n, lde)[:, :words].cpu())
    assert torch.equal(rows[0], rows[1])
