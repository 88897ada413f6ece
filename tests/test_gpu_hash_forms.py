"""The session-key hash runs as a warp per request up to four requests per SM and as two lanes per request
(16 per warp) beyond: both forms against the oracle around that line, with a last warp that is not full, and
with seed, ciphertext and key buffers at odd, even and word-aligned addresses (byte, half-word and word accesses)."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)


# plain sets, one whose ciphertext ends on a half word (6960119), and their plaintext-confirmation forms
@pytest.mark.parametrize("sid", (0, 3, 4, 5, 8), ids=("348864", "6960119", "8192128", "348864pc", "6960119pc"))
def test_hash_forms(keys, sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, sk = keys(sid % 5)
    pub, sec = gmc.PublicKey(sid, pk), gmc.SecretKey(sid, sk)
    cb = pub.sizes["ct_bytes"]
    line = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    seeds = request_seeds(sid % 5, line + 17, b"hash")
    oc, ok_, _ = O.enc_batch(sid, pk, seeds, threads=THREADS)
    cts = oc.copy()
    cts[::7, 3] ^= 4
    od, orc = O.dec_batch(sid, sk, cts, threads=THREADS)
    d_seeds = torch.zeros(seeds.size + 8, dtype=torch.uint8, device="cuda")
    for n, off in ((1, 0), (1, 3), (33, 2), (line, 1), (line + 1, 0), (line + 17, 1), (line + 17, 2)):
        c = torch.zeros(n * cb + 8, dtype=torch.uint8, device="cuda")
        k = torch.zeros(n * 32 + 8, dtype=torch.uint8, device="cuda")
        rc = torch.full((n,), 7, dtype=torch.int32, device="cuda")
        d_seeds[off:off + 32 * n] = torch.from_numpy(seeds[:n].reshape(-1)).cuda()
        pub.enc_batch_dev(c.data_ptr() + off, k.data_ptr() + off, d_seeds.data_ptr() + off, n)
        torch.cuda.synchronize()
        ch, kh = c.cpu().numpy(), k.cpu().numpy()
        assert (ch[off:off + n * cb].reshape(n, cb) == oc[:n]).all(), (n, off)
        assert (kh[off:off + n * 32].reshape(n, 32) == ok_[:n]).all(), (n, off)
        assert not ch[:off].any() and not ch[off + n * cb:].any() and not kh[:off].any() and not kh[off + n * 32:].any()
        c[off:off + n * cb] = torch.from_numpy(cts[:n].reshape(-1)).cuda()
        k.zero_()
        sec.dec_batch_dev(k.data_ptr() + off, c.data_ptr() + off, n, rc.data_ptr())
        torch.cuda.synchronize()
        kh = k.cpu().numpy()
        assert (kh[off:off + n * 32].reshape(n, 32) == od[:n]).all(), (n, off)
        assert (rc.cpu().numpy() == orc[:n]).all(), (n, off)
        assert not kh[:off].any() and not kh[off + n * 32:].any()
