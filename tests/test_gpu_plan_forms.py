"""Pipelines of a plan with two keys of one set, at sizes where they take the forms chosen by size: chained launches and
the small-batch front end, the request-sliced root finder, and with it the bit-sliced Berlekamp-Massey with split groups
and with other block shapes. A key's rows end inside a block of 256, so a wrong segment shows in the second key's
results. Against the oracle."""
import hashlib
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)
BASE = 83  # distinct ciphertexts per key


@pytest.mark.parametrize("counts,bm_warps", (((70, 91), 14), ((7001, 7500), 14), ((15001, 15500), 14),
                                             ((15001, 15500), 5), ((33000, 32001), 14)))
@pytest.mark.parametrize("sid", (0, 4), ids=("348864", "8192128"))
def test_two_keys_per_pipeline(keys, sid, counts, bm_warps):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    prev = gmc.tune_get(sid)["bm_warps"]
    pairs = [keys(sid), gmc.keypair(sid, hashlib.sha256(b"second key").digest())]
    rng = np.random.default_rng(sid)
    hold, groups, want = [], [], []
    for i, (pk, sk) in enumerate(pairs):
        pub, sec = gmc.PublicKey(sid, pk), gmc.SecretKey(sid, sk)
        cb = pub.sizes["ct_bytes"]
        seeds = request_seeds(sid, BASE, b"plan%d" % i)
        oc, ok, _ = O.enc_batch(sid, pk, seeds, threads=THREADS)
        cts = oc.copy()
        for j in range(0, BASE, 5):
            cts[j, rng.integers(0, cb)] ^= 1 << rng.integers(0, 8)
        kd, rc = O.dec_batch(sid, sk, cts, threads=THREADS)
        ne, nd = (70, 91)[i], counts[i]
        pe, pd = np.arange(ne) % BASE, np.arange(nd) % BASE
        b = [torch.from_numpy(seeds[pe]).cuda(), torch.zeros(ne, cb, dtype=torch.uint8, device="cuda"),
             torch.zeros(ne, 32, dtype=torch.uint8, device="cuda"), torch.from_numpy(cts[pd]).cuda(),
             torch.zeros(nd, 32, dtype=torch.uint8, device="cuda"), torch.full((nd,), 9, dtype=torch.int32, device="cuda")]
        groups.append((pub, ne, b[0].data_ptr(), b[1].data_ptr(), b[2].data_ptr(), 0))
        groups.append((sec, nd, b[3].data_ptr(), 0, b[4].data_ptr(), b[5].data_ptr()))
        hold.append(b)
        want.append((oc[pe], ok[pe], kd[pd], rc[pd]))
    gmc.tune_set(sid, gmc.tune_get(sid)["enc_engine"], gmc.tune_get(sid)["dec_engine"],
                 gmc.tune_get(sid)["sample_threads"], bm_warps=bm_warps)
    try:
        plan = gmc.Plan(groups)
        assert plan.info()["pipelines"] == 2
        for _ in range(2):
            for b in hold:
                for x in (b[1], b[2], b[4]):
                    x.zero_()
            plan.launch(torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            for i, (b, w) in enumerate(zip(hold, want)):
                for x, ref in zip((b[1], b[2], b[4], b[5]), w):
                    assert (x.cpu().numpy() == ref).all(), i
        plan.close()
    finally:
        gmc.tune_set(sid, gmc.tune_get(sid)["enc_engine"], gmc.tune_get(sid)["dec_engine"],
                     gmc.tune_get(sid)["sample_threads"], bm_warps=prev)
