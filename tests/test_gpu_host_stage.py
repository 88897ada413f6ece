"""The page-locked buffer of the small host-pointer calls holds no seeds and no session keys between calls: one request,
the largest call that fits the buffer and a one-request call of the libmceliece convention."""
import ctypes

import numpy as np
import pytest

from tests.conftest import request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_secrets_are_cleared(keys):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    residue = gmc.lib().gmc_host_stage_residue
    residue.restype = ctypes.c_longlong
    sid = 0
    pk, sk = keys(sid)
    pub, sec = gmc.PublicKey(sid, pk), gmc.SecretKey(sid, sk)
    cb = pub.sizes["ct_bytes"]
    for n in (1, 262144 // (cb + 64) - 1):
        c, k, _ = pub.enc_batch(request_seeds(sid, n, b"stage"))
        assert residue() == 0, n
        k2, _ = sec.dec_batch(c)
        assert residue() == 0 and (k2 == k).all() and k.any(), n
    assert (gmc.kem_dec(sid, c[0], sk)[1] == k[0].tobytes()) and residue() == 0
