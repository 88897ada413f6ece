"""Syndromes of small batches straight from the ciphertext bytes against the tensor-core and popcount products: one
request, the edges of the 16 requests a block shares, both sides of the size line, ciphertexts that start at odd
addresses, and plaintext-confirmation rows."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("pc", (0, 5), ids=("plain", "pc"))
@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_front_few(keys, sid, pc):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    z = O.sizes(sid)
    sec = gmc.SecretKey(sid + pc, keys(sid)[1])
    cb = z["ct_bytes"] + (32 if pc else 0)
    words = (2 * z["t"] * z["m"] + 31) // 32
    lds2, lde = (words + 3) // 4 * 4, ((z["n"] + 31) // 32 + 3) // 4 * 4
    line = (3 << 20) // (z["ct_bytes"] * words)
    rng = np.random.default_rng(sid)
    data = torch.from_numpy(rng.integers(0, 256, (line + 1) * cb + 1, dtype=np.uint8)).cuda()
    for n in (1, 15, 16, 17, 33, line, line + 1):
        for off in (0, 1):
            got = []
            for engine in (-1, 2, 0):
                gmc.set_gemm_engine(engine)
                try:
                    s2 = torch.zeros(n, lds2, dtype=torch.int32, device="cuda")
                    e = torch.zeros(n, lde, dtype=torch.int32, device="cuda")
                    ok = torch.zeros(n, dtype=torch.int32, device="cuda")
                    assert gmc.lib().gmc_dec_stages_dev(sec.handle, data.data_ptr() + off, n, s2.data_ptr(), lds2,
                                                        e.data_ptr(), lde, ok.data_ptr(), 0) == 0
                    torch.cuda.synchronize()
                finally:
                    gmc.set_gemm_engine(-1)
                got.append(s2[:, :words].cpu())
            assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2]), (n, off)
