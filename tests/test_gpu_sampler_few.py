"""The sampler's block-per-request form: one request, both sides of the batch size up to which it is taken, seeds at odd
addresses, dense and sparse syndromes, against the oracle."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS, request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)


@pytest.mark.parametrize("engine", (-1, 2), ids=("sparse", "dense"))
@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_sampler_few(keys, sid, engine):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, _ = keys(sid)
    z = O.sizes(sid)
    pub = gmc.PublicKey(sid, pk)
    perms = (2, 3, 4, 4, 2)[sid]
    line = (30 if sid == 4 else 36 // perms) * torch.cuda.get_device_properties(0).multi_processor_count
    base = 257
    seeds = np.frombuffer(request_seeds(sid, base, b"few").tobytes(), np.uint8).reshape(base, 32)
    oc, ok, _ = O.enc_batch(sid, pk, seeds, threads=THREADS)
    gmc.set_gemm_engine(engine)
    try:
        for n in (1, 2, base, line, line + 1):
            pick = np.arange(n) % base
            for off in (0, 1):
                buf = torch.zeros(32 * n + 1, dtype=torch.uint8)
                buf[off : off + 32 * n] = torch.from_numpy(seeds[pick].reshape(-1).copy())
                buf = buf.cuda()
                ct = torch.empty(n, z["ct_bytes"], dtype=torch.uint8, device="cuda")
                k = torch.empty(n, 32, dtype=torch.uint8, device="cuda")
                assert gmc.lib().gmc_enc_batch_dev(pub.handle, ct.data_ptr(), k.data_ptr(), buf.data_ptr() + off, n,
                                                   None, 0) == 0
                torch.cuda.synchronize()
                assert (ct.cpu().numpy() == oc[pick]).all() and (k.cpu().numpy() == ok[pick]).all(), (n, off)
    finally:
        gmc.set_gemm_engine(-1)
