"""The block-per-request sampler's exit: all warps of a block leave after the step that checked the successful attempt,
for requests that end with their first attempt, their second and so on up to the longest of the sample, each alone in
its batch and all of them mixed, several times over, against the oracle."""
import os

import numpy as np
import pytest

from oracle import pyoracle as O
from tests.conftest import SETS, request_seeds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
THREADS = min(16, os.cpu_count() or 1)


@pytest.mark.parametrize("sid", range(5), ids=SETS)
def test_sampler_exit(keys, sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    pk, _ = keys(sid)
    seeds = request_seeds(sid, 160, b"exit")
    by_attempts = {}
    for i in range(len(seeds)):
        by_attempts.setdefault(O.gen_e(sid, seeds[i].tobytes())[1], i)
    assert min(by_attempts) == 1 and len(by_attempts) >= 4
    few = [by_attempts[a] for a in sorted(by_attempts)]
    oc, ok, _ = O.enc_batch(sid, pk, seeds[few], threads=THREADS)
    pub = gmc.PublicKey(sid, pk)
    for pick in [[i] for i in range(len(few))] + [list(range(len(few))) * 12]:
        for _ in range(4):
            c, k, _ = pub.enc_batch(seeds[few][pick])
            assert (c == oc[pick]).all() and (k == ok[pick]).all(), pick
