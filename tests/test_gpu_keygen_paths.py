"""Key generation around the line between overlapping attempts per key (up to 8 systematic keys per call) and rounds of
rank tests: the most and the fewest keys of either side, with chains that need several waves of attempts, byte-exact
against the oracle and against the same keys generated one by one."""
import hashlib
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from oracle import pyoracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sid", (0, 3), ids=("348864", "6960119"))
def test_keygen_few_and_batch(sid):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as gmc

    seeds = np.frombuffer(b"".join(hashlib.sha256(b"few%d-%d" % (sid, i)).digest() for i in range(9)),
                          np.uint8).reshape(9, 32)
    with ThreadPoolExecutor(min(16, os.cpu_count() or 1)) as ex:
        ref = list(ex.map(lambda s: O.keypair(sid, bytes(s)), seeds))
    for n in (1, 5, 8, 9):
        pk, sk = gmc.keypair_batch(sid, seeds[:n])
        for i in range(n):
            assert np.array_equal(pk[i], np.asarray(ref[i][0])) and np.array_equal(sk[i], np.asarray(ref[i][1])), (n, i)
    pk, sk = gmc.keypair(sid, bytes(seeds[7]))
    assert np.array_equal(pk, np.asarray(ref[7][0])) and np.array_equal(sk, np.asarray(ref[7][1]))
