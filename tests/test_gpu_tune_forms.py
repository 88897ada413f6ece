"""The autotuner leaves a parameter alone when the timed batch takes forms of the kernels that do not read it: its value
would be picked by noise and then serve every batch size of the set."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture
def gmc():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import tensormceliece_gb300 as g
    prev = [g.tune_get(s) for s in range(5)]
    yield g
    for s, p in enumerate(prev):
        g.tune_set(s, p["enc_engine"], p["dec_engine"], p["sample_threads"], gemm_stages=p["gemm_stages"],
                   bm_warps=p["bm_warps"], root_warps=p["root_warps"], sample_sm_warps=p["sample_sm_warps"])


@pytest.mark.parametrize("dec_engine", ("popc", "tc"))
@pytest.mark.parametrize("sid", (0, 4), ids=("348864", "8192128"))
def test_small_batch_keeps_unread_parameters(gmc, sid, dec_engine):
    """64 requests: a block per request in the sampler, one kernel for the front end."""
    gmc.tune_set(sid, "sparse", dec_engine, 64, gemm_stages=3, bm_warps=11, root_warps=8, sample_sm_warps=12)
    got = gmc.autotune(sid, 64)
    assert got["dec_engine"] == dec_engine and got["sample_threads"] == 64
    assert got["sample_sm_warps"] == 12 and got["bm_warps"] == 11
    if got["enc_engine"] != "tc":
        assert got["gemm_stages"] == 3


def test_root_warps_above_the_sliced_line(gmc):
    """Batches from 14000 rows take the request-sliced root finder, but the server's still read root_warps: a tune at
    such a size replaces one warp per block (about a third of the speed of four)."""
    gmc.tune_set(0, "sparse", "tc", 128, gemm_stages=4, bm_warps=14, root_warps=1, sample_sm_warps=0)
    assert gmc.autotune(0, 16384)["root_warps"] > 1
