"""The GEMM for few rows (the library's own choice at these sizes) against the persistent kernels' forced tilings, at the edges of its tiles:
one row, a tile less, exactly and more; widths below, at and above 64 and 128; K of less than one 64-wide step, ragged, and longer than
either ring.  The same products in the same order: equal bits.  K slices are compared with the oracle: the engine runs Wo and Wdown of
up to 256 rows that way."""
import numpy as np
import pytest

from tests.gpu_util import require_cuda
from tests.test_engine_gpu import run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 51, 128, 129, 400])
@pytest.mark.parametrize("n,k", [(8, 8), (32, 1024), (64, 72), (72, 64), (136, 264), (200, 640), (1024, 520)])
def test_same_bits_as_the_persistent_tilings(m, n, k):
    torch = require_cuda()
    import vla_cpp_b200 as vb

    g = torch.Generator(device="cuda")
    g.manual_seed(m + n + k)
    x = torch.randn((m, k), device="cuda", generator=g).bfloat16()
    w = (torch.randn((n, k), device="cuda", generator=g) / k ** 0.5).bfloat16()
    got = vb.node_mul_mat(w, x)
    vb.set_gemm_tiling(1)
    want = vb.node_mul_mat(w, x)
    vb.set_gemm_tiling(0)
    assert vb.device_status() == 0
    assert torch.equal(got, want)
    ref = x.float() @ w.float().T
    assert ((got.float() - ref).norm() / ref.norm()).item() < 4e-3  # bf16 rounding of the result: 2^-9 / sqrt(3) is 1.1e-3


def test_projection_of_two_tiles_an_sm_matches_oracle(oracle):
    """16 observations: 280 tiles of 64 columns with row sums of squares, two CTAs an SM; the last row tile of 48 rows."""
    w, d = run_case(oracle, 90, n_obs=16, P=30, check_obs=[0, 7, 15], model=0, L=1, H=136, n_q=8, n_kv=1, hd=256, inter=512, chunk=50, A=32, sd=32, T=1)
    assert w < 1e-2 and d < 3e-2, (w, d)


@pytest.mark.parametrize("hd,n_obs", [(64, 1), (64, 5), (128, 2), (256, 5)])
@pytest.mark.parametrize("model", [0, 1])
def test_few_observations_match_oracle(oracle, monkeypatch, hd, n_obs, model):
    """q | k | v rotated in the product's epilogue, K slices with a ragged last tile (H = 200) and a K that does not divide evenly."""
    monkeypatch.setenv("VLAB200_CHUNK_LOOP", "0")
    w, d = run_case(oracle, 70 + hd + n_obs, n_obs=n_obs, P=70, model=model, L=2, H=200, n_q=4, n_kv=2, hd=hd, inter=1048, chunk=50, A=32, sd=32, T=2,
                    self_every=2)
    assert w < 1e-2 and d < 3e-2, (w, d)
