"""Products of more tiles than CTAs (pairs): with row statistics in contiguous ranges of tiles, without in turn."""
import pytest

from tests.gpu_util import kernels_of, require_cuda
from tests.test_engine_gpu import run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_obs", [120, 187])  # 6,120 and 9,537 rows: 96 and 152 pair tiles, 192 and 300 of one CTA; the last one ragged
@pytest.mark.parametrize("tiling", [0, 1, 3])  # the engine's choice, 256 columns of one CTA, CTA pairs
def test_more_tiles_than_units_match_the_oracle(oracle, n_obs, tiling):
    w, d = run_case(oracle, 55, n_obs=n_obs, P=20, tiling=tiling, check_obs=[0, n_obs // 2, n_obs - 1], model=0, L=1, H=1024, n_q=8, n_kv=1,
                    hd=64, inter=1024, chunk=50, A=32, sd=32, T=1)
    assert w < 1e-2 and d < 3e-2, (w, d)


@pytest.mark.parametrize("H", [480, 720, 960])  # 3,264 rows: the widths 96, 160 and 192 are those whose tiles make one wave
def test_tile_widths_that_fill_a_wave_match_the_oracle(oracle, H):
    w, d = run_case(oracle, 56, n_obs=64, P=20, check_obs=[0, 31, 63], model=0, L=2, H=H, n_q=8, n_kv=1, hd=64, inter=H // 2, chunk=50, A=32,
                    sd=32, T=1)
    assert w < 1e-2 and d < 3e-2, (w, d)


@pytest.mark.parametrize("H,width", [(480, 96), (720, 160), (960, 192)])
def test_those_widths_are_taken(H, width):
    """The rule counts tiles against SMs, so the test above covers a width only where it is the choice: the kernel by name, and the bits of
    the forced 256-column tiling."""
    torch = require_cuda()
    import vla_cpp_b200 as vb

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the widths that fill a wave are others")
    x = torch.randn((3264, H), device="cuda").bfloat16()
    w = (torch.randn((H, H), device="cuda") / H ** 0.5).bfloat16()
    got = vb.node_mul_mat(w, x)
    vb.set_gemm_tiling(1)
    want = vb.node_mul_mat(w, x)
    vb.set_gemm_tiling(0)
    assert torch.equal(got, want) and vb.device_status() == 0
    names = kernels_of(lambda: vb.node_mul_mat(w, x))
    assert any(f"dense_gemm_kernelILi{width}E" in k for k in names), names
