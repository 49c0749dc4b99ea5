"""Every tiling of the ternary product at the edges of its tiles: 64- and 128-column tiles, alone and with their K steps cut over 2 or 4 CTAs
of a cluster.  Accumulators are whole numbers, so each gives exactly the oracle's; the bf16 outputs of all tilings are the same bits."""
import numpy as np
import pytest

from tests.gpu_util import bf16_bits, require_cuda, to_dev

pytestmark = pytest.mark.gpu

TILINGS = [64, 128, 64 + (2 << 8), 128 + (2 << 8), 64 + (4 << 8), 128 + (4 << 8)]


@pytest.mark.parametrize("m", [9, 128, 129, 300])
@pytest.mark.parametrize("n,k,ws_num", [(16, 512, 1), (80, 640, 1), (192, 1152, 3), (1152, 4352, 1)])
def test_forced_tilings_exact(oracle, m, n, k, ws_num):
    torch = require_cuda()
    import vla_cpp_b200 as vb

    rng = np.random.default_rng(m + n + k)
    tern = rng.integers(-1, 2, (n, k)).astype(np.int8)
    a = rng.integers(-127, 128, (m, k)).astype(np.int8)
    s = (40.0 + rng.integers(0, 100, m)).astype(np.float32)
    ws = (0.01 + 0.001 * rng.integers(0, 50, ws_num)).astype(np.float32)
    ref = oracle.gemm_i8_i32(a, tern)
    ad, wd, sd, wsd = to_dev(a), to_dev(oracle.pack_ladder_int2(tern)), to_dev(s), to_dev(ws)
    outs = []
    for path in TILINGS:
        acc = torch.full((m, n), -7, dtype=torch.int32, device="cuda")
        out = vb.ternary_linear(ad, wd, sd, wsd, n, acc_out=acc, path=path)
        assert vb.device_status() == 0
        assert np.array_equal(acc.cpu().numpy(), ref), path
        outs.append(bf16_bits(out))
    for path, out in zip(TILINGS, outs):
        assert np.array_equal(out, outs[0]), path


def test_more_slices_than_k_steps_are_refused():
    torch = require_cuda()
    import vla_cpp_b200 as vb

    a = torch.zeros((16, 256), dtype=torch.int8, device="cuda")
    w = torch.zeros(64 * 256 // 4, dtype=torch.uint8, device="cuda")
    one = torch.ones(16, device="cuda")
    with pytest.raises(Exception):
        vb.ternary_linear(a, w, one, one[:1], 64, path=64 + (4 << 8))
    assert vb.device_status() == 0
