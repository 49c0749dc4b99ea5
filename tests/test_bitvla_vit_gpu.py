"""The BitVLA vision tower against the CPU oracle where its row kernels and the strided attention can go wrong: patch counts that do not fill
a 128-row tile, an MLP padded on the K side, and both routes (16-byte accesses; a head_dim that is no multiple of 8 takes the general
kernels).

Bar: this library sits 1.31e-2 (1 layer) and 1.75e-2 (2 layers) from the oracle at the tower's full size, the distance that last-bit
differences grow to through four int8 quantisations a layer (tests/test_bitvla_vit_ref_gpu.py); 3e-2 is that with head-room of 1.7x."""
import numpy as np
import pytest

from tests.gpu_util import bf16_bits, bits_to_bf16_tensor, rel_l2, require_cuda
from tests.test_bitvla_vit_ref_gpu import bind, drive, make_vit, vit_to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads,ffn,n_patches,n_layers", [
    (1152, 16, 4304, 131, 1), (1152, 16, 4304, 9, 1), (384, 3, 400, 257, 2), (256, 4, 512, 100, 2),
    (384, 32, 256, 40, 1),   # head_dim 12: general kernels
    (1408, 16, 512, 33, 1),  # rows longer than the register kernels hold: general kernels
    (256, 4, 272, 5, 1),     # the GEMV's rows: general kernels
])
def test_tower_matches_oracle(oracle, hidden, heads, ffn, n_patches, n_layers):
    require_cuda()
    from vla_cpp_b200 import api

    cfg = dict(hidden=hidden, n_heads=heads, ffn=ffn, n_patches=n_patches, patch_flat=588, ln_eps=1e-6, mm_out=128)
    rng = np.random.default_rng(hidden + heads + n_patches)
    w = make_vit(oracle, rng, n_layers, cfg)
    patches_h = oracle.bf16_round(rng.uniform(-1, 1, (n_patches, 588)).astype(np.float32))
    patches = bits_to_bf16_tensor(oracle.f32_to_bf16_bits(patches_h))
    lib, dw = bind(api.lib()), vit_to_dev(oracle, w)
    got = bf16_bits(drive(lib, cfg, dw, patches))
    assert api.device_status() == 0
    assert np.array_equal(got, bf16_bits(drive(lib, cfg, dw, patches)))
    err = rel_l2(oracle.bf16_bits_to_f32(got), oracle.bitvla_vit_forward(patches_h, w, cfg))
    assert err <= 3e-2, err
