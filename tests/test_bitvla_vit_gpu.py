"""The BitVLA vision tower against the CPU oracle where its row kernels and the strided attention can go wrong: patch counts that do not fill
a 128-row tile, an MLP padded on the K side, and both routes (16-byte accesses; a head_dim that is no multiple of 8 takes the general
kernels).

Bar: this library sits 1.31e-2 (1 layer) and 1.75e-2 (2 layers) from the oracle at the tower's full size, the distance that last-bit
differences grow to through four int8 quantisations a layer (tests/test_bitvla_vit_ref_gpu.py); 3e-2 is that with head-room of 1.7x."""
import ctypes as C

import numpy as np
import pytest

from tests.gpu_util import bf16_bits, bits_to_bf16_tensor, rel_l2, require_cuda
from tests.test_bitvla_vit_ref_gpu import FIELDS, LayerC, bind, drive, make_vit, vit_to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads,ffn,n_patches,n_layers", [
    (1152, 16, 4304, 131, 1), (1152, 16, 4304, 9, 1), (384, 3, 400, 257, 2), (256, 4, 512, 100, 2),
    (384, 32, 256, 40, 1),   # head_dim 12: general kernels
    (1408, 16, 512, 33, 1),  # rows longer than the register kernels hold: general kernels
    (256, 4, 272, 5, 1),     # the GEMV's rows: general kernels
    (1152, 8, 512, 200, 1), (512, 2, 256, 257, 1),  # head_dim 144 and 256 from 193 patches on: attention on CTA pairs
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


@pytest.mark.parametrize("heads", [16, 32])  # head_dim 24: 16-byte accesses; 12: the general kernels
def test_rewritten_biases_are_heard(oracle, heads):
    """set_layer binds the caller's vectors and copies only the q, k and v packs and scales: a bias rewritten in place counts from the next
    forward on, with the bits of a context that was given the new values."""
    torch = require_cuda()
    from vla_cpp_b200 import api

    cfg = dict(hidden=384, n_heads=heads, ffn=400, n_patches=40, patch_flat=588, ln_eps=1e-6, mm_out=128)
    rng = np.random.default_rng(heads)
    lib, dw = bind(api.lib()), vit_to_dev(oracle, make_vit(oracle, rng, 1, cfg))
    lw = dw["layers"][0]
    patches = bits_to_bf16_tensor(oracle.f32_to_bf16_bits(rng.uniform(-1, 1, (40, 588)).astype(np.float32)))
    ctx = lib.bitvla_vit_cuda_init(1, 384, heads, 400, 40, 588, 1e-6, 128)
    assert ctx
    try:
        lib.bitvla_vit_cuda_set_layer(ctx, 0, C.byref(LayerC(**{n: lw[n].data_ptr() for n in FIELDS})))
        lib.bitvla_vit_cuda_set_embed(ctx, dw["patch_w"].data_ptr(), dw["patch_b"].data_ptr(), dw["pos"].data_ptr())
        lib.bitvla_vit_cuda_set_mmproj(ctx, dw["mm_w1"].data_ptr(), dw["mm_b1"].data_ptr(), dw["mm_w2"].data_ptr(), dw["mm_b2"].data_ptr())
        out = torch.empty((40, 128), dtype=torch.bfloat16, device="cuda")
        before = None
        for name in (None, "q_b", "k_b", "v_b", "o_b", "fc1_b", "fc2_b"):
            if name:
                lw[name].copy_(torch.randn(lw[name].shape, device="cuda") * 0.5)
            assert lib.bitvla_vit_cuda_forward(ctx, patches.data_ptr(), out.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            torch.cuda.synchronize()
            assert torch.equal(out, drive(lib, cfg, dw, patches)), name
            # (a bias of k moves every score of a query alike but for rounding: only the comparison above is for it)
            assert before is None or name == "k_b" or not torch.equal(out, before), name
            before = out.clone()
    finally:
        lib.bitvla_vit_cuda_free(ctx)
    assert api.device_status() == 0
