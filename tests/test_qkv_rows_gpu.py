"""The folded q | k | v projection: rows that start on 16-byte boundaries only, every number of operand stages that the RoPE table leaves
room for (one CTA 4, 3, 2; pairs 6, 5, 4, 3), and more tiles than CTAs: the same bits from every tiling, and the oracle's within its bound."""
import pytest
from tests.gpu_util import require_cuda
from tests.test_denoise_attn_gpu import TOL, qkv_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_obs,n_q,n_kv,hd,S", [
    (1, 8, 1, 64, 51),     # one ragged row tile
    (40, 15, 5, 64, 51),   # six stages of pairs; 2,040 rows
    (40, 8, 1, 256, 51),   # five
    (25, 4, 2, 128, 90),   # a table of 45 KB
    (60, 3, 1, 64, 130),   # 7,800 rows, tiles that end in mid head
    (3, 2, 1, 128, 190),   # a table of 95 KB: two stages of one CTA, four of pairs
    (3, 1, 1, 256, 120),   # 120 KB: three stages of pairs, too large for one CTA
])
def test_rows_and_tilings(oracle, n_obs, n_q, n_kv, hd, S):
    torch = require_cuda()
    import vla_cpp_b200 as vb

    H, P = 320, 24
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(n_obs * S, H, device="cuda", generator=g).bfloat16()
    w = (torch.randn((n_q + 2 * n_kv) * hd, H, device="cuda", generator=g) * 0.05).bfloat16()
    rope = vb.rope_table(P, S, hd)
    n = n_obs * n_q * S * hd
    got = []
    only_pairs = hd * S > 24768
    try:
        if only_pairs:
            st = vb.KvStore(1, n_obs, n_kv, hd, P, S)
            with pytest.raises(vb.VlaB200Error):
                vb.qkv_rope_append(st, 0, x, None, w, rope, 1e-6, S, n_q)
        for tiling in (3,) if only_pairs else (0, 1, 3):
            vb.set_gemm_tiling(tiling)
            for shift in (0, 8):  # elements: 8 leaves q on a 16-byte boundary that is no 32-byte one
                st = vb.KvStore(1, n_obs, n_kv, hd, P, S)
                buf = torch.zeros(n + 16, dtype=torch.bfloat16, device="cuda")
                q = buf[shift:shift + n].view(n_obs, n_q, S, hd)
                assert q.data_ptr() % 32 == 2 * shift
                vb.qkv_rope_append(st, 0, x, None, w, rope, 1e-6, S, n_q, q_out=q)
                assert vb.device_status() == 0
                assert not buf[:shift].any() and not buf[shift + n:].any() and not st.k[0][:, :, :P].any() and not st.v[0][:, :, :P].any()
                got.append((q, st.k.clone(), st.v.clone()))
        vb.set_gemm_tiling(3 if only_pairs else 0)
        cfg = dict(H=H, n_q=n_q, n_kv=n_kv, hd=hd, S=S, P=P, eps=1e-6)
        assert qkv_case(oracle, cfg, min(n_obs, 4), seed=7, fold=True) < TOL
    finally:
        vb.set_gemm_tiling(0)
    for q, k, v in got[1:]:
        assert torch.equal(q, got[0][0]) and torch.equal(k, got[0][1]) and torch.equal(v, got[0][2])
