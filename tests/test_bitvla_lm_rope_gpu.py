"""The language model's q | k | v product with the rotation in its epilogue (one-CTA tiles of 128 columns, at some hundred rows) against the
separate rotation of the other tilings (few rows, CTA pairs): integer sums and the same roundings, so a sequence gives the same bits alone
and in a batch.  Sequence lengths that are no multiple of the tile's rows.  The captured launches tell which of the two a call took."""
import pytest

from tests.gpu_util import kernels_of, require_cuda

pytestmark = pytest.mark.gpu

NQ, NKV, HD = 20, 5, 128


# rotated in the epilogue: at a width of 2560 the pair tiling is estimated alike, at 1280 a tenth above; 854 rows run as pairs
@pytest.mark.parametrize("n_seq,seq,hidden,ffn,fused", [(5, 61, 2560, 6912, True), (3, 97, 2560, 6912, True), (14, 61, 2560, 6912, False),
                                                        (5, 61, 1280, 1024, True), (3, 128, 1280, 1024, True)])
def test_a_sequence_alone_and_in_a_batch(n_seq, seq, hidden, ffn, fused):
    torch = require_cuda()
    import vla_cpp_b200 as vb

    g = torch.Generator(device="cuda")
    g.manual_seed(n_seq)

    HID, FFN = hidden, ffn

    def tern(n, k):
        c = torch.randint(1, 4, (n * k // 4, 4), device="cuda", generator=g, dtype=torch.uint8)
        return c[:, 0] | (c[:, 1] << 2) | (c[:, 2] << 4) | (c[:, 3] << 6)

    def norm(k):
        return (1 + 0.1 * torch.randn(k, device="cuda", generator=g)).bfloat16()

    def ws(k, n=1):
        return torch.full((n,), (2 * k / 3) ** -0.5, device="cuda") * (1 + 0.1 * torch.rand(n, device="cuda", generator=g))

    hq, hkv = NQ * HD, NKV * HD
    layer = dict(attn_norm_w=norm(HID), attn_sub_norm_w=norm(hq), ffn_norm_w=norm(HID), ffn_sub_norm_w=norm(FFN), q_packed=tern(hq, HID), q_ws=ws(HID),
                 k_packed=tern(hkv, HID), k_ws=ws(HID), v_packed=tern(hkv, HID), v_ws=ws(HID), o_packed=tern(HID, hq), o_ws=ws(hq),
                 gate_up_packed=tern(2 * FFN, HID), gate_up_ws=ws(HID, 2), down_packed=tern(HID, FFN), down_ws=ws(FFN))
    lm = vb.BitvlaLM(HID, NQ, NKV, HD, FFN, [layer], norm(HID), rope_base=500000.0, rms_eps=1e-5, max_seq=seq + 3, max_batch=n_seq)
    x = torch.randn((n_seq, seq, HID), device="cuda", generator=g).bfloat16()
    together = lm.forward(x).clone()
    for i in range(n_seq):
        assert torch.equal(lm.forward(x[i:i + 1].contiguous())[0], together[i]), i
    assert vb.device_status() == 0
    split = [any("rope_split" in k for k in kernels_of(lambda: lm.forward(y))) for y in (x[:1].contiguous(), x)]
    assert split == [True, not fused], split
