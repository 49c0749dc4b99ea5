"""The whole Euler loop of one observation as one persistent kernel (csrc/chunk_loop.cu) against the launch-per-operator
path of the same engine and against the oracle (src/models/pi0.cpp:570-588, src/models/smolvla.cpp:1393-1418)."""
import os

import numpy as np
import pytest

from tests.gpu_util import require_cuda

pytestmark = pytest.mark.gpu


def _engine(torch, vb, policy, seed=3):
    import bench

    return bench.build_pi0_engine(torch, vb, torch.device("cuda", 0), 1, seed, policy)


def _with_loop(flag, fn):
    old = os.environ.get("VLAB200_CHUNK_LOOP")
    os.environ["VLAB200_CHUNK_LOOP"] = flag
    try:
        return fn()
    finally:
        if old is None:
            del os.environ["VLAB200_CHUNK_LOOP"]
        else:
            os.environ["VLAB200_CHUNK_LOOP"] = old


@pytest.fixture(autouse=True)
def loop_phases(monkeypatch):
    """Every one-observation call that these tests make with the loop kernel on must have run it, not the launch-per-operator path:
    both meet the same bounds.  -> phases per Euler step of each such call."""
    import vla_cpp_b200 as vb

    phases, denoise = [], vb.PolicyEngine.denoise

    def checked(self, x0, *a, **kw):
        out = denoise(self, x0, *a, **kw)
        if x0.shape[0] == 1 and os.environ.get("VLAB200_CHUNK_LOOP", "1") != "0":
            phases.append(self.loop_phases)
            assert phases[-1] > 0
        return out

    monkeypatch.setattr(vb.PolicyEngine, "denoise", checked)
    return phases


@pytest.mark.parametrize("policy", ["pi0", "smolvla", "pi05"])
def test_loop_kernel_matches_operator_path(policy):
    torch = require_cuda()
    import vla_cpp_b200 as vb

    eng, x0, state = _engine(torch, vb, policy)
    ref = _with_loop("0", lambda: eng.denoise(x0, state))
    out = _with_loop("1", lambda: eng.denoise(x0, state))
    again = _with_loop("1", lambda: eng.denoise(x0, state))
    torch.cuda.synchronize()
    assert vb.device_status() == 0
    assert torch.isfinite(out).all()
    rel = ((out - ref).norm() / ref.norm()).item()
    assert rel <= 1e-2, rel  # both paths round activations to bf16 at different points
    assert torch.equal(out, again)  # every sum has a fixed order


@pytest.mark.parametrize("policy", ["pi0", "pi05"])
def test_loop_kernel_rows_exchanged_over_k(policy):
    """816 prefix keys at head_dim 256: the attention rows a CTA group exchanges land where its K tiles were.  A row that arrived before
    its reader had finished would change some of the runs."""
    torch = require_cuda()
    import vla_cpp_b200 as vb

    eng, x0, state = _engine(torch, vb, policy, seed=11)
    assert eng.prefix_len == 816
    ref = _with_loop("0", lambda: eng.denoise(x0, state))
    outs = _with_loop("1", lambda: [eng.denoise(x0, state) for _ in range(40)])
    torch.cuda.synchronize()
    assert vb.device_status() == 0
    assert ((outs[0] - ref).norm() / ref.norm()).item() <= 1e-2  # both paths round activations to bf16 at different points
    assert all(torch.equal(outs[0], o) for o in outs[1:])


def test_loop_kernel_hidden_key_range_and_prefix_length():
    """SmolVLA-shaped: a pad range hides prefix keys; then the prefix in use shrinks (the phase table is rebuilt)."""
    torch = require_cuda()
    import vla_cpp_b200 as vb

    eng, x0, state = _engine(torch, vb, "smolvla", seed=7)
    pad = torch.tensor([[140, 170]], dtype=torch.int32, device="cuda")
    ref = _with_loop("0", lambda: eng.denoise(x0, state, pad_ranges=pad))
    out = _with_loop("1", lambda: eng.denoise(x0, state, pad_ranges=pad))
    plain = _with_loop("1", lambda: eng.denoise(x0, state))
    torch.cuda.synchronize()
    assert ((out - ref).norm() / ref.norm()).item() <= 1e-2
    assert ((out - plain).norm() / plain.norm()).item() > 1e-4  # the hidden keys matter
    eng.set_prefix_len(eng.prefix_len - 33)
    ref2 = _with_loop("0", lambda: eng.denoise(x0, state))
    out2 = _with_loop("1", lambda: eng.denoise(x0, state))
    torch.cuda.synchronize()
    assert vb.device_status() == 0
    assert ((out2 - ref2).norm() / ref2.norm()).item() <= 1e-2
    assert ((out2 - plain).norm() / plain.norm()).item() > 1e-4


@pytest.mark.parametrize("policy", ["pi0", "smolvla"])
def test_loop_kernel_full_depth_against_oracle(oracle, policy):
    """The benchmark configurations at full depth (18 x 10 and 16 x 10 layer-steps), one observation, forced through the
    loop kernel: final action chunk rel-L2 <= 1e-2 against the float32 oracle, as for the operator path."""
    from tests.test_engine_gpu import PI0_FULL, SMOLVLA_FULL, run_case

    if policy == "pi0":
        w, d = _with_loop("1", lambda: run_case(oracle, 71, n_obs=1, P=816, check_obs=[0], sigma=0.02, **PI0_FULL))
    else:
        w, d = _with_loop("1", lambda: run_case(oracle, 72, n_obs=1, P=177, pos_base=170, pad=(160, 176), check_obs=[0], sigma=0.02,
                                               **SMOLVLA_FULL))
    print(f"loop kernel {policy} full depth: rel_l2={w:.3e} displacement rel_l2={d:.3e}")
    assert w < 1e-2 and d < 3e-2, (w, d)


def test_loop_kernel_other_shapes_against_oracle(oracle):
    """head_dim 128 (its own kernel instantiation), and a small SmolVLA-shaped expert with cross-attention layers, a hidden key
    range and rebased suffix positions; one observation each, so both take the loop kernel."""
    from tests.test_engine_gpu import run_case

    w, d = _with_loop("1", lambda: run_case(oracle, 73, n_obs=1, P=40, model=0, L=2, H=128, n_q=2, n_kv=1, hd=128, inter=256,
                                           chunk=10, A=32, sd=32, T=2))
    assert w < 1e-2 and d < 3e-2, (w, d)
    w, d = _with_loop("1", lambda: run_case(oracle, 74, n_obs=1, P=30, pos_base=27, pad=(20, 29), model=1, L=4, H=192, n_q=6, n_kv=2,
                                           hd=64, inter=384, chunk=10, A=32, sd=32, T=2, self_every=2))
    assert w < 1e-2 and d < 3e-2, (w, d)


@pytest.mark.parametrize("kw", [
    # a CTA's share of the keys does not fit at once: several key blocks with a running maximum
    dict(P=2100, model=0, L=2, H=256, n_q=8, n_kv=1, hd=256, inter=512, chunk=50, A=32, sd=32, T=2),
    # 64 suffix rows, pi0's widths: the longest A tile, staged sums behind it
    dict(P=24, model=0, L=1, H=1024, n_q=8, n_kv=1, hd=256, inter=4096, chunk=63, A=32, sd=32, T=1),
    # widths that are no multiple of 64 columns or of the CTA groups, CTAs without keys, one action token
    dict(P=3, pos_base=3, model=1, L=3, H=208, n_q=5, n_kv=5, hd=64, inter=336, chunk=1, A=16, sd=32, T=2, self_every=2),
    # more attention units than CTA groups of two
    dict(P=70, pos_base=70, model=1, L=2, H=320, n_q=32, n_kv=32, hd=64, inter=640, chunk=50, A=48, sd=32, T=1, self_every=2),
    # a deep expert: 164 products in the phase table.  N(0, 0.02) weights as in the other deep cases: at unit scale this narrow stack
    # amplifies roundings over 40 layers until either path is 1.4e-2 from the oracle
    dict(P=20, model=0, L=40, H=128, n_q=2, n_kv=1, hd=64, inter=256, chunk=10, A=32, sd=32, T=2, sigma=0.02),
], ids=["key_blocks", "rows64", "ragged", "many_units", "deep"])
def test_loop_kernel_work_split_edges(oracle, kw):
    from tests.test_engine_gpu import run_case

    w, d = _with_loop("1", lambda: run_case(oracle, 81, n_obs=1, **kw))
    assert w < 1e-2 and d < 3e-2, (w, d)


WIDE = dict(model=0, L=1, H=1024, n_q=8, n_kv=1, hd=256, chunk=50, A=32, sd=32, T=2)


@pytest.mark.parametrize("kw", [
    # gate/up in two parts of its columns, Wdown in one; then both in parts, and a part of K that ends within a 64-column block
    dict(P=40, inter=6144, **WIDE),
    dict(P=40, inter=8192, **WIDE),
    dict(P=40, inter=12304, **WIDE),
    # 320 attention units (three rounds of them per CTA), q|k|v in parts of its columns, Wo in parts of K
    dict(P=70, model=1, L=2, H=128, n_q=160, n_kv=160, hd=64, inter=256, chunk=50, A=32, sd=32, T=2, self_every=2),
], ids=["inter6144", "inter8192", "inter12304", "heads160"])
def test_loop_kernel_products_in_several_phases(oracle, loop_phases, kw):
    from tests.test_engine_gpu import run_case

    w, d = _with_loop("1", lambda: run_case(oracle, 83, n_obs=1, **kw))
    assert loop_phases[-1] > 5 * kw["L"] + 4  # more than one phase per product
    assert w < 1e-2 and d < 3e-2, (w, d)


def test_loop_kernel_gated_residual_in_parts_of_k(oracle, loop_phases):
    """pi0.5: the gate scales every part of Wdown's K on its way into the residual stream."""
    from tests.test_pi05_gpu import run_pi05

    err = _with_loop("1", lambda: run_pi05(oracle, 84, 1, 40, L=2, H=1024, n_q=8, n_kv=1, hd=256, inter=9216, chunk=50, A=32, T=2))
    assert loop_phases[-1] > 5 * 2 + 2
    assert err <= 1e-2, err
