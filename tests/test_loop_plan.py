"""Which experts the one-observation loop kernel takes, from their sizes alone (csrc/chunk_loop.cu, host code: no GPU)."""
import pytest

COMMON = dict(steps=10, rms_eps=1e-6, rope_base=1e4, min_period=4e-3, max_period=4.0, action_dim=32, state_dim=32, self_every=1, chunk=50)
PI0 = dict(COMMON, model=0, n_layers=18, H=1024, n_q=8, n_kv=1, head_dim=256, inter=4096)
SMOLVLA = dict(COMMON, model=1, n_layers=16, H=720, n_q=15, n_kv=5, head_dim=64, inter=2048, self_every=2)


def phases(cfg, n_cta=120):
    from vla_cpp_b200 import api, build

    build.build()
    return api.loop_kernel_phases(cfg, n_cta)


@pytest.mark.parametrize("n_cta", [112, 120, 144])
def test_every_product_of_the_usual_experts_is_one_phase(n_cta):
    """Embedding (action-in, two products of the time MLP; pi0.5: action-in alone), five per layer, head."""
    assert phases(PI0, n_cta) == 3 + 18 * 5 + 1
    assert phases(SMOLVLA, n_cta) == 3 + 16 * 5 + 1
    assert phases(dict(PI0, model=2), n_cta) == 1 + 18 * 5 + 1


@pytest.mark.parametrize("H,inter", [(1024, 16), (1024, 4096), (1024, 5760), (1024, 5776), (1024, 8192), (1024, 12304), (768, 8704),
                                     (768, 8720), (768, 16384), (64, 16384)])
@pytest.mark.parametrize("chunk", [1, 50, 63])
def test_wide_mlps_take_more_phases(H, inter, chunk):
    if chunk == 63:  # 64 rows: half as wide
        inter = max(16, inter // 32 * 16)
    n = phases(dict(PI0, H=H, inter=inter, chunk=chunk))
    assert 94 <= n <= 3 + 18 * 8 + 1
    if (H, chunk) == (1024, 50):
        assert n == 94 + 18 * {16: 0, 4096: 0, 5760: 0, 5776: 1, 8192: 2, 12304: 3}[inter]


def test_fewer_ctas_take_more_phases():
    counts = [phases(PI0, n) for n in (120, 64, 32)]
    assert counts[0] < counts[1] < counts[2]


def test_what_does_not_fit():
    assert phases(dict(PI0, chunk=64)) == 0  # 65 suffix rows
    assert phases(dict(PI0, H=1032)) == 0  # no multiple of 16
    assert phases(dict(PI0, head_dim=96)) == 0
    assert phases(dict(PI0, inter=16384)) == 0  # nine phases a layer: a launch per operator is as fast
    assert phases(dict(PI0, n_layers=60)) == 0  # the phase table
    assert phases(PI0, 100) == 0 and phases(PI0, 0) == 0  # no whole clusters of eight
