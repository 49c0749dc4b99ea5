"""The engine's attention of a few observations, whose keys are cut over the CTAs of a cluster and merged there: every number of slices,
ragged last blocks, row tiles that are not full, head sizes 64, 128 and 256, and slices whose keys are all hidden."""
import pytest

from tests.test_engine_gpu import run_case

pytestmark = pytest.mark.gpu


# P + chunk + 1 keys in blocks of 64, at least two blocks a slice; rows = (n_q / n_kv) * (chunk + 1) in tiles of 128
@pytest.mark.parametrize("n_obs,P,hd,n_q,n_kv,chunk,pad", [
    (2, 206, 256, 8, 1, 50, None),       # 5 blocks: 2 slices of 2 and 3
    (2, 333, 256, 8, 1, 50, (2, 330)),   # 6 blocks: 3 slices, the middle one hidden
    (5, 816, 256, 8, 1, 50, (3, 810)),   # 14 blocks: 7 slices, five of them hidden
    (2, 1100, 256, 8, 1, 50, None),      # 18 blocks: 8 slices of 2 or 3
    (2, 600, 128, 4, 2, 10, (0, 599)),   # 10 blocks: 5 slices of one part-filled row tile
    (9, 816, 256, 8, 1, 50, None),       # 36 units: 4 slices an SM each
    (2, 800, 64, 6, 2, 20, (1, 500)),    # 13 blocks: 6 slices, two CTAs an SM
])
def test_key_slices_match_the_oracle(oracle, n_obs, P, hd, n_q, n_kv, chunk, pad):
    # inputs are rounded to bf16 on the way (2^-9 each): the bounds of the engine's own small cases
    w, d = run_case(oracle, 77, n_obs=n_obs, P=P, pad=pad, check_obs=[0, n_obs - 1], model=0, L=1, H=256, n_q=n_q, n_kv=n_kv, hd=hd,
                    inter=256, chunk=chunk, A=32, sd=32, T=2)
    assert w < 1e-2 and d < 3e-2, (w, d)
