"""arcs_logprobs_batch over regions of equal logits: which of them are among the alternatives (the lowest
ids), where such a region begins, ends or fills the row, with as many better elements as wanted, one
fewer, or none. Ids bit-exact against the CPU oracle, log probabilities within 1e-6."""
import numpy as np
import pytest

from arcinfer_b200 import synth
from test_gpu_logprobs_masked import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("top_n", [1, 20, 64, 65, 256])
@pytest.mark.parametrize("B,V", [(8, 8192), (448, 41001), (8, 41001), (8, 151937)])
def test_regions_of_equal_logits(bf16, top_n, B, V):
    g = np.random.default_rng(V + top_n)
    if B > 400 and top_n not in (20, 256):
        pytest.skip("the wide case once for either threshold")
    for level in (-np.inf, -1e30, 0.25):
        x = np.full((B, V), level, np.float32)
        x[0] = 0.5                                                                     # nothing else
        x[1, 7 * V // 8 :] = g.standard_normal(V - 7 * V // 8) * 3 + 20                # ordinary ones behind it
        x[2, 3 * V // 4 :] = g.standard_normal(V - 3 * V // 4) * 3 + 20
        x[3, : V // 16] = g.standard_normal(V // 16) * 3 + 20                          # before it
        x[4, g.permutation(V)[: top_n - 1]] = 1.0 + g.random(top_n - 1)                # one fewer than wanted
        x[5, g.permutation(V)[:top_n]] = 1.0 + g.random(top_n)                         # as many
        x[6, V // 2 : V // 2 + 50] = 2.0                                               # two levels
        x[7, : V // 3] = np.linspace(1, 2, V // 3)                                     # rising, then level
        if bf16:
            x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(x))
        # (row 4 is -inf throughout when one is wanted at that level: its sum is not defined, log 0 - inf)
        _check(x, bf16, top_n, [r for r in range(8) if not (r == 4 and top_n == 1 and level == -np.inf)])
        if B > 400:
            _check(x[::-1].copy(), bf16, top_n, range(B - 8, B))


@pytest.mark.parametrize("top_n", [20, 256])
def test_numbers_behind_nan(top_n):
    """a first tile without numbers gives no threshold"""
    import arcinfer_b200 as ab
    import torch

    V = 60000
    x = np.full((3, V), np.nan, np.float32)
    x[0, 9000:] = 0.5
    x[1, 9000:] = -np.inf
    x[1, 30000] = 1.0
    x[2, 100:110] = 3.0
    x[2, 20000:] = np.random.default_rng(1).standard_normal(V - 20000)
    out = ab.logprobs_batch(torch.from_numpy(x).cuda(), None, top_n)
    got = out["top_id"].cpu().numpy()
    for r in range(3):
        v = np.where(np.isnan(x[r]), -np.inf, x[r]).astype(np.float64)
        order = np.lexsort((np.arange(V), -v))
        want = order[~np.isnan(x[r][order])][:top_n]
        assert np.array_equal(got[r, : len(want)], want), r
    z = np.exp(x[2][~np.isnan(x[2])].astype(np.float64)).sum()
    assert abs(out["lse"][2].item() - np.log(z)) <= 1e-6
