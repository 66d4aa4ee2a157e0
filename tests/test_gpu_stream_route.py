"""The streaming route of sample_batch (stream and finish kernel), which serves every unmasked call
whose rows do not fit on the chip or whose lists are long: the batteries and the overflowing rows of
test_gpu_sample.py at sizes that take it. Few rows (cut into segments, merged by a CTA a row) go
there by a bound on the history above what rows on the chip take, wide batches (a row to an item,
finished by a warp) by their size. Each call's route is asked for beforehand. Bit-exact against the
CPU oracle, probabilities within 1e-6, as there."""
import numpy as np
import pytest

from arcinfer_b200 import capi, synth
from cases import rand_logits, rand_params, rand_recent
from test_gpu_sample import _batch

pytestmark = pytest.mark.gpu
LONG = 2049  # a history bound that no row on the chip has


def _run(x, bf16, params, hists, us, biases, rows=None, long=True, **kw):
    from gpuutil import check_rows, run_gpu_sample

    B, V = x.shape
    bound = max(LONG if long else 0, max(len(h) for h in hists))
    assert capi.lib.arcs_sample_launches(B, V, int(bf16), 0, bound, max(len(b) for b in biases) if biases else 0) == 2
    xb = synth.f32_to_bf16_bits(x) if bf16 else x
    out = run_gpu_sample(xb, bf16, params, hists, us, biases, max_hist=bound, **kw)
    check_rows(out, xb, bf16, params, hists, us, biases, rows=rows, tag=str(kw))


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("pen", [False, True])
def test_few_rows(bf16, pen):
    g = np.random.default_rng(600 + 2 * bf16 + pen)
    for V, B in [(2, 3), (33, 4), (257, 5), (1000, 8), (4099, 6), (8192, 4), (20000, 6), (151936, 3), (262144, 2)]:
        x, params, hists, us, biases, _ = _batch(g, B, V, pen, [0, 1, 2])
        for stride, off in [(None, 0), (V + 5, 3)]:
            _run(x, bf16, params, hists, us, biases, stride=stride, offset=off)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,V", [(300, 32001), (900, 5003)])
def test_wide_batches(bf16, B, V):
    """rows of all settings side by side: greedy, few candidates, 256 of them, raising penalties"""
    g = np.random.default_rng(B)
    V *= 1 + bf16  # (so that rows of either type take as much room)
    x, params, hists, us, biases, _ = _batch(g, B, V, True, [0, 1, 2])
    _run(x, bf16, params, hists, us, biases, rows=range(0, len(x), 13), long=False, stride=V + 5, offset=3)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,V", [(4, 60000), (310, 33000)])
def test_long_bias_lists_and_raising_penalties(bf16, B, V):
    """every listed token in the table: more than 64 bias entries, bans, ids that repeat, penalties that raise"""
    g = np.random.default_rng(V)
    V *= 1 + bf16
    x = np.stack([rand_logits(g, V, b % 3) for b in range(B)])
    params = synth.make_params(B, top_p=0.95)
    params["top_k"] = np.array([1, 20, 64, 65, 256, 0])[np.arange(B) % 6]
    params["temperature"] = np.array([0.0, 0.7, 1.0, 1.5])[np.arange(B) % 4]
    params["repeat_penalty"] = np.array([0.8, 1.0, 1.3])[np.arange(B) % 3]
    params["presence_penalty"] = np.array([-0.4, 0.5])[np.arange(B) % 2]
    params["frequency_penalty"] = np.array([-0.1, 0.3, 0.0])[np.arange(B) % 3]
    params["repeat_last_n"] = np.array([64, -1, 0])[np.arange(B) % 3]
    hists = [np.concatenate([g.integers(0, V, 200), g.integers(0, 40, 60), [V - 1, -1, V]]).astype(np.int32) for _ in range(B)]
    biases = [[(int(t), float(v)) for t, v in zip(g.integers(0, V, n), g.choice([-100.0, -3.0, 2.5, 40.0], n))] for n in g.integers(3, 200, B)]
    for b in biases:
        b += [b[0], (b[1][0], -0.5)]  # ids that repeat
    _run(x, bf16, params, hists, g.random(B), biases, rows=range(0, B, max(1, B // 24)), long=B < 100)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,V", [(5, 40000), (300, 32768)])
def test_rows_that_overflow_the_lists(bf16, B, V):
    """ascending logits make every element a survivor of the stream: the per-item lists overflow and
    the finishing step reads the rows again"""
    g = np.random.default_rng(B + V)
    V *= 1 + bf16
    x = np.tile(np.sort((g.standard_normal((5, V), dtype=np.float32) * 3).astype(np.float32), axis=1), (B // 5, 1))
    x[1] = x[1, ::-1]  # nothing after the first elements survives
    x[2, ::7] = x[2, 5]  # masses of equal values
    x[3] = 0.25
    ps, biases, hists = [], [], []
    for _ in range(B):
        p, bias = rand_params(g, V, True)
        ps.append(p)
        biases.append(bias)
        hists.append(np.concatenate([rand_recent(g, V), np.arange(V - 40, V)]).astype(np.int32))  # the best tokens are penalised
    _run(x, bf16, np.concatenate(ps), hists, g.random(B), biases, rows=list(range(5)) + list(range(5, B, 37)), long=B < 100)
