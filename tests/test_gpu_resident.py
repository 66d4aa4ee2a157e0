"""Rows held whole on the chip: sizes about a slice's and a cluster's borders, unaligned rows, lists
that repeat ids, k from 1 to 256, rows that overflow a slice's candidates (masses of equal
logits), and the number of rows at which the call changes to the streaming kernels (the columns of
vocabulary shards: test_gpu_vocab_shard.py). Ids, counts and adjusted logits bit-exact against the CPU oracle, probabilities within
1e-6 (the last rounding of a float exponential: 2^-24, with the same sums in the same order)."""
import numpy as np
import pytest

from arcinfer_b200 import synth
from cases import rand_logits

pytestmark = pytest.mark.gpu


def _lists(g, B, V, H):
    hists = [np.concatenate([g.integers(0, V, H), g.integers(0, min(V, 40), H // 2), np.full(3, V - 1), np.full(2, -1), np.full(1, V)]).astype(np.int32) for _ in range(B)]
    biases = [[(int(t), float(v)) for t, v in zip(g.integers(0, V, 9), g.choice([-100.0, -3.0, 2.5, 40.0], 9))] for _ in range(B)]
    for b in biases:
        b += [b[0], (b[1][0], -0.5)]  # ids that repeat
    return hists, biases


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("V", [1, 8, 63, 65, 1023, 4097, 32771, 65536, 262147])
def test_sizes(bf16, V):
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(V)
    B = 6
    x = np.stack([rand_logits(g, V, b % 3) for b in range(B)])
    xb = synth.f32_to_bf16_bits(x) if bf16 else x
    params = synth.make_params(B, top_p=0.95)
    params["top_k"] = [1, 20, 64, 65, 256, 40]
    params["temperature"] = [0.0, 0.7, 1.0, 1.0, 1.5, 1.0]
    params["repeat_penalty"] = [1.0, 1.1, 1.3, 0.8, 1.0, 1.1]
    params["presence_penalty"] = [0.0, 0.5, -0.4, 0.0, 0.0, 0.2]
    params["frequency_penalty"] = [0.0, 0.3, 0.0, -0.1, 0.0, 0.0]
    params["repeat_last_n"] = [64, 64, -1, 10, 64, 0]
    hists, biases = _lists(g, B, V, 200)
    us = g.random(B)
    for stride, off in [(None, 0), (V + 3, 1)]:
        out = run_gpu_sample(xb, bf16, params, hists, us, biases, stride=stride, offset=off)
        check_rows(out, xb, bf16, params, hists, us, biases, tag=f"stride={stride}")


@pytest.mark.parametrize("bf16", [False, True])
def test_equal_and_infinite_logits(bf16):
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(3)
    V, B = 50000, 5
    x = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    x[0] = 1.25
    x[1, 100:] = -np.inf
    x[2, 7:] = -np.inf
    x[3, ::2] = 9.0
    x[4].sort()
    params = synth.make_params(B, top_k=40, top_p=1.0, repeat_penalty=1.1, repeat_last_n=-1)
    hists = [np.arange(50, dtype=np.int32) for _ in range(B)]
    us = g.random(B)
    xb = synth.f32_to_bf16_bits(x) if bf16 else x
    out = run_gpu_sample(xb, bf16, params, hists, us)
    check_rows(out, xb, bf16, params, hists, us, rows=[0, 1, 3, 4])
    assert 0 <= out["token"][2] < 7


@pytest.mark.parametrize("V", [1100, 1536, 2047, 60000])
def test_slices_that_overflow(V):
    """more candidates than a slice keeps: narrow rows give fewer chunks than the 256 wanted, so that
    no threshold is found; equal and infinite logits all reach theirs. Many rows, again and again: the
    threads of a slice must all go the same way"""
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(V)
    B = 24
    x = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    x[::3] = 0.5
    x[1::6] = -np.inf
    x[1::6, V // 2] = 1.0
    xb = synth.f32_to_bf16_bits(x)
    params = synth.make_params(B, top_k=256, top_p=1.0)
    us = g.random(B)
    first = run_gpu_sample(xb, True, params, None, us)
    check_rows(first, xb, True, params, None, us)
    for _ in range(20):
        again = run_gpu_sample(xb, True, params, None, us)
        assert all(np.array_equal(again[k], first[k]) for k in ("token", "n_cand", "cand_id"))


@pytest.mark.parametrize("V,B", [(151936, 55), (151936, 56), (32000, 222), (32000, 223), (32000, 445)])
def test_where_the_route_changes(V, B):
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(B)
    x = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    params = synth.make_params(B, top_k=50, top_p=0.95, repeat_penalty=1.1, repeat_last_n=-1)
    hists = [g.integers(0, V, 300).astype(np.int32) for _ in range(B)]
    us = g.random(B)
    out = run_gpu_sample(x, False, params, hists, us)
    check_rows(out, x, False, params, hists, us, rows=range(0, B, max(1, B // 12)))


@pytest.mark.parametrize("H", [1, 31, 33, 257, 1100, 2000])
def test_histories_that_repeat(H):
    """one id throughout, few ids, ids as text repeats them, low ids only; windows that begin inside;
    biases on ids of the history and on others"""
    from arcinfer_b200 import capi
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(H)
    V, B = 30011, 8
    assert all(capi.lib.arcs_sample_launches(B, V, t, 0, H, 4) == 1 for t in (0, 1))
    x = (g.standard_normal((B, V), dtype=np.float32) * 2).astype(np.float32)
    kinds = [np.full(H, 17), g.integers(0, 3, H), np.minimum(g.zipf(1.3, H), V) - 1, g.integers(0, 300, H), g.integers(0, V, H), np.arange(H) % 40, np.full(H, V - 1), g.integers(-2, V + 3, H)]
    hists = [k.astype(np.int32) for k in kinds]
    x[:, :40] += 8.0  # what repeats is likely
    params = synth.make_params(B, top_k=40, top_p=0.95, repeat_penalty=1.15, presence_penalty=0.2, frequency_penalty=0.01)
    params["repeat_last_n"] = [-1, 64, 10, 256, 0, 5, 64, -1]
    biases = [[(17, 1.5), (int(h[0]), -0.5), (int(h[-1]), -100.0 if b % 4 == 3 else 2.0), (V - 2, 3.0)] for b, h in enumerate(hists)]
    us = g.random(B)
    for bf16 in (False, True):
        xb = synth.f32_to_bf16_bits(x) if bf16 else x
        for bias in (None, biases):
            out = run_gpu_sample(xb, bf16, params, hists, us, bias)
            check_rows(out, xb, bf16, params, hists, us, bias)


def test_long_lists_take_the_other_route():
    from gpuutil import check_rows, run_gpu_sample

    g = np.random.default_rng(9)
    V, B = 20000, 3
    x = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    params = synth.make_params(B, top_k=30, top_p=0.95, repeat_penalty=1.1, repeat_last_n=-1)
    us = g.random(B)
    for H in (2048, 2049):
        hists = [g.integers(0, V, H).astype(np.int32) for _ in range(B)]
        out = run_gpu_sample(x, False, params, hists, us)
        check_rows(out, x, False, params, hists, us)
