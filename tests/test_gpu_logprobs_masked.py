"""arcs_logprobs_batch on rows masked with a large negative number (or with logits far from zero in
general): what is masked adds nothing to the sum, wherever it lies, and a row of nothing else has the
sum of its equals. And the selector's path probability over such rows. Against the CPU oracle's fp64
sums: ids bit-exact, log probabilities within 1e-6 (as for other rows) plus the last place of an fp64
number of their size."""
import numpy as np
import pytest
import torch

import orc
from arcinfer_b200 import synth
from test_gpu_dflash import _run
from test_oracle_pin import dflash_case

pytestmark = pytest.mark.gpu
TOL = 1e-6
LOWEST = {False: float(np.finfo(np.float32).min), True: -3.3895313892515355e38}  # the types' own


def _mask(x, where, fill):
    V = x.shape[1]
    if where == "front":
        x[:, : V - V // 4] = fill
    elif where == "back":
        x[:, V // 4 :] = fill
    elif where == "all but a few":
        keep = x[:, V // 3 : V // 3 + 5].copy()
        x[:] = fill
        x[:, V // 3 : V // 3 + 5] = keep
    elif where == "all":
        x[:] = fill
    elif where == "ends":  # the threads' first elements masked in some places, not in others
        x[:, : V // 2 : 2] = fill
        x[:, V // 2 :] = fill


def _check(x, bf16, top_n, rows):
    import arcinfer_b200 as ab

    lg = torch.from_numpy(x).cuda()
    out = ab.logprobs_batch(lg.bfloat16() if bf16 else lg, None, top_n)
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert got["status"][0] == 0
    for r in rows:
        lse, _, ids, tlp = orc.logprobs(x[r], -1, min(top_n, x.shape[1]))
        tol = TOL + 2.0**-52 * abs(lse)
        assert abs(got["lse"][r] - lse) <= tol, (r, got["lse"][r], lse)
        n = len(ids)
        if n:
            assert np.array_equal(got["top_id"][r, :n], ids), r
            assert np.allclose(got["top_logprob"][r, :n], tlp, rtol=2.0**-51, atol=tol)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,V,top_n", [(1, 151936, 20), (3, 8000, 0), (3, 41003, 256), (460, 21000, 0), (460, 21000, 20)])
def test_masked_rows(bf16, B, V, top_n):
    g = np.random.default_rng(V + top_n)
    base = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    for fill in (-1e9, -1e12, -1e30, LOWEST[bf16], -np.inf):
        for where in ("front", "back", "all but a few", "ends", "all"):
            if where == "all" and fill == -np.inf:
                continue  # (no sum to speak of)
            x = base.copy()
            _mask(x, where, fill)
            if bf16:
                x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(x))
            _check(x, bf16, top_n, range(0, B, max(1, B // 4)))


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("size", [2.0**24, 2.0**25, 1e10, 1e30, 3e38])
def test_large_logits(bf16, size):
    """the largest logit far from zero, on its own and among others near it; and both signs"""
    g = np.random.default_rng(7)
    V = 30011
    x = (g.standard_normal((5, V)) * 3).astype(np.float32)
    x[0, 20000] = size
    x[1] = (size * (1 + 1e-7 * g.standard_normal(V))).astype(np.float32)
    x[2] = (-size * (1 + 1e-7 * g.standard_normal(V))).astype(np.float32)
    x[3] = (size * g.uniform(-1, 1, V)).astype(np.float32)
    x[4, ::2] = -size
    if bf16:
        x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(x))
    _check(x, bf16, 12, range(5))


@pytest.mark.parametrize("fill", [-1e9, -1e30, LOWEST[False]])
def test_selector_over_masked_logits(fill):
    """the path probability, and where it cuts, when the front of the vocabulary is masked"""
    g = np.random.default_rng(11)
    V, rank, nd, slots = 40000, 64, 5, 3
    lgs, hps = [], []
    for _ in range(slots):
        l, h, pred, succ = dflash_case(g, V, rank, nd, 0.5)
        l[:, : V // 2] = fill
        lgs.append(l)
        hps.append(h)
    logits, hproj = np.stack(lgs), np.stack(hps)
    tok = g.integers(0, V, slots).astype(np.int32)
    cuts = 0
    for min_p in (0.02, 0.5):
        out = _run(logits, hproj, pred, succ, tok, 16, nd, min_p)
        for s in range(slots):
            want, pp = orc.dflash_select(logits[s], hproj[s], pred, succ, 16, nd, int(tok[s]), min_p)
            n = int(out["n_out"][s])
            assert n == len(want) and np.array_equal(out["tokens"][s, :n], want), s
            seen = ~np.isnan(pp)
            assert np.array_equal(seen, ~np.isnan(out["path_p"][s]))
            assert np.allclose(out["path_p"][s][seen], pp[seen], rtol=2e-5, atol=0)  # (the reference's float sums over blocks)
            cuts += n < nd
    assert cuts > 0
