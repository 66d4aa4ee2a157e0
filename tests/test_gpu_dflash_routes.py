"""The selector on either side of the rule that chooses how a path is found (all pairs scored first,
or walked position by position): ranks odd and even, K from 1 to 64, more positions than the first
route takes, rows with fewer numbers than K. Drafts bit for bit against the CPU restatement."""
import numpy as np
import pytest

import orc
from test_gpu_dflash import _run
from test_oracle_pin import dflash_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,rank,nd,topk,slots", [(700, 64, 3, 16, 2), (700, 64, 4, 16, 2), (700, 64, 4, 17, 2), (700, 64, 2, 8, 2), (700, 64, 3, 8, 2), (700, 64, 3, 9, 2),
                                                  (700, 1024, 4, 16, 2), (500, 32, 4, 16, 148), (500, 32, 4, 16, 149)])
def test_about_the_rule(V, rank, nd, topk, slots):
    test_either_route(V, rank, nd, topk, slots)


@pytest.mark.parametrize("V,rank,nd,topk,slots", [(900, 1, 7, 16, 3), (900, 7, 8, 1, 2), (900, 33, 8, 33, 3), (900, 255, 9, 16, 2), (700, 256, 1, 64, 2),
                                                  (700, 400, 7, 64, 3), (700, 1024, 3, 64, 2), (600, 256, 7, 16, 150), (600, 256, 7, 32, 40)])
def test_either_route(V, rank, nd, topk, slots):
    g = np.random.default_rng(V + rank + topk)
    lgs, hps = [], []
    for s in range(slots):
        l, h, pred, succ = dflash_case(g, V, rank, nd, 1.0)
        if s == 1:
            l[:, 3:] = np.nan  # fewer numbers than candidates
        lgs.append(l)
        hps.append(h)
    logits, hproj = np.stack(lgs), np.stack(hps)
    tok = g.integers(0, V, slots).astype(np.int32)
    for min_p in (0.0, 0.05):
        out = _run(logits, hproj, pred, succ, tok, topk, nd, min_p)
        for s in range(0, slots, max(1, slots // 8)):
            if s == 1:
                assert (out["tokens"][s][: int(out["n_out"][s])] < 3).all()
                continue
            want, _ = orc.dflash_select(logits[s], hproj[s], pred, succ, topk, nd, int(tok[s]), min_p)
            n = int(out["n_out"][s])
            assert n == len(want) and np.array_equal(out["tokens"][s, :n], want), (s, min_p)
