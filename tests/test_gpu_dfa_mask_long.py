"""The automaton mask over tokens at the borders of what a thread holds in registers: 1, 7, 8, 9, 15,
16, 17 and up to 70 bytes, under an automaton that lets most bytes live; against the CPU walk."""
import numpy as np
import pytest
import torch

import orc
from arcinfer_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("classes", [31, 32])
def test_long_tokens(classes):
    import arcinfer_b200 as ab

    g = np.random.default_rng(classes)
    V, S = 3333, 40
    ln = g.choice([0, 1, 7, 8, 9, 15, 16, 17, 24, 33, 70], V)
    off = np.zeros(V + 1, np.uint32)
    off[1:] = np.cumsum(ln)
    by = g.integers(0, 256, int(off[-1])).astype(np.uint8)
    table, dead = synth.make_dfa(g, S=S, classes=classes)
    states = np.array([0, 3, dead, S - 1, 7], np.int32)
    out = ab.dfa_mask(torch.from_numpy(table.view(np.int16)).cuda(), dead, torch.from_numpy(states).cuda(), torch.from_numpy(off.view(np.int32)).cuda(),
                      torch.from_numpy(by).cuda())
    got = out.cpu().numpy().view(np.uint32)
    for i, s in enumerate(states):
        assert np.array_equal(got[i], orc.dfa_mask(table, dead, int(s), off, by)), s
    assert got[0].any()
