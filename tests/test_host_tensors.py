"""Tensors on the host are refused before anything is launched: the kernels would be given host addresses."""
import numpy as np
import pytest
import torch

import arcinfer_b200 as ab
from arcinfer_b200 import capi, synth


def _calls():
    lg, u = torch.zeros(2, 64), torch.zeros(2, dtype=torch.float64)
    p = capi.params_to_device(synth.make_params(2), "cpu")
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    table = torch.zeros(1, 256, dtype=torch.int16)
    book = torch.zeros(64, 8, dtype=torch.int16)
    return {
        "arcs_accept_batch": lambda: ab.accept_batch(i32(1, 2), i32(0, 2), i32(1), i32(0, 1)),
        "arcs_dfa_mask": lambda: ab.dfa_mask(table, 0, i32(0), i32(0, 1), torch.zeros(1, dtype=torch.uint8)),
        "arcs_adjusted_batch": lambda: ab.adjusted_batch(lg, p),
        "arcs_logprobs_batch": lambda: ab.logprobs_batch(lg, None, 2),
        "arcs_dflash_select": lambda: ab.dflash_select(lg.view(1, 2, 64), torch.zeros(1, 2, 8), book, book, i32(0), topk=4, max_drafts=2),
        "arcs_sample_batch": lambda: capi.SamplePlan(lg, p, u).launch(),
        "arcs_merge_batch": lambda: ab.merge_batch(torch.zeros(1, 2, 256, dtype=torch.int32), torch.zeros(1, 2, 256), torch.zeros(1, 2, dtype=torch.int32), p, u, 64),
    }


@pytest.mark.parametrize("name", sorted(_calls()))
def test_refused(name, monkeypatch):
    launched = []
    monkeypatch.setattr(capi.lib, name, lambda *a: launched.append(a) or 0)
    # (as on a machine with a GPU, whose current device a tensor without a device index must not fall back to)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: 0, raising=False)
    monkeypatch.setattr(capi, "_workspaces", {})
    with pytest.raises(ValueError):
        _calls()[name]()
    assert not launched
