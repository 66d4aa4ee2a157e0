"""arcs_logprobs_batch where its rows are cut and its thresholds are odd: rows whose pieces end on
and beside a unit's border, one and several rows to a CTA, rows of mostly -inf or NaN, many
alternatives; and the call without a workspace. Against the CPU oracle: ids bit-exact, log
probabilities within 1e-6. A term's exponent x = (l - ref) * log2 e is rounded once, to 2^-24 |x|, which
is 2^-24.5 |x| of the term; the special-function unit adds 2^-22.5, the fp32 sums over a chunk 3 * 2^-24.
Weighted by the terms' shares of the sum the |x| come to 12.5 at most with 131073 of them (one term of a
tenth of the sum, all others alike), so that the sum, and with it its logarithm, is within 8.7e-7 even
if no two errors cancel."""
import ctypes as C

import numpy as np
import pytest
import torch

import orc
from arcinfer_b200 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _rows(g, B, V, kind):
    x = (g.standard_normal((B, V), dtype=np.float32) * 3).astype(np.float32)
    if kind == "mostly -inf":
        x[:, : V - V // 8] = -np.inf
        x[0] = -np.inf
        x[0, V // 2] = 1.5
    elif kind == "nan":
        x[:, ::5] = np.nan
    elif kind == "ascending":
        x.sort(axis=1)
    return x


def _check(x, got, top_n, rows):
    for r in rows:
        lse, _, ids, tlp = orc.logprobs(x[r], -1, min(top_n, x.shape[1]))
        assert abs(got["lse"][r] - lse) <= TOL, (r, got["lse"][r], lse)
        n = len(ids)
        assert np.array_equal(got["top_id"][r, :n], ids), (r, got["top_id"][r, :n], ids)
        assert np.allclose(got["top_logprob"][r, :n], tlp, rtol=0, atol=TOL)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,V,top_n", [(1, 131072, 20), (2, 131071, 20), (2, 131073, 256), (5, 2049, 8), (11, 100003, 64), (11, 100003, 65), (739, 4097, 5), (741, 2048, 3), (900, 6001, 20)])
def test_cut_rows(bf16, B, V, top_n):
    import arcinfer_b200 as ab

    g = np.random.default_rng(V + top_n)
    x = _rows(g, B, V, "normal")
    if bf16:
        x = synth.bf16_bits_to_f32(synth.f32_to_bf16_bits(x))
    lg = torch.from_numpy(x).cuda()
    out = ab.logprobs_batch(lg.bfloat16() if bf16 else lg, None, top_n)
    got = {k: v.cpu().numpy() for k, v in out.items()}
    assert got["status"][0] == 0
    _check(x, got, top_n, range(0, B, max(1, B // 40)))


@pytest.mark.parametrize("kind", ["mostly -inf", "nan", "ascending"])
@pytest.mark.parametrize("V,top_n", [(50000, 20), (9000, 256)])
def test_odd_rows(kind, V, top_n):
    import arcinfer_b200 as ab

    x = _rows(np.random.default_rng(5), 4, V, kind)
    out = ab.logprobs_batch(torch.from_numpy(x).cuda(), None, top_n)
    got = {k: v.cpu().numpy() for k, v in out.items()}
    if kind == "nan":  # (the oracle is not defined on NaN: they are skipped)
        x = np.where(np.isnan(x), -np.inf, x).astype(np.float32)
        top_n = min(top_n, 200)
        got["top_id"], got["top_logprob"] = got["top_id"][:, :top_n], got["top_logprob"][:, :top_n]
    _check(x, got, top_n, range(1, 4))
    lse, _, ids, _ = orc.logprobs(x[0], -1, 1)
    assert abs(got["lse"][0] - lse) <= TOL and got["top_id"][0, 0] == ids[0]


def test_without_workspace():
    """444 rows or more, or rows of at most 8192 columns, are served without a workspace"""
    import arcinfer_b200 as ab

    for B, V in ((500, 20000), (3, 8000)):
        x = _rows(np.random.default_rng(B), B, V, "normal")
        lg = torch.from_numpy(x).cuda()
        want = ab.logprobs_batch(lg, None, 4)
        got = {"lse": torch.zeros(B, dtype=torch.float64, device="cuda"), "top_id": torch.zeros(B, 4, dtype=torch.int32, device="cuda"),
               "top_logprob": torch.zeros(B, 4, dtype=torch.float64, device="cuda")}
        a = ab.capi.LogprobArgs()
        a.logits, a.dtype, a.B, a.V, a.row_stride, a.top_n, a.top_stride = lg.data_ptr(), 0, B, V, V, 4, 4
        a.lse, a.top_id, a.top_logprob = (got[k].data_ptr() for k in ("lse", "top_id", "top_logprob"))
        assert ab.lib.arcs_logprobs_batch(C.byref(a), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert torch.equal(got["top_id"], want["top_id"]) and torch.allclose(got["lse"], want["lse"], rtol=0, atol=TOL)
    a.B, a.V, a.row_stride = 3, 8193, 8193
    assert ab.lib.arcs_logprobs_batch(C.byref(a), None) != 0


@pytest.mark.parametrize("off", [0, 4])
def test_rows_that_are_not_cut_leave_the_workspace_alone(off):
    """whatever it holds and wherever it begins: such calls may share one, and overlap"""
    import arcinfer_b200 as ab

    g = torch.Generator(device="cuda").manual_seed(5)
    for B, V in ((444, 20000), (1500, 9000), (3, 8192)):
        lg = torch.from_numpy(_rows(np.random.default_rng(B), B, V, "normal")).cuda()
        want = ab.logprobs_batch(lg, None, 4)
        ws = torch.randint(0, 256, (1 << 24,), dtype=torch.uint8, device="cuda", generator=g)
        kept = ws.clone()
        got = {"lse": torch.zeros(B, dtype=torch.float64, device="cuda"), "top_id": torch.zeros(B, 4, dtype=torch.int32, device="cuda"),
               "top_logprob": torch.zeros(B, 4, dtype=torch.float64, device="cuda")}
        a = ab.capi.LogprobArgs()
        a.logits, a.dtype, a.B, a.V, a.row_stride, a.top_n, a.top_stride = lg.data_ptr(), 0, B, V, V, 4, 4
        a.lse, a.top_id, a.top_logprob = (got[k].data_ptr() for k in ("lse", "top_id", "top_logprob"))
        a.workspace, a.workspace_bytes = ws.data_ptr() + off, ws.numel() - off
        assert ab.lib.arcs_logprobs_batch(C.byref(a), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert torch.equal(got["top_id"], want["top_id"]) and torch.equal(got["lse"], want["lse"]) and torch.equal(ws, kept)
        assert ab.lib.arcs_logprobs_workspace_bytes(B, V, 256) == 16
