"""The workloads whose time matters to a user of this library: one decoding step of each kind
through the public entry points, from one request on its own to a thousand rows at once.

A case is a dict of plain values; `kind` names the call:
  sample       SamplePlan.launch: a serving loop's step over device-resident logits
  mixed        sample_batch: rows of different users, each with settings and a bias list of its own
  host         HostContext.sample: logits in (pinned) host memory, tokens back in host memory
  verify       sample_batch + accept_batch: drafts verified under sampling
  constrained  dfa_mask + SamplePlan.launch: rows held to a byte automaton
  argmax       argmax_batch with slots: greedy verification of drafts
  confidence   argmax_batch with want_lse: the drafter's (max, sum exp)
  logprobs     logprobs_batch: a token's log probability (and the alternatives) of every row
  dflash       dflash_select: the candidate selector over slots x draft positions
"""
import numpy as np
import torch

import arcinfer_b200 as ab
from arcinfer_b200 import synth

DEV = "cuda"


def listed():
    return [
        # one request alone: the smallest step there is, with the sampler's default-like settings
        dict(name="single-row", kind="sample", B=1, V=151936, bf16=False, sigma=2.5, H=64, temperature=0.7, top_k=20, top_p=0.8, min_p=0.0,
             repeat_penalty=1.05, presence=0.0, frequency=0.0, last_n=64),
        # the same step for an application that keeps its logits in host memory (the drop-in for Sampler::sample)
        dict(name="host-row", kind="host", B=1, V=151936, bf16=False, sigma=2.5, H=64, temperature=0.7, top_k=20, top_p=0.8, min_p=0.0,
             repeat_penalty=1.05, presence=0.0, frequency=0.0, last_n=64),
        # a handful of slots decoding together, presence and frequency penalties over long histories
        dict(name="multi-slot", kind="sample", B=8, V=262144, bf16=False, sigma=3.0, H=256, temperature=1.0, top_k=64, top_p=0.95, min_p=0.05,
             repeat_penalty=1.0, presence=0.5, frequency=0.3, last_n=64),
        # a server's batch: every row has its own settings (greedy, few candidates, the 256 of top_k 0,
        # penalties that lower and that raise), its own history and bias list; an odd vocabulary, so
        # that rows start at any element; the candidate lists are asked for
        dict(name="mixed-rows", kind="mixed", B=48, V=128003, bf16=True, sigma=3.0, H=300),
        # drafts verified under sampling: 8 slots x (7 drafts + 1)
        dict(name="sampled-verify", kind="verify", slots=8, rows=8, V=151936, bf16=True, sigma=2.0, H=256, top_k=40),
        # the widest step: a thousand rows, long histories
        dict(name="wide-batch", kind="sample", B=1024, V=262144, bf16=True, sigma=3.0, H=512, temperature=1.0, top_k=50, top_p=0.95, min_p=0.0,
             repeat_penalty=1.1, presence=0.0, frequency=0.0, last_n=-1),
        # a schema or a tool call: the mask of every automaton state in use, then the rows under it
        dict(name="constrained", kind="constrained", B=32, V=151936, bf16=False, sigma=3.0, dfa_states=96, temperature=0.8, top_k=20, top_p=0.9),
        # greedy verification: 8 slots x (7 drafts + 1)
        dict(name="spec-verify", kind="argmax", slots=8, rows=8, V=151936, bf16=True, sigma=2.0),
        # the drafter's confidence of a few slots
        dict(name="draft-confidence", kind="confidence", B=8, V=151936, bf16=False, sigma=2.5),
        # the `logprobs` entry of every row of a wide batch, with the 20 alternatives served at most
        dict(name="logprobs", kind="logprobs", B=1024, V=262144, bf16=True, sigma=3.0, top_n=20),
        # scoring a text (perplexity): the target's log probability alone
        dict(name="scoring", kind="logprobs", B=512, V=151936, bf16=False, sigma=3.0, top_n=0),
        # a drafter's candidate selection: 8 slots x 7 positions
        dict(name="dflash", kind="dflash", slots=8, nd=7, V=151936, bf16=False, rank=256, topk=16, min_p=0.3),
    ]


_MOST = 1024 * 262144 * 2  # bytes of logits in the largest listed case


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    """One more case: any kind, rows over the logarithm of their range, vocabularies of any size
    (mostly not a multiple of anything), either type, the options that are used in earnest."""
    kind = rng.choice(["sample", "sample", "mixed", "host", "verify", "constrained", "argmax", "confidence", "logprobs", "logprobs", "dflash"])
    V = _log_int(rng, 30000, 262144)
    if rng.random() < 0.25:
        V = min(262144, -(-V // 128) * 128)  # a padded vocabulary
    bf16 = rng.random() < 0.5
    elt = 2 if bf16 else 4
    rows = lambda hi: min(_log_int(rng, 1, hi), max(1, _MOST // (V * elt)))  # noqa: E731
    c = dict(kind=kind, V=V, bf16=bf16)
    if kind in ("sample", "host"):
        pen = rng.choice(["repeat", "presence", "none"])
        c.update(B=rows(1024 if kind == "sample" else 16), sigma=round(rng.uniform(2.0, 3.5), 2), H=0 if pen == "none" else _log_int(rng, 16, 1024),
                 temperature=rng.choice([0.6, 0.7, 0.8, 1.0, 1.2]), top_k=rng.choice([20, 40, 50, 64]), top_p=rng.choice([0.8, 0.9, 0.95, 1.0]),
                 min_p=rng.choice([0.0, 0.0, 0.05]), repeat_penalty=rng.choice([1.05, 1.1]) if pen == "repeat" else 1.0,
                 presence=0.5 if pen == "presence" else 0.0, frequency=0.3 if pen == "presence" else 0.0, last_n=rng.choice([64, -1]))
    elif kind == "mixed":
        c.update(B=rows(256), sigma=round(rng.uniform(2.0, 3.5), 2), H=_log_int(rng, 16, 400))
    elif kind == "verify":
        c.update(slots=_log_int(rng, 1, 32), rows=rng.randint(2, 8), sigma=round(rng.uniform(2.0, 3.0), 2), H=_log_int(rng, 16, 1024), top_k=rng.choice([20, 40, 50]))
    elif kind == "constrained":
        c.update(B=rows(64), sigma=round(rng.uniform(2.0, 3.5), 2), dfa_states=_log_int(rng, 16, 256), temperature=rng.choice([0.7, 0.8, 1.0]),
                 top_k=rng.choice([20, 40]), top_p=rng.choice([0.9, 0.95]))
    elif kind == "argmax":
        c.update(slots=_log_int(rng, 1, 64), rows=rng.randint(2, 8), sigma=round(rng.uniform(2.0, 3.0), 2))
    elif kind == "confidence":
        c.update(B=rows(64), sigma=round(rng.uniform(2.0, 3.0), 2))
    elif kind == "logprobs":
        c.update(B=rows(1024), sigma=round(rng.uniform(2.0, 3.5), 2), top_n=rng.choice([0, 0, 1, 5, 20]))
    else:
        c.update(slots=_log_int(rng, 1, 16), nd=rng.randint(2, 7), rank=rng.choice([64, 128, 256]), topk=rng.choice([8, 16, 32]), min_p=rng.choice([0.0, 0.3]))
    return c


# ---------------------------------------------------------------- inputs
def _logits(gen, B, V, sigma, bf16):
    x = torch.empty(B, V, dtype=torch.bfloat16 if bf16 else torch.float32, device=DEV)
    step = max(1, (1 << 25) // V)
    for r0 in range(0, B, step):
        r1 = min(B, r0 + step)
        x[r0:r1] = torch.randn(r1 - r0, V, generator=gen, device=DEV) * sigma
    # a few tokens stand out in every row, as they do after a trained head
    at = torch.randint(0, V, (B, 8), generator=gen, device=DEV)
    x.scatter_add_(1, at, torch.full((B, 8), 2.0 * sigma, dtype=x.dtype, device=DEV))
    return x


def _history(gen, B, V, H):
    off = torch.arange(B + 1, device=DEV, dtype=torch.int32) * H
    return off, torch.randint(0, V, (B * H,), generator=gen, device=DEV, dtype=torch.int32)


def _settings(c, B):
    return synth.make_params(B, temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"], min_p=c["min_p"], presence_penalty=c["presence"],
                             frequency_penalty=c["frequency"], repeat_penalty=c["repeat_penalty"], repeat_last_n=c["last_n"])


def _mixed_settings(g, B):
    p = synth.make_params(B)
    for b in range(B):
        what = b % 6
        p["temperature"][b] = (0.0, 0.7, 1.0, 0.6, 1.2, 0.8)[what]
        p["top_k"][b] = (20, 20, 0, 64, 40, 100)[what]
        p["top_p"][b] = g.choice([0.8, 0.9, 0.95])
        p["min_p"][b] = (0.0, 0.0, 0.05, 0.0, 0.02, 0.0)[what]
        p["repeat_penalty"][b] = (1.0, 1.1, 1.0, 1.05, 1.0, 1.3)[what]
        p["repeat_last_n"][b] = (64, 64, -1, 256, -1, 64)[what]
        p["presence_penalty"][b] = (0.0, 0.0, 0.5, 0.0, -0.2, 0.0)[what]   # (negative: asked for by clients that want repetition)
        p["frequency_penalty"][b] = (0.0, 0.0, 0.3, 0.0, 0.0, 0.1)[what]
    return p


def prepare(case, seed):
    c = case
    kind, V, bf16 = c["kind"], c["V"], c["bf16"]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    g = np.random.default_rng(seed)
    s = {"kind": kind}
    if kind in ("sample", "host"):
        B, H = c["B"], c["H"]
        x = _logits(gen, B, V, c["sigma"], bf16)
        u = torch.rand(B, generator=gen, device=DEV, dtype=torch.float64)
        p = _settings(c, B)
        off, ids = _history(gen, B, V, H) if H else (None, None)
        if kind == "sample":
            s["plan"] = ab.capi.SamplePlan(x, ab.capi.params_to_device(p, DEV), u, hist_off=off, hist_ids=ids, max_hist=H)
        else:
            pin = lambda t: None if t is None else t.cpu().pin_memory()  # noqa: E731
            s["ctx"] = ab.capi.HostContext(0, B, V, bf16, max_hist_total=max(1, B * H))
            s["args"] = (pin(x), p, pin(u))
            s["out"] = {k: torch.zeros(B, dtype=torch.int32).pin_memory() for k in ("token", "n_cand", "n_kept")}
            s["lists"] = dict(hist_off=pin(off), hist_ids=pin(ids), max_hist=H) if H else {}
    elif kind == "mixed":
        B, H = c["B"], c["H"]
        hist = [g.integers(0, V, int(n)).astype(np.int32) for n in g.integers(0, H + 1, B)]
        bias = [g.choice(V, int(n), replace=False).astype(np.int32) for n in g.integers(0, 17, B)]
        ho, hi = synth.csr(hist)
        bo, bi = synth.csr(bias)
        bv = g.choice(np.array([-100.0, -3.0, 1.5, 4.0], np.float32), max(1, len(bi))).astype(np.float32)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a if len(a) else np.zeros(1, a.dtype))).to(DEV)  # noqa: E731
        s["args"] = (_logits(gen, B, V, c["sigma"], bf16), ab.capi.params_to_device(_mixed_settings(g, B), DEV), torch.rand(B, generator=gen, device=DEV, dtype=torch.float64))
        s["lists"] = dict(hist_off=dev(ho), hist_ids=dev(hi), max_hist=H, bias_off=dev(bo), bias_ids=dev(bi), bias_vals=dev(bv), max_bias=16)
    elif kind in ("verify", "argmax"):
        slots, rows = c["slots"], c["rows"]
        R = slots * rows
        x = _logits(gen, R, V, c["sigma"], bf16)
        best = x.argmax(dim=1).to(torch.int32).cpu().numpy().reshape(slots, rows)[:, : rows - 1]
        drafts = np.where(g.random((slots, rows - 1)) < 0.7, best, g.integers(0, V, (slots, rows - 1))).astype(np.int32)
        if kind == "argmax":
            s["args"] = (x,)
            s["lists"] = dict(row_off=torch.arange(slots + 1, device=DEV, dtype=torch.int32) * rows, draft=torch.from_numpy(drafts.reshape(-1).copy()).to(DEV),
                              draft_off=torch.arange(slots + 1, device=DEV, dtype=torch.int32) * (rows - 1))
        else:
            hist = [g.integers(0, V, c["H"]).astype(np.int32) for _ in range(slots)]
            ho, hi, ro, do, di = (torch.from_numpy(a).to(DEV) for a in ab.capi.verification_histories(hist, list(drafts)))
            p = synth.make_params(R, temperature=0.7, top_k=c["top_k"], top_p=0.9, repeat_penalty=1.05, repeat_last_n=64)
            s["args"] = (x, ab.capi.params_to_device(p, DEV), torch.rand(R, generator=gen, device=DEV, dtype=torch.float64))
            s["lists"] = dict(hist_off=ho, hist_ids=hi, max_hist=c["H"] + rows - 1)
            s["drafts"] = (ro, di, do)
    elif kind == "constrained":
        B = c["B"]
        off, by = synth.make_vocab(g, V)
        table, dead = synth.make_dfa(g, S=c["dfa_states"])
        S = c["dfa_states"]
        n = max(1, round(S * (1.0 - (1.0 - 1.0 / S) ** B)))  # (as many states in use as B rows at random have on average)
        states = np.sort(g.choice(S, n, replace=False))
        inv = g.integers(0, n, B)
        dev = lambda a: torch.from_numpy(a).to(DEV)  # noqa: E731
        mask = torch.zeros(n, (V + 31) // 32, dtype=torch.int32, device=DEV)
        x = _logits(gen, B, V, c["sigma"], bf16)
        p = synth.make_params(B, temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"])
        s["mask"] = mask
        s["dfa"] = (dev(table.view(np.int16)), dead, dev(states.astype(np.int32)), dev(off.view(np.int32)), dev(by))
        s["plan"] = ab.capi.SamplePlan(x, ab.capi.params_to_device(p, DEV), torch.rand(B, generator=gen, device=DEV, dtype=torch.float64), mask=mask,
                                       mask_row=dev(inv.astype(np.int32)))
    elif kind == "confidence":
        s["args"] = (_logits(gen, c["B"], V, c["sigma"], bf16),)
    elif kind == "logprobs":
        s["args"] = (_logits(gen, c["B"], V, c["sigma"], bf16), torch.randint(0, V, (c["B"],), generator=gen, device=DEV, dtype=torch.int32), c["top_n"])
    else:
        slots, nd, rank = c["slots"], c["nd"], c["rank"]
        x = _logits(gen, slots * nd, V, 2.0, bf16)
        # (the drafter is sure of most positions: one token well above the rest)
        x.scatter_(1, torch.randint(0, V, (slots * nd, 1), generator=gen, device=DEV), (torch.randn(slots * nd, 1, generator=gen, device=DEV) * 2.0 + 16.0).to(x.dtype))
        x = x.view(slots, nd, V)
        book = lambda: (torch.randn(V, rank, generator=gen, device=DEV) * 0.3).to(torch.bfloat16).view(torch.int16)  # noqa: E731
        s["args"] = (x, torch.randn(slots, nd, rank, generator=gen, device=DEV), book(), book(), torch.randint(0, V, (slots,), generator=gen, device=DEV, dtype=torch.int32))
        s["lists"] = dict(topk=c["topk"], max_drafts=nd, min_p=c["min_p"])
    return s


def run(state):
    s = state
    kind = s["kind"]
    if kind == "sample":
        return s["plan"].launch()
    if kind == "host":
        logits, params, u = s["args"]
        out = s["out"]
        s["ctx"].sample(logits, params, u, out["token"], n_cand=out["n_cand"], n_kept=out["n_kept"], **s["lists"])
        return out
    if kind == "mixed":
        return ab.sample_batch(*s["args"], want_cands=True, **s["lists"])
    if kind == "verify":
        out = ab.sample_batch(*s["args"], **s["lists"])
        accepted, following = ab.accept_batch(out["token"], *s["drafts"])
        return {**out, "accepted": accepted, "next": following}
    if kind == "constrained":
        ab.dfa_mask(*s["dfa"], out=s["mask"])
        return {**s["plan"].launch(), "mask": s["mask"]}
    if kind == "argmax":
        return ab.argmax_batch(*s["args"], **s["lists"])
    if kind == "confidence":
        return ab.argmax_batch(*s["args"], want_lse=True)
    if kind == "logprobs":
        return ab.logprobs_batch(*s["args"])
    return ab.dflash_select(*s["args"], **s["lists"])


def work(case):
    """Every logit, list entry and table once, the outputs once; one comparison a logit, and the
    exponential and its addition where the path sums them."""
    c = case
    kind, V = c["kind"], c["V"]
    elt = 2 if c["bf16"] else 4
    rows = c["B"] if "B" in c else c["slots"] * c["nd"] if kind == "dflash" else c["slots"] * c["rows"]
    by = rows * V * elt
    fl = rows * V
    if kind in ("sample", "host", "mixed", "verify"):
        by += rows * (32 + 8 + 16) + rows * c["H"] * 4 // (2 if kind == "mixed" else 1)
        if kind == "mixed":
            by += rows * 8 * 8 + rows * 256 * 12
    elif kind == "constrained":
        states = min(rows, c["dfa_states"])
        by += int(V * (2.85 + 4)) + c["dfa_states"] * 512 + 2 * states * V // 8 + rows * 56
    elif kind == "argmax":
        by += rows * 8
    elif kind == "confidence":
        by += rows * 12
        fl *= 3
    elif kind == "logprobs":
        by += rows * (20 + 12 * c["top_n"])
        fl *= 3
    else:
        by += rows * c["rank"] * (4 + 2 * (c["topk"] + 1))
        fl = fl * 3 + rows * c["topk"] * c["rank"] * 2
    return {"bytes": by, "flops": fl}


def tolerance(case):
    """Ids, counts, flags, masks and the tokens drawn are the same whatever the order of the work.
    Probabilities and sums are compared with their 64-bit values: `rel` is about four times the
    difference measured."""
    kind = case["kind"]
    if kind == "mixed":
        return {"rel": 1.5e-7, "max": 1e-6}     # probabilities of fp32 exponentials
    if kind == "confidence":
        return {"rel": 4e-7, "max": 1e-6}       # fp32 (max, sum exp)
    if kind == "logprobs":
        return {"rel": 4e-8, "max": 1e-7}       # fp32 exponentials summed in fp64, the logarithm of the sum
    if kind == "dflash":
        return {"rel": 3e-7, "max": 8e-7}       # path probabilities from such sums
    return "exact"


def exact(case, seed):
    """The computed numbers of `run` in 64 bits (log-sum-exps and what follows from them); the rest
    of the outputs are ids, counts and flags, or (mixed, dflash) depend on which ids were chosen."""
    kind = case["kind"]
    if kind not in ("confidence", "logprobs"):
        return None
    x, *rest = prepare(case, seed)["args"]
    top = torch.empty(x.shape[0], dtype=torch.float64, device=DEV)
    lse, z = torch.empty_like(top), torch.empty_like(top)
    for r in range(x.shape[0]):
        d = x[r].double()
        top[r] = d.max()
        z[r] = torch.exp(d - top[r]).sum()
        lse[r] = top[r] + torch.log(z[r])
    if kind == "confidence":
        return {"argmax": None, "max_sumexp": torch.stack([top, z], dim=1), "status": None}
    token, n = rest
    out = {"lse": lse, "status": None, "logprob": x.gather(1, token[:, None].long())[:, 0].double() - lse}
    if n > 0:
        best = torch.stack([torch.topk(x[r].float(), n).values for r in range(x.shape[0])])
        out.update(top_id=None, top_logprob=best.double() - lse[:, None])
    return out
