"""The work that a user of this sampler has it do, as measurable cases: one dict per case, inputs made on the GPU from a
seed, one pass through the public Python entry points, and the same result in 64 bits by plain torch.

Logits are a language model's head output as the benchmark configurations describe it: N(0, 2^2) with eight spikes
U(8, 15) per row; histories are Zipf(1.1) token ids, the most frequent ids lowest; masks allow 2 % of the vocabulary, half
of it in four contiguous runs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mako_b200 import BatchSampler, SamplingParams, _lib
from mako_b200.sampler import Sampler, pack_params

DEV = "cuda"

# What every case of a batch of rows says; a case overrides what it needs.
_ROWS = {"kind": "sample", "batch": 1, "vocab": 129280, "packed": False, "temperature": 0.8, "top_k": 0, "top_p": 1.0,
         "min_p": 0.0, "repetition": 1.0, "presence": 0.0, "frequency": 0.0, "history": 0, "ragged_history": False,
         "mask": False, "bias": 0, "mixed": False}
_PENALTIES = {"repetition": 1.1, "presence": 0.5, "frequency": 0.3}


def _case(name, **kw):
    c = dict(_ROWS, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a request's own sampler object, one token at a time: sample() and a draft's verify(), results on the host
        _case("request_object", kind="request", vocab=151552, temperature=0.7, top_k=40, top_p=0.95, history=256),
        # one sequence being decoded, chat defaults with a top_k
        _case("decode_1_top_k", vocab=151552, temperature=0.7, top_k=40, top_p=0.95),
        # a few sequences under top_p alone, the default of chat APIs
        _case("decode_4_top_p", batch=4, top_p=0.9),
        # a server's decode step with penalties over long histories
        _case("penalised_256", batch=256, top_p=0.9, min_p=0.05, history=4096, **_PENALTIES),
        # grammar-constrained decoding: allowed-token masks and a sparse bias, pure draw
        _case("constrained_128", batch=128, vocab=151552, temperature=1.0, mask=True, bias=64),
        # a server's step over requests that all have parameters of their own, greedy ones among them
        _case("mixed_requests_128", batch=128, vocab=151552, mixed=True, history=1024, ragged_history=True),
        # a vocabulary that is no multiple of four, rows packed tightly, histories of different lengths
        _case("packed_rows_256", batch=256, vocab=50257, packed=True, top_k=50, top_p=0.95, history=1024, ragged_history=True,
              repetition=1.1),
        # a large offline batch, top_p alone after penalties
        _case("offline_1024_top_p", batch=1024, vocab=151552, top_p=0.9, history=4096, **_PENALTIES),
        # speculative decoding with one draft a sequence: accept or redraw, penalties over the sequences' histories
        _case("verify_192", kind="verify", batch=192, top_p=0.9, min_p=0.05, history=1024, ragged_history=True, **_PENALTIES),
        # speculative decoding against a drafter's distribution, 64 sequences of five positions
        _case("draft_vs_target_320", kind="pq", batch=320, temperature=0.6, top_p=0.95),
        # one rank of eight of a vocabulary-parallel head: its shard's records, and the merge of all ranks' records
        _case("vocab_shard_1024", kind="shard", batch=1024, vocab=151552, shards=8, keys=64, top_p=0.9, history=4096,
              **_PENALTIES),
        # the drafter's Markov head, one step for eight sequences
        _case("drafter_pick_8", kind="pick", batch=8, rank=256, dim=1024),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample"] * 6 + ["request", "verify", "pq", "shard", "pick"])
    vocab = _between(rng, 32000, 163840)
    c = _case(None, kind=kind, vocab=vocab, packed=rng.random() < 0.3, temperature=round(rng.uniform(0.4, 1.2), 2))
    how = rng.choice(["top_k", "top_p", "min_p", "both", "plain", "greedy"])
    if how in ("top_k", "both"):
        c["top_k"] = _between(rng, 2, 200)
    if how in ("top_p", "both", "min_p"):
        c["top_p"] = round(rng.uniform(0.5, 0.98), 2)
    if how == "min_p":
        c["min_p"] = round(rng.uniform(0.01, 0.2), 3)
    if how == "plain":  # a pure draw goes with a grammar
        c["mask"] = True
    if how == "greedy":
        c["temperature"] = 0.0
    if rng.random() < 0.5:
        c["history"] = _between(rng, 16, 4096)
        c["ragged_history"] = rng.random() < 0.5
        c.update(repetition=round(rng.uniform(1.0, 1.3), 2), presence=round(rng.uniform(0, 1), 2),
                 frequency=round(rng.uniform(0, 0.5), 2))
    if kind in ("sample", "verify") and rng.random() < 0.25:
        c["bias"] = _between(rng, 4, 128)
    c["batch"] = _between(rng, 1, max(1, min(1024, 64_000_000 // vocab)))
    if kind == "sample" and rng.random() < 0.15:
        c.update(mixed=True, history=_between(rng, 16, 2048), ragged_history=True)
    if kind == "request":
        c.update(batch=1, history=min(c["history"], 512), ragged_history=False, mask=False, packed=False)
        if how == "plain":
            c["top_k"] = 50
    if kind == "verify":
        c.update(mask=False, batch=min(c["batch"], 256), min_p=0.03 if how == "plain" else c["min_p"])
    if kind == "pq":
        c.update(batch=max(1, c["batch"] // 2), mask=False, history=0, temperature=max(c["temperature"], 0.4))
        if how in ("plain", "greedy"):
            c["top_p"] = 0.95
    if kind == "shard":
        c.update(shards=rng.choice([2, 4, 8]), keys=64, mask=False, packed=False, temperature=max(c["temperature"], 0.4))
        if how == "plain":
            c["top_k"] = 40
        c["ragged_history"] = False
    if kind == "pick":
        c.update(batch=rng.randint(1, 8), rank=rng.choice([64, 128, 256]), dim=_between(rng, 256, 4096), packed=False)
    return c


# ---- inputs -----------------------------------------------------------------------------------------------------------

def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _logits(c, seed, rows, salt=1):
    """[rows, vocab], the rows 16-byte aligned unless the case packs them tightly; and the spikes' columns."""
    v = c["vocab"]
    ld = v if c["packed"] else (v + 3) // 4 * 4
    g = _gen(seed, salt)
    x = torch.randn(rows, ld, generator=g, device=DEV)
    x *= 2.0
    x = x[:, :v]
    spikes = torch.randint(0, v, (rows, 8), generator=g, device=DEV)
    x.scatter_(1, spikes, torch.rand(rows, 8, generator=g, device=DEV) * 7.0 + 8.0)
    return x, spikes


def _history(c, seed, rows):
    if not c["history"]:
        return None, None
    g = _gen(seed, 2)
    w = torch.arange(1, c["vocab"] + 1, device=DEV, dtype=torch.float64).pow(-1.1).cumsum(0)
    at = torch.rand(rows, c["history"], generator=g, device=DEV, dtype=torch.float64) * w[-1]
    hist = torch.searchsorted(w, at).clamp_(max=c["vocab"] - 1).to(torch.int32)
    n = None
    if c["ragged_history"]:
        n = torch.randint(0, c["history"] + 1, (rows,), generator=g, device=DEV).to(torch.int32)
    return hist, n


def _mask(c, seed, rows, spikes):
    if not c["mask"]:
        return None
    v, g = c["vocab"], _gen(seed, 3)
    ok = torch.rand(rows, v, generator=g, device=DEV) < 0.01
    run = max(1, v // 400)
    col = torch.arange(v, device=DEV)
    for _ in range(4):
        at = torch.randint(0, v - run, (rows, 1), generator=g, device=DEV)
        ok |= (col >= at) & (col < at + run)
    ok.scatter_(1, spikes, torch.rand(rows, 8, generator=g, device=DEV) < 0.5)
    words = ((v + 31) // 32 + 3) // 4 * 4
    bits = torch.zeros(rows, words * 32, dtype=torch.int64, device=DEV)
    bits[:, :v] = ok
    packed = (bits.view(rows, words, 32) << torch.arange(32, device=DEV)).sum(2)
    return torch.where(packed >= 1 << 31, packed - (1 << 32), packed).to(torch.int32)


def _bias(c, seed, rows):
    if not c["bias"]:
        return None
    g = _gen(seed, 4)
    step = c["vocab"] // c["bias"]  # one id from each of as many ranges: distinct within a row
    ids = torch.arange(c["bias"], device=DEV) * step + torch.randint(0, step, (rows, c["bias"]), generator=g, device=DEV)
    vals = torch.rand(rows, c["bias"], generator=g, device=DEV) * 10.0 - 5.0
    return torch.stack([ids.to(torch.int32), vals.view(torch.int32)], dim=2).contiguous()


def _params(c):
    return SamplingParams(temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"], min_p=c["min_p"],
                          presence_penalty=c["presence"], frequency_penalty=c["frequency"],
                          repetition_penalty=c["repetition"])


def _row_params(c, seed, rows):
    """One SamplingParams a row: the case's own, or a server's mixture."""
    if not c["mixed"]:
        return [_params(c)] * rows
    rng, out = np.random.RandomState(int(seed) & 0x7FFFFFFF), []
    for _ in range(rows):
        p = SamplingParams(temperature=float(np.float32(rng.uniform(0.5, 1.0))))
        how = rng.randint(5)
        if how == 0:
            p.temperature = 0.0
        if how in (1, 2):
            p.top_p = float(np.float32(rng.uniform(0.8, 0.95)))
        if how in (2, 3):
            p.top_k = int(rng.randint(20, 61))
        if how == 4:
            p.min_p = float(np.float32(rng.uniform(0.02, 0.1)))
        if rng.rand() < 0.5:
            p.repetition_penalty, p.frequency_penalty = 1.1, 0.2
        out.append(p)
    return out


def _inputs(c, seed):
    kind, rows = c["kind"], c["batch"]
    d = {}
    d["logits"], spikes = _logits(c, seed, rows)
    d["history"], d["history_len"] = _history(c, seed, rows)
    d["mask"] = _mask(c, seed, rows, spikes)
    d["bias"] = _bias(c, seed, rows)
    g = _gen(seed, 5)
    d["u"], d["u2"], d["u3"] = (torch.rand(rows, generator=g, device=DEV) for _ in range(3))
    if kind in ("verify", "request"):  # half of the drafts are likely tokens
        other = torch.randint(0, c["vocab"], (rows,), generator=g, device=DEV)
        likely = torch.rand(rows, generator=g, device=DEV) < 0.5
        d["draft"] = torch.where(likely, d["logits"].argmax(1), other).to(torch.int32)
    if kind == "pq":
        d["draft_logits"] = d["logits"] + torch.randn(rows, c["vocab"], generator=_gen(seed, 6), device=DEV)
    return d


def _shard_width(c):
    return ((c["vocab"] + c["shards"] - 1) // c["shards"] + 3) // 4 * 4


def prepare(case, seed):
    c = dict(case)
    kind, batch, vocab = c["kind"], c["batch"], c["vocab"]
    s = {"case": c}
    if kind == "pick":
        g = _gen(seed, 7)
        n = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
        s.update(logits=_logits(c, seed, batch)[0], head=n(vocab, c["rank"]) * 0.1, embed=n(vocab, c["rank"]), x=n(batch, c["dim"]),
                 w=n(c["dim"] + c["rank"]) * 0.02,
                 prev=torch.randint(0, vocab, (batch,), generator=g, device=DEV).to(torch.int32), sampler=BatchSampler(vocab, batch))
        return s
    d = _inputs(c, seed)
    s.update(d)
    if kind == "request":
        s["sampler"] = Sampler(_params(c), vocab, int(seed) & 0xFFFFFFFF)
        for t in (d["history"][0].tolist() if c["history"] else []):
            s["sampler"].accept(t)
        s["row"], s["draft"] = d["logits"][0], int(d["draft"][0])
        return s
    s["params"] = _params(c)
    if kind == "shard":
        w, k = _shard_width(c), c["keys"]
        s["sampler"] = BatchSampler(w, batch)
        s["merger"] = BatchSampler(vocab, 1 if batch == 1 else batch)
        record = _lib.lib.mk_vp_record_bytes(k)
        s["gathered"] = torch.zeros(c["shards"], batch, record, dtype=torch.uint8, device=DEV)
        mine = c["shards"] // 2
        for r in range(c["shards"]):  # what the other ranks send
            part = d["logits"][:, r * w: min(vocab, (r + 1) * w)]
            s["sampler"].vp_local(part.contiguous(), s["params"], k, s["gathered"][r], id_offset=r * w, history=d["history"])
        s["offset"] = mine * w
        s["part"] = d["logits"][:, mine * w: min(vocab, (mine + 1) * w)].contiguous()
        s["record"] = s["gathered"][mine]
        del s["logits"]
        return s
    if c["mixed"]:
        s["params"] = torch.from_numpy(pack_params(_row_params(c, seed, batch))).to(DEV)
    s["sampler"] = BatchSampler(vocab, d["logits"].shape[0])
    s["side"] = {k: d[k] for k in ("history", "history_len", "mask", "bias")}
    return s


def _result(r, **more):
    return {"token": r.token, "prob": r.prob, "flags": r.flags, "n_cand": r.n_cand, **more}


def run(s):
    c = s["case"]
    kind, sampler = c["kind"], s["sampler"]
    if kind == "sample":
        return _result(sampler.sample(s["logits"], s["params"], s["u"], **s["side"]))
    if kind == "request":
        token = sampler.sample(s["row"])
        verified, accepted = sampler.verify(s["row"], s["draft"])
        return {"token": token, "verified": verified, "accepted": accepted}
    if kind == "verify":
        r = sampler.verify(s["logits"], s["params"], s["draft"], s["u"], s["u2"], **s["side"])
        return _result(r, accepted=r.accepted)
    if kind == "pq":
        r = sampler.verify_pq(s["logits"], s["draft_logits"], s["params"], s["u"], s["u2"], s["u3"])
        return {"token": r.token, "draft_token": r.draft_token, "accepted": r.accepted, "flags": r.flags}
    if kind == "shard":
        sampler.vp_local(s["part"], s["params"], c["keys"], s["record"], id_offset=s["offset"], history=s["history"])
        r = s["merger"].vp_merge(s["gathered"], c["shards"], c["batch"], c["keys"], c["vocab"], s["params"], s["u"])
        rec = s["record"]
        lists = rec[:, 16:].view(torch.int32).view(c["batch"], c["keys"], 2)
        return _result(r, row_max=rec[:, 0:4].view(torch.float32), row_sum=rec[:, 8:16].view(torch.float64),
                       best=lists[:, :, 0].view(torch.float32), best_ids=lists[:, :, 1])
    draft, conf = sampler.draft_pick(s["logits"], s["head"], s["embed"], s["x"], s["w"], s["prev"])
    return {"draft": draft, "conf": conf}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def work(case):
    c = case
    v, b = c["vocab"], c["batch"]
    if c["kind"] == "pick":
        return {"bytes": 4 * v * c["rank"] + 4 * b * (v + c["dim"] + 2 * c["rank"] + 3), "flops": 2 * b * v * c["rank"]}
    rows = b
    cols = min(_shard_width(c), v - c["shards"] // 2 * _shard_width(c)) if c["kind"] == "shard" else v
    side = rows * (4 * ((v + 31) // 32) if c["mask"] else 0) + 8 * rows * c["bias"]
    side += 4 * b * c["history"] // (2 if c["ragged_history"] else 1) + 4 * rows * 5
    if c["mixed"]:
        side += 28 * rows
    passes = 2 if c["kind"] in ("pq", "request") else 1
    if c["kind"] == "shard":
        side += rows * (16 + 8 * c["keys"]) * (c["shards"] + 1)
    # an exponential, a comparison and an addition a column
    return {"bytes": passes * 4 * rows * cols + side, "flops": 3 * passes * rows * cols}


def tolerance(case):
    """Tokens follow the reference's own float arithmetic and are equal to the bit wherever a decision does not lie within
    the margin of an approximate sum (rows a flag names: under 1 % of the rows of a top_p draw). Probabilities are a
    quotient of two floats; a row whose nucleus is one token longer differs by that token's weight."""
    if case["kind"] in ("request", "pq"):
        return {"rel": 0.0, "max": 0.0, "differ": 0.01}
    if case["kind"] == "pick":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------

def _weights(l, p, hist):
    """Penalties, temperature, min_p, top_k, top_p of one row in 64 bits: (weight, column) in draw order."""
    if p.temperature <= 0.0:
        best = l.argmax().view(1)
        return torch.ones(1, dtype=torch.float64, device=DEV), best
    if hist is not None and hist.numel():
        ids, n = hist.long().unique(return_counts=True)
        x = l[ids]
        if p.repetition_penalty != 1.0:
            x = torch.where(x > 0, x / p.repetition_penalty, x * p.repetition_penalty)
        l[ids] = x - (p.presence_penalty + p.frequency_penalty * n.double())
    q = ((l - l.max()) / p.temperature).exp()
    ids = torch.nonzero((q >= min(p.min_p, 1.0)) & (q > 0)).view(-1)
    q = q[ids]
    if (0 < p.top_k < q.numel()) or p.top_p < 1.0:
        q, order = q.sort(descending=True, stable=True)
        ids = ids[order]
        if 0 < p.top_k < q.numel():
            q, ids = q[: p.top_k], ids[: p.top_k]
        if p.top_p < 1.0:
            run = q.cumsum(0)
            n = int((run < p.top_p * run[-1]).sum()) + 1
            q, ids = q[:n], ids[:n]
    return q, ids


def _drawn(q, u):
    run = q.cumsum(0)
    return min(int((run <= u * run[-1]).sum()), q.numel() - 1)


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    if kind in ("request", "pq"):
        return None
    if kind == "pick":
        s = prepare(c, seed)
        xe = torch.cat([s["x"].double(), s["embed"][s["prev"].long()].double()], 1)
        return {"draft": None, "conf": torch.sigmoid(xe @ s["w"].double())}
    d = _inputs(c, seed)
    params = _row_params(c, seed, c["batch"])
    if kind == "shard":
        w, p, out = _shard_width(c), params[0], {}
        lo = c["shards"] // 2 * w
        row_max, row_sum, best = [], [], []
        for b in range(c["batch"]):
            l = d["logits"][b].double()
            if d["history"] is not None and p.temperature > 0:
                ids, n = d["history"][b].long().unique(return_counts=True)
                x = l[ids]
                if c["repetition"] != 1.0:
                    x = torch.where(x > 0, x / c["repetition"], x * c["repetition"])
                l[ids] = x - (c["presence"] + c["frequency"] * n.double())
            l = l[lo: lo + w]
            row_max.append(l.max())
            row_sum.append(((l - l.max()) / c["temperature"]).exp().sum())
            best.append(l.topk(c["keys"])[0])
        out = {k: None for k in ("token", "prob", "flags", "n_cand", "best_ids")}
        return dict(out, row_max=torch.stack(row_max).view(-1, 1), row_sum=torch.stack(row_sum).view(-1, 1), best=torch.stack(best))
    prob = []
    for row in range(c["batch"]):
        l = d["logits"][row].double()
        if d["bias"] is not None:
            l[d["bias"][row, :, 0].long()] += d["bias"][row, :, 1].contiguous().view(torch.float32).double()
        hist = None
        if d["history"] is not None:
            hist = d["history"][row]
            if d["history_len"] is not None:
                hist = hist[: int(d["history_len"][row])]
        if d["mask"] is not None:
            bit = (d["mask"][row].view(-1, 1) >> torch.arange(32, device=DEV)) & 1
            off = bit.reshape(-1)[: c["vocab"]] == 0
            l[off] = -math.inf
        q, ids = _weights(l, params[row], hist)
        u = float(d["u"][row])
        if kind == "verify":
            at = torch.nonzero(ids == int(d["draft"][row])).view(-1)
            if at.numel() and (params[row].temperature <= 0 or u * q.sum() < q[at[0]]):
                prob.append(q[at[0]] / q.sum())
                continue
            if at.numel() and q.numel() > 1:
                q = q[torch.arange(q.numel(), device=DEV) != at[0]]
            u = float(d["u2"][row])
        prob.append(q[_drawn(q, u)] / q.sum())
    return {"prob": torch.stack(prob), **{k: None for k in ("token", "flags", "n_cand") + (("accepted",) if kind == "verify" else ())}}
