"""Rows of top_p alone whose nucleus runs to many tokens (flat_rows.cu): sizes at the edges of its groups, tables and
lists, rows on every alignment, weights that crowd one bucket, cuts from a sample that has nothing to say. Token ids,
candidate lists and weights against the reference, bit for bit, except in rows that report a guard band."""
import numpy as np
import pytest

from helpers import Inputs, oracle_sample_rows
from mako_b200.sampler import SamplingParams

pytestmark = pytest.mark.gpu

P = dict(repetition_penalty=1.1, presence_penalty=0.5, frequency_penalty=0.3)
CASES = {  # vocabulary, batch, parameters, inputs, what is done to the logits
    "ragged_small": (4099, 5, dict(temperature=1.0, top_p=0.9), dict(n_spikes=0), None),
    "smallest": (33, 3, dict(temperature=1.0, top_p=0.97), dict(n_spikes=0, sigma=0.3), None),
    "everything_edited": (20001, 6, dict(temperature=1.0, top_p=0.9, **P), dict(n_history=4000, n_bias=96, with_mask=True,
                                                                             mask_fraction=0.5, n_spikes=2), None),
    "aligned_history": (129280, 3, dict(temperature=0.8, top_p=0.95, **P), dict(n_history=4096, n_spikes=2), None),
    "history_too_long_for_the_tables": (32000, 4, dict(temperature=1.0, top_p=0.9, **P), dict(n_history=4096, n_bias=8, n_spikes=0), None),
    "longer_than_shared_memory": (151552, 3, dict(temperature=1.5, top_p=0.97), dict(n_spikes=0), None),
    "ties_of_sixteenths": (65536, 3, dict(temperature=1.0, top_p=0.9), dict(n_spikes=0), lambda x: np.round(x * 16) / 16),
    "ties_of_halves": (50257, 3, dict(temperature=1.0, top_p=0.9), dict(n_spikes=2), lambda x: np.round(x * 2) / 2),
    "all_equal": (10000, 2, dict(temperature=1.0, top_p=0.50005), dict(n_spikes=0), lambda x: np.zeros_like(x)),
    "low_top_p": (100003, 4, dict(temperature=1.5, top_p=0.3), dict(n_spikes=8), None),
    "sample_misses_the_heavy": (131072, 2, dict(temperature=1.0, top_p=0.5), dict(n_spikes=0),
                                lambda x: np.where((np.arange(x.shape[1]) % 512 >= 128) & (np.arange(x.shape[1]) % 1700 < 3), 7.0, x * 0.1)),
}


@pytest.mark.parametrize("name", CASES)
def test_flat_rows_equal_the_reference(gpu_sampler_factory, ref, name):
    import torch
    v, batch, p, kw, change = CASES[name]
    p, cap = SamplingParams(**p), 256
    inp = Inputs(7000 + len(name), batch, v, **kw)
    if change is not None:
        inp.logits = np.ascontiguousarray(change(inp.logits).astype(np.float32))
    s = gpu_sampler_factory(v, 8, cap)
    g = inp.to_gpu()
    res = s.sample(g["logits"], p, g["u"], **g["kw"])
    torch.cuda.synchronize()
    tok, n, flags = res.token.cpu().numpy(), res.n_cand.cpu().numpy(), res.flags.cpu().numpy()
    ids, qs = res.cand_ids.cpu().numpy(), res.cand_q.cpu().numpy()
    sure = 0
    for b, w in enumerate(oracle_sample_rows(ref, p, inp, cap=cap)):
        assert not flags[b] & 0x50
        if flags[b] & 0x2:
            continue
        sure += 1
        k = min(w["n_cand"], cap)
        assert (tok[b], n[b]) == (w["token"], w["n_cand"]), f"row {b}"
        assert np.array_equal(ids[b, :k], w["cand_ids"][:k])
        assert np.array_equal(qs[b, :k].view(np.uint32), w["cand_q"][:k].view(np.uint32))
    assert sure
    # the same rows as verification rows: drafts in the list and outside it
    draft = np.where(np.arange(batch) % 2 == 0, ids[:, 0], (tok + 1) % v).astype(np.int32)
    ver = s.verify(g["logits"], p, torch.from_numpy(draft).cuda(), g["u2"], g["u3"], **g["kw"])
    torch.cuda.synchronize()
    for b in range(batch):
        if not ver.flags[b].item() & 0x2:
            want = ref.verify(p, inp.logits[b], int(draft[b]), inp.u2[b], inp.u3[b], **inp.row_kwargs(b))
            assert (ver.token[b].item(), bool(ver.accepted[b].item())) == (want[0], bool(want[1])), f"row {b}"


def _flat_inputs(seed, batch, v, settled_every):
    """Rows of nuclei of some thousand tokens, with a peaked one (settled by the first launch) after every few of them."""
    inp = Inputs(seed, batch, v, n_spikes=0, sigma=0.4)
    if settled_every:
        inp.logits[::settled_every, 7] = 25.0
    return inp


@pytest.mark.parametrize("batch,settled_every", [(149, 0), (320, 3), (1025, 0), (2100, 5)])
def test_every_marked_row_is_taken_once(gpu_sampler_factory, ref, batch, settled_every):
    """More marked rows than CTAs, and more rows than a CTA looks at in one go: each is drawn, none twice, call after call."""
    import torch
    v, p = 4099, SamplingParams(temperature=1.0, top_p=0.9)
    inp = _flat_inputs(9000 + batch, batch, v, settled_every)
    g = inp.to_gpu()
    s = gpu_sampler_factory(v, batch, 16)
    want = oracle_sample_rows(ref, p, inp, cap=16)
    assert sum(w["n_cand"] > 1000 for w in want) >= batch // 2
    for call in range(3):
        s.token.fill_(-7)
        s.n_cand.zero_()
        res = s.sample(g["logits"], p, g["u"])
        torch.cuda.synchronize()
        tok, n, flags = res.token.cpu().numpy(), res.n_cand.cpu().numpy(), res.flags.cpu().numpy()
        ids, qs = res.cand_ids.cpu().numpy(), res.cand_q.cpu().numpy()
        assert (tok >= 0).all()
        for b, w in enumerate(want):
            if flags[b] & 0x2:
                continue
            k = min(w["n_cand"], 16)
            assert (tok[b], n[b]) == (w["token"], w["n_cand"]), f"call {call} row {b}"
            assert np.array_equal(ids[b, :k], w["cand_ids"][:k]), f"call {call} row {b}"
            assert np.array_equal(qs[b, :k].view(np.uint32), w["cand_q"][:k].view(np.uint32)), f"call {call} row {b}"


def test_two_sets_of_marked_rows_side_by_side(gpu_sampler_factory, ref):
    """p/q verification of flat rows: the drafter's and the target's marked rows are taken by two grids that compete for the
    device, so the later CTAs of one start when its first rows are done."""
    import torch
    from mako_b200 import synth
    v, batch, p = 4099, 320, SamplingParams(temperature=1.0, top_p=0.9)
    inp = _flat_inputs(9400, batch, v, 0)
    lq = synth.add_noise(9400, inp.logits, v, sigma=0.3)
    g, lq_dev = inp.to_gpu(), torch.from_numpy(lq).cuda()
    s = gpu_sampler_factory(v, batch, 16)
    want = [ref.verify_pq(p, inp.logits[b], lq[b], inp.u[b], inp.u2[b], inp.u3[b]) for b in range(batch)]
    for call in range(3):
        res = s.verify_pq(g["logits"], lq_dev, p, g["u"], g["u2"], g["u3"])
        torch.cuda.synchronize()
        d, acc, tok, flags = (t.cpu().numpy() for t in (res.draft_token, res.accepted, res.token, res.flags))
        assert not (flags & 0x50).any() and (tok >= 0).all()
        for b in range(batch):
            if not flags[b] & 0x2:
                assert (d[b], bool(acc[b]), tok[b]) == want[b], f"call {call} row {b}"
    assert 0 < sum(w[1] for w in want) < batch


def _top_p_beside(q, k, delta):
    """The float nearest to (mass of the k heaviest) * (1 + delta), and how far off that mass it is, relative to the total."""
    q = np.sort(q)[::-1]
    share = q[:k].sum() / q.sum()
    p = np.float32(share * (1.0 + delta))
    return float(p), abs(float(p) - share)


def test_the_first_launch_settles_what_its_margin_allows(gpu_sampler_factory, ref):
    """A dozen heavy tokens over a rest of 1.4 %: the row's total is the kept tokens' exact weights and an approximate rest, so a
    nucleus that ends a millionth of the total beside its bound is further off than the margin (1e-5 of the rest) and decided by the
    first launch: no flag, and no stamp of the flat rows' kernel."""
    import torch
    from mako_b200 import lib
    from mako_b200.sampler import pack_params
    v, batch, cap = 50000, 16, 32
    rng = np.random.default_rng(77)
    rows = rng.normal(0, 0.5, size=(batch, v)).astype(np.float32)
    ps = []
    for b in range(batch):
        cols = rng.choice(v, size=12, replace=False)
        rows[b, cols] = (14.0 - 0.35 * np.arange(12) + rng.uniform(0, 0.05, 12)).astype(np.float32)
        q = np.exp(rows[b].astype(np.float64) - float(rows[b].max()))
        top_p, off = _top_p_beside(q, 3 + b % 7, -1e-6 if b % 2 else 1e-6)
        rest = (q.sum() - np.sort(q)[::-1][:12].sum()) / q.sum()
        assert 2e-5 * rest < off < 1.5e-6 and rest < 0.02
        ps.append(SamplingParams(temperature=1.0, top_p=top_p))
    u = np.linspace(0.01, 0.99, batch).astype(np.float32)
    s = gpu_sampler_factory(v, batch, cap)
    stamps = torch.zeros((batch, 64), dtype=torch.int64, device="cuda")
    assert lib.mk_debug_set_timing(s._h, stamps.data_ptr()) == 0
    try:
        res = s.sample(torch.from_numpy(rows).cuda(), torch.from_numpy(pack_params(ps)).cuda(), torch.from_numpy(u).cuda())
        torch.cuda.synchronize()
    finally:
        lib.mk_debug_set_timing(s._h, None)
    assert not (res.flags.cpu().numpy() & 0x2).any()
    assert (stamps[:, 14] == 0).all() and (stamps[:, 3] != 0).all()
    for b in range(batch):
        w = ref.sample(ps[b], rows[b], u[b], cap=cap)
        assert (res.token[b].item(), res.n_cand[b].item()) == (w["token"], w["n_cand"]), f"row {b}"


def test_short_lists_are_decided_by_exact_weights(gpu_sampler_factory, ref):
    """Rows of 4000 columns and nuclei of hundreds: every column above the loose bound counts with its exact weight, so a nucleus that
    ends a few ten-millionths of the total beside its bound is decided without a guard band."""
    import torch
    from mako_b200.sampler import pack_params
    v, batch, cap = 4000, 24, 64
    rows = np.random.default_rng(78).normal(0, 1.0, size=(batch, v)).astype(np.float32)
    ps, n_close = [], 0
    for b in range(batch):
        q = np.exp(rows[b].astype(np.float64) - float(rows[b].max()))
        top_p, off = _top_p_beside(q, 300 + 61 * b, -2e-7 if b % 2 else 2e-7)
        n_close += 1e-8 < off < 5e-7
        ps.append(SamplingParams(temperature=1.0, top_p=top_p))
    assert n_close >= batch - 4
    u = np.linspace(0.01, 0.99, batch).astype(np.float32)
    s = gpu_sampler_factory(v, batch, cap)
    res = s.sample(torch.from_numpy(rows).cuda(), torch.from_numpy(pack_params(ps)).cuda(), torch.from_numpy(u).cuda())
    torch.cuda.synchronize()
    assert not (res.flags.cpu().numpy() & 0x2).any()
    for b in range(batch):
        w = ref.sample(ps[b], rows[b], u[b], cap=cap)
        assert (res.token[b].item(), res.n_cand[b].item()) == (w["token"], w["n_cand"]), f"row {b}"
        assert w["n_cand"] > 100


@pytest.mark.parametrize("kind", ["speculative round", "long history", "wide vocabulary"])
def test_rows_the_flat_kernel_does_not_take(gpu_sampler_factory, ref, kind):
    """Their second launch streams the row again, so the first one settles a nucleus of up to 24 tokens by itself: the count of
    collected elements that the general finish leaves in the stamps is then a few dozen at most, not a second launch's
    thousands. A row with a NaN and a flat one among them do take the second launch."""
    import torch
    from mako_b200 import lib
    v, batch, cap = (170000 if kind == "wide vocabulary" else 50000), 12, 64
    p = SamplingParams(temperature=1.0, top_p=0.88, frequency_penalty=0.01)
    rng = np.random.default_rng(79)
    rows = rng.normal(0, 0.5, size=(batch, v)).astype(np.float32)
    for b in range(batch - 1):
        rows[b, 10000 + rng.choice(v - 10000, size=26, replace=False)] = rng.uniform(13.4, 14.6, 26)
    rows[2, 17] = np.nan
    hist = np.zeros((batch, 4200 if kind == "long history" else 8), dtype=np.int32)  # (id 0, over and over)
    u = rng.uniform(0.01, 0.99, batch).astype(np.float32)
    s = gpu_sampler_factory(v, batch, cap)
    stamps = torch.zeros((batch, 64), dtype=torch.int64, device="cuda")
    lg, hist_dev = torch.from_numpy(rows).cuda(), torch.from_numpy(hist).cuda()
    assert lib.mk_debug_set_timing(s._h, stamps.data_ptr()) == 0
    try:
        if kind == "speculative round":  # rounds of a bonus row alone
            us = torch.from_numpy(np.stack([u, u], 1)).cuda()
            res = s.spec_round(lg, p, torch.zeros((batch, 0), dtype=torch.int32, device="cuda"), us, history=hist_dev)[2]
        else:
            res = s.sample(lg, p, torch.from_numpy(u).cuda(), history=hist_dev)
        torch.cuda.synchronize()
    finally:
        lib.mk_debug_set_timing(s._h, None)
    collected, flags = stamps[:, 9].tolist(), res.flags.cpu().numpy()
    n_within = 0
    for b in range(batch):
        w = ref.sample(p, rows[b], u[b], cap=cap, history=hist[b])
        assert not flags[b] & 0x52
        k = min(w["n_cand"], cap)
        assert (res.token[b].item(), res.n_cand[b].item()) == (w["token"], w["n_cand"]), f"row {b}"
        assert np.array_equal(res.cand_ids[b, :k].cpu().numpy(), w["cand_ids"][:k]), f"row {b}"
        if b in (2, batch - 1):
            assert collected[b] > 512
        elif w["n_cand"] <= 24:
            assert collected[b] <= 512, f"row {b}"
            n_within += w["n_cand"] > 20
    assert n_within >= 4


@pytest.mark.parametrize("v", [4096, 100000])
def test_a_min_p_that_is_no_number(gpu_sampler_factory, ref, v):
    """No weight is at least NaN: there is no candidate, whatever top_p would have kept, and the first maximum is returned."""
    import torch
    p, batch = SamplingParams(temperature=1.0, top_p=0.9, min_p=float("nan")), 3
    rows = np.zeros((batch, v), dtype=np.float32)  # (all equal: more than the one-warp finish looks at)
    rows[1] = np.random.default_rng(80).normal(0, 0.4, v)
    rows[2, 77] = 9.0
    u = np.full(batch, 0.7, dtype=np.float32)
    s = gpu_sampler_factory(v, batch, 16)
    for split in (True, False):
        s.set_split(split)
        res = s.sample(torch.from_numpy(rows).cuda(), p, torch.from_numpy(u).cuda())
        torch.cuda.synchronize()
        want = [ref.sample(p, rows[b], u[b], cap=16) for b in range(batch)]
        assert [w["token"] for w in want] == rows.argmax(1).tolist()
        assert res.token.tolist() == [w["token"] for w in want] and res.n_cand.tolist() == [1] * batch
        assert all(f & 0x4 for f in res.flags.tolist())
    s.set_split(True)
