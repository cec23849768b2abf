"""Rows split over several CTAs give what one CTA per row gives, for every kind of bound the slices keep their elements by, on
slices of one tile and of several, call after call on one handle (the slices' tickets start over by themselves)."""
import pytest
import torch

from helpers import Inputs
from mako_b200.sampler import SamplingParams

pytestmark = pytest.mark.gpu

KINDS = {
    "greedy": SamplingParams(temperature=0.0),
    "top_k_40": SamplingParams(temperature=0.7, top_k=40, top_p=0.95),
    "top_k_200": SamplingParams(temperature=0.9, top_k=200),
    "top_k_above_a_slice": SamplingParams(temperature=0.9, top_k=9000, top_p=0.5),
    "min_p": SamplingParams(temperature=0.8, top_p=0.9, min_p=0.02, repetition_penalty=1.1, frequency_penalty=0.3),
    "top_p": SamplingParams(temperature=0.8, top_p=0.9, repetition_penalty=1.1),
    "plain": SamplingParams(temperature=1.0),
}


@pytest.mark.parametrize("batch", [1, 9, 40, 64])
@pytest.mark.parametrize("masked", [False, True])
def test_split_rows_equal_whole_rows(gpu_sampler_factory, batch, masked):
    v, cap = 100003, 64  # 25 tiles, rows on every alignment
    inp = Inputs(500 + batch, batch, v, n_history=700, n_bias=16, with_mask=masked)
    g = inp.to_gpu()
    g["logits"][batch - 1, 0] = float("nan")
    if batch > 1:
        g["logits"][0] = float("-inf")
    s = gpu_sampler_factory(v, 64, cap)
    drafts = g["logits"].nan_to_num(-1e30).argmax(1).to(torch.int32)
    for name, p in KINDS.items():
        got = []
        for on in (True, False, True):
            s.set_split(on)
            r = s.sample(g["logits"], p, g["u"], **g["kw"])
            n = r.n_cand.clone()
            keep = torch.arange(cap, device="cuda") < n[:, None]
            got.append([r.token.clone(), r.prob.clone(), r.flags.clone(), n, r.cand_ids * keep, r.cand_q * keep])
            w = s.verify(g["logits"], p, drafts, g["u2"], g["u3"], **g["kw"])
            got[-1] += [w.token.clone(), w.accepted.clone()]
        s.set_split(True)
        banded = (got[0][2] | got[1][2]) & 0x2  # a row total summed in another order may decide another way there
        for a, b, c in zip(*got):
            sure = (banded == 0).view(-1, *([1] * (a.dim() - 1))).expand_as(a)
            assert torch.equal(a[sure], b[sure]), name
            assert torch.equal(a, c), name


def _copies(r):
    """A result's values as they are now (its tensors are views of the handle's buffers, which the next call writes again)."""
    keep = None if r.cand_ids is None else torch.arange(r.cand_ids.shape[1], device="cuda") < r.n_cand[:, None]
    return [r.token.clone(), r.prob.clone(), r.n_cand.clone()] + ([] if keep is None else [r.cand_ids * keep, r.cand_q * keep])


def _same_where_sure(a, b, sure, what):
    for x, y in zip(a, b):
        at = sure.view(-1, *([1] * (x.dim() - 1))).expand_as(x)
        assert torch.equal(x[at], y[at]), what


@pytest.mark.parametrize("overlap", [1, 2])
def test_split_rows_behind_one_another(overlap):
    """Launches that follow one another programmatically share the handle's tickets and parts: 60 in a row, of other shapes in
    turn, each equal to whole rows in plain stream order."""
    from mako_b200 import BatchSampler
    v, cap = 100003, 64
    sets = [(Inputs(800 + b, b, v, n_history=300), b) for b in (1, 5, 48)]
    gs = [i.to_gpu() for i, _ in sets]
    whole, split = BatchSampler(v, 48, 0, cap), BatchSampler(v, 48, 0, cap)
    whole.set_split(False)
    split.set_overlap(overlap)
    for name in ("top_k_40", "min_p", "top_p"):
        want = []
        for g in gs:
            r = whole.sample(g["logits"], KINDS[name], g["u"], **g["kw"])
            want.append((_copies(r), r.flags.clone()))
        torch.cuda.synchronize()
        got = []
        for call in range(60):
            g = gs[call % 3]
            r = split.sample(g["logits"], KINDS[name], g["u"], **g["kw"])
            got.append((_copies(r), r.flags.clone()))
        torch.cuda.synchronize()
        for call, (g, f) in enumerate(got):
            w, wf = want[call % 3]
            _same_where_sure(g, w, ((f | wf) & 0x2) == 0, f"{name}, call {call}")


def test_split_rows_with_parameters_of_their_own(gpu_sampler_factory):
    from mako_b200.sampler import pack_params
    v, cap, batch = 100003, 64, 14
    inp = Inputs(860, batch, v, n_history=700, n_bias=16)
    g = inp.to_gpu()
    ps = list(KINDS.values())
    params = torch.from_numpy(pack_params([ps[b % len(ps)] for b in range(batch)])).cuda()
    s = gpu_sampler_factory(v, 64, cap)
    got = []
    for on in (True, False):
        s.set_split(on)
        r = s.sample(g["logits"], params, g["u"], **g["kw"])
        got.append((_copies(r), r.flags.clone()))
    s.set_split(True)
    _same_where_sure(got[0][0], got[1][0], ((got[0][1] | got[1][1]) & 0x2) == 0, "per-row parameters")


@pytest.mark.parametrize("batch", [1, 9, 32])
@pytest.mark.parametrize("kind", ["top_k_40", "top_p"])
def test_split_rows_of_both_distributions(gpu_sampler_factory, batch, kind):
    """p/q verification splits two row sets at a time, each with tickets of its own."""
    from mako_b200 import synth
    v = 130007  # 32 tiles
    inp = Inputs(870 + batch, batch, v)
    g = inp.to_gpu()
    lq = torch.from_numpy(synth.add_noise(870, inp.logits, v, sigma=1.0)).cuda()
    s = gpu_sampler_factory(v, 32, 0)
    got = []
    for on in (True, False, True):
        s.set_split(on)
        r = s.verify_pq(g["logits"], lq, KINDS[kind], g["u"], g["u2"], g["u3"])
        got.append(([r.draft_token.clone(), r.accepted.clone(), r.token.clone()], r.flags.clone()))
    s.set_split(True)
    sure = ((got[0][1] | got[1][1] | got[2][1]) & 0x2) == 0
    assert sure.any()
    _same_where_sure(got[0][0], got[1][0], sure, "split against whole")
    _same_where_sure(got[0][0], got[2][0], sure, "split again")


def test_a_new_handle_is_ready_on_any_stream(ref):
    """Created while the default stream is busy, on memory that was something else before, and used at once on a stream that does
    not wait for the default one: the first call's tickets are zero all the same."""
    from mako_b200 import BatchSampler
    from helpers import oracle_sample_rows
    v, batch, p = 151552, 4, KINDS["top_k_40"]
    inp = Inputs(880, batch, v)
    g = inp.to_gpu()
    want = [w["token"] for w in oracle_sample_rows(ref, p, inp)]
    junk = torch.full((1 << 28,), -1, dtype=torch.int32, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    torch.cuda._sleep(200_000_000)  # the default stream is busy for some 100 ms
    with torch.cuda.stream(side):
        s = BatchSampler(v, batch, 0)
        tok = s.sample(g["logits"], p, g["u"]).token.clone()
    side.synchronize()
    assert tok.tolist() == want
