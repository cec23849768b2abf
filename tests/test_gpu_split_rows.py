"""Rows split over several CTAs give what one CTA per row gives, for every kind of bound the slices keep their elements by, on
slices of one tile and of several, call after call on one handle (the slices' tickets start over by themselves)."""
import pytest

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
    import torch
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
