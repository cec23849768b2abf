"""Rows that start at any four-byte boundary (packed vocabularies, views into a wider buffer): the kernels take them from the
16-byte boundary before, so every edit, mask bit and id has to move with them. Whatever stands in front of a row must
not matter, least of all a larger value or a NaN."""
import numpy as np
import pytest

from helpers import Inputs, oracle_sample_rows
from mako_b200.sampler import SamplingParams

pytestmark = pytest.mark.gpu

PARAMS = {
    "greedy": SamplingParams(temperature=0.0),
    "min_p": SamplingParams(temperature=0.8, top_p=0.9, min_p=0.05, repetition_penalty=1.1, frequency_penalty=0.3),
    "top_k": SamplingParams(temperature=0.7, top_k=40, top_p=0.95),
    "top_p": SamplingParams(temperature=1.0, top_p=0.9, repetition_penalty=1.1),
    "plain": SamplingParams(temperature=1.0),
}


@pytest.mark.parametrize("v", [1, 29, 4093, 8195, 50257])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("masked", [False, True])
def test_rows_at_every_offset(gpu_sampler_factory, ref, v, offset, masked):
    import torch
    batch, cap = 4, 64
    inp = Inputs(31 + v + offset, batch, v, n_history=min(v, 300), with_mask=masked, n_bias=min(v, 8), n_spikes=min(v, 2),
                 mask_fraction=0.5)
    g = inp.to_gpu()
    wide = torch.full((batch * (v + 8) + 8,), float("nan"), device="cuda")
    logits = wide[offset:].as_strided((batch, v), (v + 5, 1))  # rows 5 mod 4 apart: every row on another boundary
    for b in range(batch):  # what stands between the rows would win if it were read
        wide[offset + b * (v + 5) + v: offset + (b + 1) * (v + 5)] = float("nan") if b % 2 else 1e30
    logits.copy_(g["logits"])
    s = gpu_sampler_factory(v, batch, cap)
    for name, p in PARAMS.items():
        res = s.sample(logits, p, g["u"], **g["kw"])
        torch.cuda.synchronize()
        for b, w in enumerate(oracle_sample_rows(ref, p, inp, cap=cap)):
            f = res.flags[b].item()
            assert not f & 0x50, name
            if f & 0x2:
                continue
            k = min(w["n_cand"], cap)
            assert (res.token[b].item(), res.n_cand[b].item()) == (w["token"], w["n_cand"]), (name, b)
            assert np.array_equal(res.cand_ids[b, :k].cpu().numpy(), w["cand_ids"][:k]), (name, b)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_a_row_without_a_maximum(gpu_sampler_factory, offset):
    """A NaN in the first column, and a row of nothing but -inf: the first column is returned."""
    import torch
    v = 5003
    wide = torch.randn(2 * v + 8, device="cuda")
    logits = wide[offset: offset + 2 * v].view(2, v)
    logits[0, 0] = float("nan")
    logits[1] = float("-inf")
    res = gpu_sampler_factory(v, 4, 64).sample(logits, SamplingParams(temperature=1.0, top_p=0.9), torch.full((2,), 0.5, device="cuda"))
    torch.cuda.synchronize()
    assert res.token.tolist() == [0, 0] and all(f & 0x4 for f in res.flags.tolist())
