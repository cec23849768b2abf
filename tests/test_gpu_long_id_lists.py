"""More than 8192 candidates in ascending id (a pure draw whose mask allows that many): where in the vocabulary the allowed ids lie
changes neither the result nor, by much, the time."""
import numpy as np
import pytest

from helpers import Inputs, compare_sample, oracle_sample_rows
from mako_b200.sampler import SamplingParams

pytestmark = pytest.mark.gpu

V, ALLOWED, BATCH = 151552, 20000, 2


def _inputs(first):
    inp = Inputs(600, BATCH, V, with_mask=True)
    bits = np.zeros((BATCH, inp.mask.shape[1] * 32), dtype=np.uint8)
    bits[:, first:first + ALLOWED] = 1
    inp.mask = np.ascontiguousarray(np.packbits(bits, axis=1, bitorder="little").view(np.uint32))
    return inp


@pytest.mark.parametrize("first", [0, 1, 77777, V - ALLOWED])
def test_runs_of_allowed_ids_anywhere(gpu_sampler_factory, ref, first):
    import torch
    inp, p = _inputs(first), SamplingParams(temperature=1.0)
    inp.u[:] = (0.0, 0.999)
    g = inp.to_gpu()
    s = gpu_sampler_factory(V, BATCH, 64)
    want = oracle_sample_rows(ref, p, inp, cap=64)
    assert min(w["n_cand"] for w in want) > 8192
    compare_sample(s.sample(g["logits"], p, g["u"], **g["kw"]), want, cap=64)
    # drafts that are rejected: the first allowed id (whose weight heads the list), a likely one, one that is not allowed
    for draft in (first, int(np.argmax(inp.logits[0][first:first + ALLOWED])) + first, (first + ALLOWED) % V):
        d = torch.full((BATCH,), draft, dtype=torch.int32, device="cuda")
        r = s.verify(g["logits"], p, d, g["u3"], g["u2"], **g["kw"])
        torch.cuda.synchronize()
        for b in range(BATCH):
            wt, wa = ref.verify(p, inp.logits[b], draft, inp.u3[b], inp.u2[b], **inp.row_kwargs(b))
            assert (r.token[b].item(), bool(r.accepted[b].item())) == (wt, bool(wa)), (draft, b)


def test_high_ids_take_no_longer_than_low_ones(gpu_sampler_factory):
    import torch
    p, s, us = SamplingParams(temperature=1.0), gpu_sampler_factory(V, BATCH, 64), []
    for first in (0, V - ALLOWED):
        g = _inputs(first).to_gpu()
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            s.sample(g["logits"], p, g["u"], **g["kw"])
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        us.append(float(np.median(times)))
    assert us[1] < 2.0 * us[0] + 50.0, us
