"""What a call returns are views of the handle's output tensors as they are at that call: a caller that reshapes one, or gives the
handle other tensors to write to, gets what it asked for from the next call."""
import torch

from mako_b200.sampler import BatchSampler


def _handle(max_batch, cand_cap):
    s = BatchSampler.__new__(BatchSampler)  # (no device here: the outputs alone)
    s.max_batch, s.cand_cap = max_batch, cand_cap
    s.token, s.prob, s.flags, s.n_cand = (torch.arange(max_batch) + 10 * i for i in range(4))
    s.cand_ids = s.cand_q = torch.zeros((max_batch, cand_cap)) if cand_cap else None
    return s


def test_every_call_has_views_of_its_own():
    for b in (4, 3):
        s = _handle(4, 2)
        first, second = s._result(b), s._result(b)
        first.token.unsqueeze_(0)
        assert second.token.shape == s._result(b).token.shape == (b,)
        assert first.token.data_ptr() == second.token.data_ptr() == s.token.data_ptr()
        assert second.cand_ids.shape == (b, 2) and s.token.shape == (4,)


def test_outputs_may_be_replaced():
    for b in (4, 3):
        s = _handle(4, 0)
        s._result(b)
        s.token = torch.full((6,), -5)
        assert s._result(b).token.tolist() == [-5] * b and s._result(b).cand_ids is None
