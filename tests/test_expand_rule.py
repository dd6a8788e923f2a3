"""Which steps spell the keys and values of a latent attention out (kernels.latent_expand_pays), without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from forge_b200 import kernels

# (cached, new) of the step's requests, width of a head, and whether spelling out was the faster form where both were measured (None: not near the line)
STEPS = [([(0, 1600)], 128, True), ([(700, 512), (0, 1024)], 128, True), ([(1000, 24)], 128, True), ([(0, 400)], 64, True), ([(1000, 100)], 64, True),
         ([(4000, 8)], 128, True), ([(4000, 1)] * 40 + [(0, 24)], 128, False), ([(2000, 1)] * 64 + [(0, 8)], 64, False),
         ([(0, 1), (0, 1)], 128, False), ([(30000, 40000)], 128, False)]


@pytest.mark.parametrize("reqs,D,pays", STEPS)
def test_which_steps(monkeypatch, reqs, D, pays):
    monkeypatch.setattr(kernels, "_sm_count", lambda device: 148)
    starts = [0]
    for _, n in reqs:
        starts.append(starts[-1] + n)
    batch = SimpleNamespace(num_requests=len(reqs), num_tokens=starts[-1], host_q_start=starts, host_context_before=[c for c, _ in reqs], attention_plan={},
                            positions=torch.empty(0))
    assert kernels.latent_expand_pays(batch, 32, D, D // 2, D, 4 * D) is pays
    assert kernels.latent_expand_pays(batch, 32, D, D // 2, D, 4 * D) is pays            # ... as asked once more in the same step
    batch.decode_only, batch.attention_plan = True, {}
    assert kernels.latent_expand_pays(batch, 32, D, D // 2, D, 4 * D) is False           # a step that a graph replays never does


def test_requests_that_bring_nothing_have_nothing_before():
    """A batch that was not laid out by the engine: an empty request has no first token to look at, at the end, in the middle or before another's."""
    batch = SimpleNamespace(num_requests=4, num_tokens=5, host_q_start=[0, 2, 2, 5, 5], positions=torch.tensor([7, 8, 30, 31, 32], dtype=torch.int32), attention_plan={})
    assert kernels._tokens_before(batch) == [7, 0, 30, 0] == batch.host_context_before
    assert kernels._tokens_before(SimpleNamespace(num_requests=2, host_q_start=[0, 0, 1], positions=torch.tensor([4], dtype=torch.int32))) == [0, 4]
    # the tiles of a step with such requests: (first token, tokens, request, first position), furthest first
    assert kernels.shaped_plan(batch, 2, torch.device("cpu")).tolist() == [[4, 1, 2, 32], [2, 2, 2, 30], [0, 2, 0, 7]]
