"""Which steps spell the keys and values of a latent attention out (kernels.latent_expand_pays), without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from forge_b200 import kernels

# (cached, new) of the step's requests, width of a head, and what the rule says.  Spelling out was measured to be the faster form wherever it says so, and
# the slower one with 8 single tokens behind 4,000 and with 16 behind 1,000, of which the steps here have more; two single tokens are no portion, and
# 70,000 rows are more than the scratch may hold.
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


def test_a_step_stays_absorbed_where_its_scratch_does_not_fit(monkeypatch):
    """What the device has left decides where the open workspace has to grow; a step that fits into it asks nobody."""
    monkeypatch.setattr(kernels, "_sm_count", lambda device: 148)
    device, asked = torch.device("cuda", 0), []
    left = lambda n: monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d: asked.append(d) or (n, 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda d: 3 << 20)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda d: 1 << 20)
    ws = SimpleNamespace(hold=0, device=device, offset=20 << 20, back=0, capacity=30 << 20)
    monkeypatch.setattr(kernels, "_active_workspace", [ws])

    def pays(cached, tokens):
        batch = SimpleNamespace(num_requests=1, num_tokens=tokens, host_q_start=[0, tokens], host_context_before=[cached], attention_plan={},
                                positions=SimpleNamespace(device=device))
        return kernels.latent_expand_pays(batch, 32, 128, 64, 128, 512)

    need = 2 * (20100 * (32 * 256 + 576) + 100 * 32 * 192)
    grown = (need + ws.offset) * 9 // 8 - ws.capacity
    left(grown - (2 << 20))
    assert pays(20000, 100) and len(asked) == 1
    left(grown - (2 << 20) - 1)
    assert not pays(20000, 100)
    asked.clear()
    ws.capacity = ws.offset + need
    left(0)
    assert pays(20000, 100) and not asked                     # the workspace holds it
    ws.capacity = 0
    assert pays(1000, 100) and not asked                      # little enough not to ask
    assert pays(0, 8000) and not asked                        # the other form would take more
    monkeypatch.setattr(kernels, "_active_workspace", [None])
    assert not pays(20000, 100) and asked == [device]


def test_a_workspace_that_grows_gives_its_buffer_back_first(monkeypatch):
    ws = kernels.StepWorkspace("cpu")
    ws.reserve(1000)
    with ws.step():
        kernels.new_tensor((500,), torch.float32, ws.device)
        kernels.new_tensor((500,), torch.float32, ws.device)
        take, seen = torch.empty, []
        monkeypatch.setattr(torch, "empty", lambda *a, **k: seen.append((ws.buf, ws.typed)) or take(*a, **k))
    assert seen == [(None, {})] and ws.capacity >= 4000 and ws.canary_intact()
