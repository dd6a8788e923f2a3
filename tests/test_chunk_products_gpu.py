"""The gated delta rule's chunks with their products on the tensor cores: more requests than the walk sorts by length, equal and empty ones among
them, and a number that is none, which reaches no token before its own.

Against the recurrence in 64 bits token by token; fp32 sums over up to 64 channels and a chunk's 32 tokens: 1e-5 of the largest number."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(lens, N, V, seed, poison=None, in_state=None):
    from forge_b200 import kernels
    r = torch.Generator().manual_seed(seed)
    T, starts = sum(lens), [0]
    for n in lens:
        starts.append(starts[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(num_requests=len(lens), num_tokens=T, q_start=i32(starts), slots=i32(list(range(len(lens)))), positions=i32([j for n in lens for j in range(n)]))
    qkv = torch.randn(T, 2 * N * 64 + N * V, generator=r)
    qkv[:, :2 * N * 64] = torch.nn.functional.normalize(qkv[:, :2 * N * 64].view(T, 2 * N, 64), dim=2).view(T, -1)
    if poison is not None:
        qkv[poison, -1] = float("nan")
    g, beta = torch.exp(-0.1 * torch.rand(T, N, generator=r)), torch.rand(T, N, generator=r)
    state0 = torch.randn(len(lens), N * 64 * V, generator=r)
    if in_state is not None:
        state0[0, 5 * V + 3] = in_state
    state = state0.to(DEV)
    got = kernels.gated_delta_scan(qkv.to(DEV), g.to(DEV), beta.to(DEV), batch, state, N, N, 64, V, by_chunks=True)
    q, k = (qkv[:, i * N * 64:(i + 1) * N * 64].double().view(T, N, 64) for i in range(2))
    v, want, S_end = qkv[:, 2 * N * 64:].double().view(T, N, V), [], []
    for s, (lo, hi) in enumerate(zip(starts, starts[1:])):
        S = state0[s].double().view(N, 64, V)
        for t in range(lo, hi):
            S = g[t].double()[:, None, None] * S
            S = S + k[t][:, :, None] * (beta[t].double()[:, None] * (v[t] - torch.einsum("nkv,nk->nv", S, k[t])))[:, None, :]
            want.append(torch.einsum("nkv,nk->nv", S, q[t]).reshape(-1))
        S_end.append(S.reshape(-1))
    return got.double().cpu(), torch.stack(want), state.double().cpu(), torch.stack(S_end)


@pytest.mark.parametrize("lens", [[40] * 3 + [0, 40, 33], [32], list(range(1, 38)), [0] * 31 + [70]])
def test_requests_in_any_order(lens):
    got, want, state, S = _run(lens, 2, 64, len(lens))
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert float((state - S).abs().max()) <= 1e-5 * float(S.abs().max())


@pytest.mark.parametrize("at", [0, 17, 31, 45])
def test_a_number_that_is_none(at):
    got, want, state, S = _run([70], 2, 64, 3, poison=at)
    assert torch.equal(torch.isnan(got[:at]), torch.isnan(want[:at])) and not bool(torch.isnan(want[:at]).any())
    ok = ~torch.isnan(want)                                   # the channels beside it, and all tokens before it
    assert bool(torch.isnan(got[~ok]).all()) and float((got[ok] - want[ok]).abs().max()) <= 1e-5 * float(want[ok].abs().max())
    assert torch.equal(torch.isnan(state), torch.isnan(S))


def test_numbers_that_round_to_a_bfloat16_infinity():
    """A state near the largest fp32 number, above bfloat16's: outputs and state to 1e-5 of the largest number of the value channel that it is in (an fp32
    sum's error goes with its addends), and of all others of the rest."""
    got, want, state, S = _run([70], 2, 64, 4, in_state=3.398e38)
    assert bool(torch.isfinite(got).all()) and bool(torch.isfinite(state).all())
    got, want, state, S = got.view(70, 2, 64), want.view(70, 2, 64), state.view(2, 64, 64), S.view(2, 64, 64)
    for a, b in ((got, want), (state, S)):
        rest = torch.arange(64) != 3
        assert float((a[..., 3] - b[..., 3]).abs().max()) <= 1e-5 * float(b[..., 3].abs().max())
        assert float((a[..., rest] - b[..., rest]).abs().max()) <= 1e-5 * float(b[..., rest].abs().max())


@pytest.mark.parametrize("kind", ["retention", "lightning"])
@pytest.mark.parametrize("where", ["state", "key"])
def test_infinities_stay_infinities(kind, where):
    """Fixed decays: an infinity in the state or in one token's key gives what the recurrence gives token by token, infinities with their sign.  (In a value
    or a query it does not, by the form itself: q.k times an infinite value is infinite, where a row of the state has infinities of both signs to add.)"""
    from forge_b200 import kernels
    N, V, T = 2, 64, 70
    r = torch.Generator().manual_seed(8)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(num_requests=1, num_tokens=T, q_start=i32([0, T]), slots=i32([0]), positions=i32(list(range(T))))
    p, state0 = 0.3 * torch.randn(T, N * (128 + V), generator=r), torch.randn(1, N * 64 * V, generator=r)
    decay = torch.tensor([0.9, 1.0])
    if where == "state":
        state0[0, 5 * V + 3] = float("inf")
    else:
        p[37, N * 64 + 9] = float("inf")
    state, pd = state0.to(DEV), p.to(DEV)
    q, k, v = p[:, :N * 64].double().view(T, N, 64), p[:, N * 64:N * 128].double().view(T, N, 64), p[:, N * 128:].double().view(T, N, V)
    if kind == "lightning":
        got = kernels.lightning_scan(pd, 0, decay.to(DEV), batch, state, N, 64, V, by_chunks=True)
        q, k, v = (z * torch.sigmoid(z) for z in (q, k, v))
    else:
        got = kernels.retention_scan((pd, 0), (pd, N * 64), (pd, N * 128), batch, None, 0.125, decay.to(DEV), state, N, 64, V, by_chunks=True)
        k = k * 0.125
    S, want = state0[0].double().view(N, 64, V), []
    for t in range(T):
        S = decay.double()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        want.append((S * q[t][:, :, None]).sum(dim=1).reshape(-1))
    for a, b in ((got.double().cpu(), torch.stack(want)), (state.double().cpu().view(-1), S.reshape(-1))):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.isinf(a), torch.isinf(b))
        assert bool(torch.isinf(b).any())
        assert torch.equal(a[torch.isinf(b)], b[torch.isinf(b)])
        fine = torch.isfinite(b)
        assert float((a[fine] - b[fine]).abs().max()) <= 1e-5 * float(b[fine].abs().max())
