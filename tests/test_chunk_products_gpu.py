"""The gated delta rule's chunks with their products on the tensor cores: more requests than the walk sorts by length, equal and empty ones among
them, and a number that is none, which reaches no token before its own.

Against the recurrence in 64 bits token by token; fp32 sums over up to 64 channels and a chunk's 32 tokens: 1e-5 of the largest number."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(lens, N, V, seed, poison=None):
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
