"""The gated delta rule's preparation: the kernel of four channels a lane against the one of a channel a lane (which takes rows that do not begin on 16 bytes),
bit for bit, over portions that begin, end and are cut anywhere in a warp's run of tokens, behind rings that are full and that are not."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("reqs", [[(0, 1), (5, 2), (0, 3), (1, 4), (2, 17), (100, 40), (0, 5)], [(0, 700)], [(3, 1), (64, 1), (0, 1)]])
@pytest.mark.parametrize("N,M,V,taps", [(4, 2, 64, 4), (3, 3, 128, 3), (8, 1, 32, 2), (2, 1, 192, 4), (32, 16, 64, 4)])
def test_both_kernels(reqs, N, M, V, taps):
    from forge_b200 import kernels
    K = 64
    C = 2 * M * K + N * V
    g = torch.Generator().manual_seed(N + V)
    starts = [0]
    for _, n in reqs:
        starts.append(starts[-1] + n)
    T, S = starts[-1], len(reqs)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(num_requests=S, num_tokens=T, q_start=i32(starts), slots=i32(list(range(S))[::-1]), tok_req=i32([s for s, (_, n) in enumerate(reqs) for _ in range(n)]),
                            positions=i32([c + j for c, n in reqs for j in range(n)]))
    width = (C + 2 * N + 3) // 4 * 4
    p = torch.randn(T, width, generator=g).to(DEV)
    conv = torch.randn(taps, C, generator=g).to(DEV)
    rate, dt = torch.rand(N, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    state0 = torch.randn(S, (N * K * V + taps * C + 3) // 4 * 4, generator=g).to(DEV)
    got = []
    for col in (0, 1):
        rows = torch.full((T, width + 4 * col), 7.0, device=DEV)
        rows[:, col:col + width] = p
        state = state0.clone()
        got.append(kernels.gated_delta_prepare(rows, col, col + C, col + C + N, conv, rate, dt, batch, state, N, M, K, V) + (state,))
    for a, b in zip(*got):
        assert bool(torch.isfinite(a).all()) and torch.equal(a, b)


def test_the_filter_may_come_from_the_kernel_ahead():
    """The filter is looked up in a table, another one each time into the same buffer, by a kernel launched right before the preparation: none of the
    buffer's old numbers may enter."""
    from forge_b200 import kernels
    N, M, K, V, taps, T = 64, 32, 64, 64, 4, 40
    C = 2 * M * K + N * V
    g = torch.Generator().manual_seed(5)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(num_requests=1, num_tokens=T, q_start=i32([0, T]), slots=i32([0]), tok_req=i32([0] * T), positions=i32(list(range(T))))
    p = torch.randn(T, C + 2 * N, generator=g).to(DEV)
    rate, dt = torch.rand(N, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV)
    state = torch.zeros(1, N * K * V + taps * C, device=DEV)
    tables = [torch.randn(1024, C, generator=g).to(DEV) for _ in range(3)]
    ids = torch.arange(1023, -1, -1, dtype=torch.int32, device=DEV)
    prepare = lambda conv: kernels.gated_delta_prepare(p, 0, C, C + N, conv, rate, dt, batch, state, N, M, K, V)[0]
    wants = [prepare(t.flip(0)[-taps:].contiguous()) for t in tables]
    torch.cuda.synchronize()
    got = []
    for i in range(12):
        rows = kernels.embedding(ids, tables[i % 3])
        got.append(prepare(rows[-taps:]))                     # (the rows that the kernel ahead writes last)
        del rows                                              # its buffer is the next round's
    for i, y in enumerate(got):
        assert torch.equal(y, wants[i % 3]), i


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("col", [0, 1])
def test_a_number_that_is_none_reaches_as_far_as_the_filter(taps, col):
    """A NaN among the inputs of one token reaches that token and the taps - 1 tokens behind it, in both kernels, wherever it lies in a warp's run."""
    from forge_b200 import kernels
    N, M, K, V, T = 2, 1, 64, 64, 40
    C = 2 * M * K + N * V
    g = torch.Generator().manual_seed(taps)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(num_requests=1, num_tokens=T, q_start=i32([0, T]), slots=i32([0]), tok_req=i32([0] * T), positions=i32(list(range(T))))
    rate, dt, conv = torch.rand(N, generator=g).to(DEV), torch.randn(N, generator=g).to(DEV), torch.randn(taps, C, generator=g).to(DEV)
    for at in (0, 5, 14, 15, 16, 39):
        p = torch.randn(T, C + 2 * N + 4 * col, generator=g)
        p[at, col:col + C] = float("nan")
        state = torch.zeros(1, (N * K * V + taps * C + 3) // 4 * 4, device=DEV)
        qkv = kernels.gated_delta_prepare(p.to(DEV), col, col + C, col + C + N, conv, rate, dt, batch, state, N, M, K, V)[0].cpu()
        none = torch.zeros(T, dtype=torch.bool)
        none[at:at + taps] = True
        assert bool(torch.isnan(qkv[none]).all()) and bool(torch.isfinite(qkv[~none]).all()), at
