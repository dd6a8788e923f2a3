"""Single tokens of retention with the state's packs in shared memory: up to 4, 8 and 16 packs a thread (the last one's 64 KB), one pack less and a row
of threads that has none, held as the step of the other sizes is."""
from types import SimpleNamespace

import pytest
import torch

import test_chunk_scans_gpu as scans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,V,rot", [(2, 64, 128, 64), (2, 128, 64, 32), (1, 128, 128, 128), (1, 127, 128, 0), (3, 65, 64, 2), (1, 40, 100, 8)])
def test_packs_of_a_thread(N, K, V, rot):
    scans.test_one_token_of_every_request_in_one_retention_kernel(torch.float32, N, K, V, rot)


@pytest.mark.parametrize("K,V", [(64, 64), (64, 128), (128, 128), (33, 100)])
def test_registers_and_shared_memory_give_the_same_bits(K, V):
    """Steps of a few and of many requests, on both sides of where the state's packs wait in registers: a request's numbers are the same in each."""
    from forge_b200 import kernels
    N, most = 4, 120
    g = torch.Generator().manual_seed(K + V)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    p, state0 = torch.randn(most, N * (2 * K + 2 * V), generator=g).cuda(), torch.randn(most, -(-N * K * V // 4) * 4, generator=g).cuda()
    decay, weight, freq = torch.rand(N, generator=g).cuda(), torch.randn(V, generator=g).cuda(), torch.rand(K // 4, generator=g).cuda()

    def step(B):
        batch = SimpleNamespace(num_requests=B, num_tokens=B, q_start=i32(list(range(B + 1))), slots=i32(list(range(B))), positions=i32([7 * i for i in range(B)]))
        state = state0.clone()
        cols = [0, N * K, 2 * N * K, N * (2 * K + V)]
        return kernels.retention_token(*[(p[:B].contiguous(), c) for c in cols], batch, freq, 0.1, decay, state, N, K, V, weight, 1e-4, torch.float32), state

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    out, state = step(most)                                   # 480 CTAs: shared memory, whatever the heads
    for B in (1, sms // N, sms // N + 1, 2 * sms // N, 2 * sms // N + 1, 3 * sms // N, 3 * sms // N + 1):
        o, st = step(B)
        assert torch.equal(o, out[:B]) and torch.equal(st[:B], state[:B]) and torch.equal(st[B:], state0[B:]), B
