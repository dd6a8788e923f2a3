"""The prepare step of attention with shaped scores four channels at a time, against the same channel by channel (rows that begin one number further on,
which no vector load fits)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 255, 256, 300])
@pytest.mark.parametrize("H,G,M,D,E,rot,norm,temp", [(4, 2, 2, 64, 64, 64, True, 0.0), (16, 2, 2, 64, 128, 16, False, 0.1), (2, 1, 1, 4, 4, 0, True, 0.0),
                                                     (3, 3, 1, 256, 12, 256, True, 0.2), (1, 1, 2, 20, 8, 8, False, 0.0)])
def test_four_channels_at_a_time(H, G, M, D, E, rot, norm, temp, T, dtype):
    """An element is the same few operations either way: 4 roundings of 32 bits of it and its partner, the norm's sum of up to 4,096 squares in another order
    (2^-20), and in bfloat16 one rounding (2^-8) more."""
    from forge_b200 import kernels
    g = torch.Generator().manual_seed(H * D + T)
    cols = (H + G) * M * D + G * E
    rows = torch.randn(T, cols, generator=g).to(DEV)
    shifted = torch.zeros(T, cols + 5, device=DEV)
    shifted[:, 1:cols + 1] = rows
    pos = torch.randint(0, 3000, (T,), generator=g).int().to(DEV)
    slots = torch.randperm(T + 7, generator=g)[:T].int().to(DEV)
    slots[-1] = -1
    freq = (torch.rand(rot // 2, generator=g) ** 3).to(DEV) if rot else None
    qn, kn = ((1 + 0.2 * torch.randn(n, generator=g)).to(DEV) if norm else None for n in (H * M * D, G * M * D))
    out = []
    for proj, col in ((rows, 0), (shifted, 1)):
        cache = torch.zeros(-(-(T + 7) // 16), 16 * G * (M * D + E), device=DEV, dtype=dtype)
        q = kernels.scored_prepare(proj, pos, slots, cache, H, G, M, D, E, 16, dtype, inv_freq=freq, q_norm=qn, k_norm=kn, eps=1e-5, temp_coef=temp,
                                   temp_every=100.0 if temp else 0.0, col=col)
        out.append((q.float(), cache.float()))
    bound = 2.0 ** -19 if dtype == torch.float32 else 2.0 ** -7
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= bound * float(b.abs().max())
    assert torch.equal(out[0][1] != 0, out[1][1] != 0)
