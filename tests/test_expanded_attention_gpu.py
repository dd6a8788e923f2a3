"""Latent attention with keys and values spelled out per head (kernels.latent_expand, kernels.expanded_attention), against the definition in 64 bits.
Portions shorter and longer than a tile of 128 tokens, behind cached tokens, pages shorter and longer than a tile of keys, shared key channels that do not
fill a block of 64, keys and values of different widths; numbers that are none behind a request's last token.

The attention's inputs are bfloat16 and enter exactly; allowed as for the other prompt attentions: 2^-8 of a value and 1e-3 of the largest.  The queries'
rounding moves a number by 2^-9 of itself, their rotation by a few 2^-24 of the pair: 2^-8 of a value and 1e-6 of the pair are allowed."""
import math
from types import SimpleNamespace

import pytest
import torch

from test_attention_shaped_gpu import DEV, _batch, _close, _fill, _softmax_out, _visible

pytestmark = pytest.mark.gpu
REQS = [(0, 1), (70, 37), (0, 130), (200, 5), (0, 257)]          # (cached, new) of the step's requests


@pytest.mark.parametrize("H,C,D,R,E,ps,halves,col", [(4, 512, 128, 64, 128, 64, False, 0), (3, 256, 64, 32, 64, 16, True, 3), (2, 64, 64, 16, 192, 8, False, 4),
                                                     (1, 128, 128, 128, 64, 128, True, 0), (5, 64, 192, 48, 256, 64, False, 1)])
def test_expanded(H, C, D, R, E, ps, halves, col):
    from forge_b200 import kernels
    assert kernels.library("attention_shaped").forge_expanded_sm100_supports.fn(H, D, R, E)
    KD = C + R
    batch, table, n_pages, g = _batch(REQS, ps, KD, seed=H + C)
    cache = torch.empty(n_pages, ps * KD, dtype=torch.bfloat16)
    rows = _fill(cache.view(n_pages, ps, KD), table, REQS, ps, g)
    T, W = batch.num_tokens, D + R
    p = torch.randn(T, col + H * W + 2, generator=g)
    freq = 10000.0 ** (-2.0 * torch.arange(R // 2) / R)
    sink = torch.randn(H, generator=g) if halves else None
    scale, group = 2.0 * W ** -0.5, SimpleNamespace(block_table=table.to(DEV))
    qr, c, kr, row_start = kernels.latent_expand((p.to(DEV), col), cache.to(DEV), group, batch, H, C, D, R, ps, freq.to(DEV), 1.5, halves)
    # rows, packed request behind request, bit for bit
    want = torch.cat(rows)
    assert row_start.tolist() == [sum(a + b for a, b in REQS[:s]) for s in range(len(REQS))]
    assert torch.equal(c.double().cpu(), want[:, :C]) and torch.equal(kr.double().cpu(), want[:, C:])
    # queries
    q = p[:, col:col + H * W].double().view(T, H, W)
    # (the angle is a product in 32 bits, as everywhere in the engine)
    a = (batch.positions.cpu().float()[:, None] * freq.float()).double()[:, None, :]
    cs, sn = torch.cos(a) * 1.5, torch.sin(a) * 1.5
    u, v = (q[..., D:D + R // 2], q[..., D + R // 2:]) if halves else (q[..., D::2], q[..., D + 1::2])
    turned = torch.cat([u * cs - v * sn, v * cs + u * sn], -1) if halves else torch.stack([u * cs - v * sn, v * cs + u * sn], -1).flatten(-2)
    ref = torch.cat([q[..., :D], turned], -1)
    got = qr.double().cpu().view(T, H, W)
    pair = 1.5 * (u.abs() + v.abs())
    pair = torch.cat([pair, pair], -1) if halves else torch.stack([pair, pair], -1).flatten(-2)
    assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6 * torch.cat([torch.zeros_like(q[..., :D]), pair], -1)).all())
    # attention, over keys and values of any values
    kv = torch.randn(len(want), H * (D + E), generator=g).to(torch.bfloat16)
    wide = torch.full((T, H * E + 6), 3.0, dtype=torch.bfloat16, device=DEV)
    for out in (None, (wide, 2)):
        launches = kernels.launch_count()
        res = kernels.expanded_attention(qr, kv.to(DEV), kr, row_start, batch, H, D, R, E, scale, sink=None if sink is None else sink.to(DEV), out=out)
        assert kernels.launch_count() - launches == 1
        kernels.check_kernel_status(DEV)
        o = (res if out is None else wide[:, 2:2 + H * E]).double().cpu().view(T, H, E)
        at = base = 0
        for c0, n in REQS:
            ok, _ = _visible(c0, n, 0, 0)
            seen = slice(base, base + c0 + n)
            for h in range(H):
                k = torch.cat([kv[seen, h * (D + E):h * (D + E) + D].double(), kr[seen].double().cpu()], -1)
                s = (got[at:at + n, h] @ k.t() * scale).masked_fill(~ok, -math.inf)
                _close(o[at:at + n, h], _softmax_out(s, kv[seen, h * (D + E) + D:(h + 1) * (D + E)].double(), None if sink is None else sink[h].double()))
            at, base = at + n, base + c0 + n
    assert bool((wide[:, :2] == 3.0).all()) and bool((wide[:, 2 + H * E:] == 3.0).all())


def test_rows_behind_a_request_are_never_seen():
    """A request's last tile of keys reaches into the rows of the next one: numbers that are none there change nothing."""
    from forge_b200 import kernels
    H, D, R, E, reqs = 2, 64, 32, 64, [(0, 70), (0, 70)]
    batch, _, _, g = _batch(reqs, 64, 64, seed=1)
    q = torch.randn(140, H * (D + R), generator=g).to(torch.bfloat16).to(DEV)
    kv, kr = torch.randn(140, H * (D + E), generator=g).to(torch.bfloat16).to(DEV), torch.randn(140, R, generator=g).to(torch.bfloat16).to(DEV)
    starts = torch.tensor([0, 70], dtype=torch.int32, device=DEV)
    whole = kernels.expanded_attention(q, kv, kr, starts, batch, H, D, R, E, 0.1)[:70].clone()
    kv[70:] = float("nan")
    kr[70:] = float("nan")
    assert torch.equal(kernels.expanded_attention(q, kv, kr, starts, batch, H, D, R, E, 0.1)[:70], whole)


def test_positions_may_come_from_the_kernel_ahead():
    """The tokens' positions are written by a kernel launched right before, other ones each time into the same buffer: none of the old ones may enter."""
    from forge_b200 import kernels
    H, C, D, R, ps, T = 2, 64, 64, 32, 64, 64
    batch, table, n_pages, g = _batch([(0, T)], ps, C + R, seed=2)
    cache, group = torch.zeros(n_pages, ps * (C + R), dtype=torch.bfloat16, device=DEV), SimpleNamespace(block_table=table.to(DEV))
    q, freq = torch.randn(T, H * (D + R), generator=g).to(DEV), (10000.0 ** (-2.0 * torch.arange(R // 2) / R)).to(DEV)
    places = [torch.randint(0, 20000, (T,), generator=g) for _ in range(3)]
    rows = [torch.nn.functional.one_hot(p, 20000).float().to(DEV) for p in places]

    def expand(positions):
        batch.positions = positions
        return kernels.latent_expand(q, cache, group, batch, H, C, D, R, ps, freq)[0]

    wants = [expand(p.to(torch.int32).to(DEV)) for p in places]
    torch.cuda.synchronize()
    got = []
    for i in range(12):
        got.append(expand(kernels.argmax(rows[i % 3])))
        batch.positions = None                                # its buffer is the next round's
    for i, y in enumerate(got):
        assert torch.equal(y, wants[i % 3]), i


@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_a_value_that_is_none_reaches_no_token_before_its_own(bad):
    """Values of one channel in the middle of a tile of 128 tokens, at its edges and at the end: the tokens before them keep their results, those from
    there on have none in that channel, and all else is as it was bit for bit."""
    from forge_b200 import kernels
    H, D, R, E, reqs = 3, 64, 32, 128, [(90, 300), (0, 40)]
    batch, _, _, g = _batch(reqs, 64, 64, seed=3)
    q = torch.randn(340, H * (D + R), generator=g).to(torch.bfloat16)
    kv, kr = torch.randn(430, H * (D + E), generator=g).to(torch.bfloat16), torch.randn(430, R, generator=g).to(torch.bfloat16)
    starts = torch.tensor([0, 390], dtype=torch.int32, device=DEV)
    run = lambda kv: kernels.expanded_attention(q.to(DEV), kv.to(DEV), kr.to(DEV), starts, batch, H, D, R, E, 0.1).double().cpu().view(340, H, E)
    whole = run(kv)
    spots = [(90 + 17, 0, 5), (90 + 127, 1, 40), (90 + 128, 1, 100), (90 + 299, 2, 127), (390 + 39, 0, 64)]          # (row, head, channel)
    for row, h, e in spots:
        kv[row, h * (D + E) + D + e] = bad
    got = run(kv)
    kernels.check_kernel_status(DEV)
    want, again = whole.clone(), torch.zeros(340, H, E, dtype=torch.bool)
    for row, h, e in spots:
        t = row - 90 if row < 390 else 300 + row - 390
        end = 300 if row < 390 else 340
        want[t:end, h, e] = math.nan
        first = t - t % 128 if row < 390 else 300
        again[first:t, h, e // 32 * 32:e // 32 * 32 + 32] = True          # (added up anew: the same number but for the sums' order)
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    fine = torch.isfinite(want)
    assert torch.equal(got[fine & ~again], want[fine & ~again])
    # (two roundings of sums that differ by some 2^-16 of the weights' two terms: neighbouring bfloat16 numbers at most, 2^-7 of the smaller one apart)
    off, size = (got - whole).abs()[fine & again], whole.abs()[fine & again]
    assert bool((off <= 2.0 ** -7 * size + 1e-5).all()) and float((off > 0).double().mean()) < 0.05, float((off - 2.0 ** -7 * size).max())
