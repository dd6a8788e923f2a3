"""A page of -1 inside the range that a token sees: its keys and values count as zeros in the tcgen05 attentions of prompt portions, bit for bit what a page of
zeros gives, for pages that hold a whole tile of 64 keys and for shorter ones, behind enough keys that every slot of the rings has held others."""
from types import SimpleNamespace

import pytest
import torch

from test_attention_mma_gpu import make_case
from test_attention_shaped_gpu import DEV, _batch, _fill

pytestmark = pytest.mark.gpu
REQS = [(900, 70), (0, 200)]


def _missing(table, ps):
    """(request, place in its table) of the pages that are taken away: amid the first request's cached tokens, and amid the second's own."""
    return [(0, 600 // ps), (0, 700 // ps), (1, 70 // ps)]


def _both(table, ps, clear, run):
    """run() with the pages in the table and zeros in them, and without them."""
    whole, holes = table.clone(), table.clone()
    for s, i in _missing(table, ps):
        clear(int(table[s, i]))
        holes[s, i] = -1
    want = run(SimpleNamespace(block_table=whole.to(DEV))).clone()
    return run(SimpleNamespace(block_table=holes.to(DEV))), want


@pytest.mark.parametrize("nh,nkv,hd,ps", [(8, 2, 64, 64), (8, 2, 128, 64), (6, 2, 64, 16), (4, 1, 128, 8)])
def test_paged(nh, nkv, hd, ps):
    from forge_b200 import kernels as k
    q, cache, group, batch, _, _ = make_case(nh, nkv, hd, ps, REQS)
    got, want = _both(group.block_table.cpu(), ps, lambda page: cache[page].zero_(),
                      lambda g: k.paged_attention_sm100(q, cache, g, batch, nh, nkv, hd, ps, shares=1)[0])
    k.check_kernel_status()
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)


@pytest.mark.parametrize("H,C,R,ps", [(32, 512, 64, 64), (4, 256, 32, 128), (5, 64, 16, 8)])
def test_latent(H, C, R, ps):
    from forge_b200 import kernels as k
    batch, table, n_pages, g = _batch(REQS, ps, C + R, seed=H)
    cache = torch.empty(n_pages, ps * (C + R), dtype=torch.bfloat16)
    _fill(cache.view(n_pages, ps, C + R), table, REQS, ps, g)
    cache = cache.to(DEV)
    q = torch.randn(batch.num_tokens, H * (C + R), generator=g).to(torch.bfloat16).to(DEV)
    got, want = _both(table, ps, lambda page: cache[page].zero_(), lambda gr: k.latent_attention(q, cache, gr, batch, H, C, R, ps, 0.05))
    k.check_kernel_status(DEV)
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)


@pytest.mark.parametrize("H,G,M,D,E,ps", [(16, 2, 2, 64, 128, 64), (8, 2, 1, 128, 64, 16)])
def test_scored(H, G, M, D, E, ps):
    from forge_b200 import kernels as k
    batch, table, n_pages, g = _batch(REQS, ps, M * D, seed=H)
    cache = torch.empty(n_pages, G * ps * (M * D + E), dtype=torch.bfloat16)
    _fill(cache[:, :G * ps * M * D].unflatten(1, (G, ps, M * D)).transpose(1, 2), table, REQS, ps, g)
    _fill(cache[:, G * ps * M * D:].unflatten(1, (G, ps, E)).transpose(1, 2), table, REQS, ps, g)
    cache = cache.to(DEV)
    q = torch.randn(batch.num_tokens, H * M * D, generator=g).to(torch.bfloat16).to(DEV)
    got, want = _both(table, ps, lambda page: cache[page].zero_(), lambda gr: k.scored_attention(q, cache, gr, batch, H, G, M, D, E, ps, 0.1, lam=0.5, post=0.5, eps=1e-5))
    k.check_kernel_status(DEV)
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)
