"""The latent attention part where a step's keys and values are spelled out: the branch that a step takes, the matrix of key and value rows that the part
makes, its product and the attention over it, with and without a query latent, sinks, rows that another layer wrote, outputs among a wider
matrix's columns.  Against the definition in 64 bits over the cache's rows, and against the form that moves the matrices to query and output.

On the way the query latent, the queries, a row's keys and values and the result are rounded to bfloat16 (2^-9 of a number each; the other form has as many),
weights and sums are not: 5 * 2^-9 of the result's 2-norm for either form, twice that between them."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, PS = "cuda:0", 16
REQS = [(70, 130), (0, 37), (300, 5), (20, 1)]            # (cached, new) of the step's requests
H, D, R, C, W = 3, 64, 32, 256, 192


def _part(E, q_rank, sink, own, gen):
    from forge_b200.config.base import PartSpec
    from forge_b200.parts import Runtime, build_part
    part = build_part("mixer", PartSpec("latent_attention", dict(
        hidden_size=W, num_heads=H, head_dim=D, rot_dim=R, v_head_dim=E, kv_rank=C, q_rank=q_rank, scale=1.5 * (D + R) ** -0.5, eps=1e-5, own_latent=own, sink=sink,
        position=PartSpec("rope_pairs", {"head_dim": R, "rotary_dims": R, "theta": 10000.0}))), Runtime(torch.device(DEV), torch.bfloat16))
    tensors = {}
    for name, spec in part.tensor_specs().items():
        t = torch.randn(tuple(spec.shape), generator=gen)
        tensors[name] = (1.0 + 0.1 * t if spec.role == "norm" else t if spec.role == "bias" else t * spec.shape[-1] ** -0.5).to(torch.bfloat16)
    part.bind({n: t.to(DEV) for n, t in tensors.items()})
    return part, {n[len("mix."):]: t.double() for n, t in tensors.items()}


def _step(part, gen):
    from forge_b200.cache.storage import CacheStorage
    from forge_b200.engine import StepEntry
    from forge_b200.engine.batch import build_step_batch
    pages = sum(-(-(c + n) // PS) for c, n in REQS) + 1
    store = CacheStorage([part.cache_spec()], [None], PS, pages, len(REQS), torch.bfloat16, torch.device(DEV))
    for i, (c, _) in enumerate(REQS):
        store.manager.admit(i)
        if c:
            store.manager.append(i, c)
    cache = store.layers[0]
    cache.kv.copy_(torch.randn(cache.kv.shape, generator=gen).to(torch.bfloat16))
    return store, cache, build_step_batch([StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(REQS)], store.manager, torch.device(DEV),
                                          max(-(-(c + n) // PS) for c, n in REQS))


def _oracle(part, t, x, cache, batch, E, sink):
    h = x.double().cpu()
    if part.q_rank is None:
        q = h @ t["q"].T
    else:
        cq = h @ t["dq"].T
        q = (cq / torch.sqrt((cq * cq).mean(dim=1, keepdim=True) + 1e-5) * t["dq.norm"]) @ t["uq"].T
    q = q.view(-1, H, D + R)
    rows = cache.kv.double().cpu().view(-1, PS, C + R)
    table, out, at = batch.groups[cache.group].block_table.cpu(), [], 0
    for s, (c, n) in enumerate(REQS):
        a = torch.arange(c, c + n).double()[:, None, None] * part.position.inv_freq.double().cpu()
        cs, sn = torch.cos(a), torch.sin(a)
        qs = q[at:at + n]
        u, v = qs[..., D::2], qs[..., D + 1::2]
        qs = torch.cat([qs[..., :D], torch.stack([u * cs - v * sn, v * cs + u * sn], -1).flatten(-2)], -1)
        r = torch.stack([rows[table[s, j // PS], j % PS] for j in range(c + n)])
        hidden = torch.arange(c + n)[None, :] > torch.arange(c, c + n)[:, None]
        for h_ in range(H):
            k = torch.cat([r[:, :C] @ t["uk"].view(H, D, C)[h_].T, r[:, C:]], -1)
            sc = (qs[:, h_] @ k.T * part.scale).masked_fill(hidden, float("-inf"))
            if sink:
                sc = torch.cat([sc, t["sink"][h_].expand(n, 1)], -1)
            out.append((at, h_, torch.softmax(sc, -1)[:, :c + n] @ (r[:, :C] @ t["uv"].view(H, E, C)[h_].T)))
        at += n
    o = torch.empty(at, H, E, dtype=torch.float64)
    for a0, h_, y in out:
        o[a0:a0 + len(y), h_] = y
    return o.view(at, H * E)


@pytest.mark.parametrize("E,q_rank,sink,own,placed", [(64, 96, False, True, False), (128, None, True, True, True), (64, None, False, False, False), (64, 96, True, False, True)])
def test_a_step_of_the_part(monkeypatch, E, q_rank, sink, own, placed):
    from forge_b200 import kernels
    gen = torch.Generator().manual_seed(E + (q_rank or 0) + sink)
    part, t = _part(E, q_rank, sink, own, gen)
    assert part.w_kv is not None and tuple(part.w_kv.shape) == (H * (D + E), C)
    _, cache, batch = _step(part, gen)
    T = batch.num_tokens
    x = torch.randn(T, W, generator=gen).to(torch.bfloat16).to(DEV)
    if not own:                                               # the rows are another layer's
        writer, _ = _part(E, q_rank, sink, True, gen)
        writer.mix(writer.proj.forward(x), 0, batch, cache)
    ran, attend = [], kernels.expanded_attention
    monkeypatch.setattr(kernels, "expanded_attention", lambda *a, **k: ran.append(1) or attend(*a, **k))
    got = []
    for pays in (True, False):
        monkeypatch.setattr(kernels, "latent_expand_pays", lambda *a: pays)
        wide = torch.full((T, H * E + 6), 3.0, dtype=torch.bfloat16, device=DEV)
        y = part.mix(part.proj.forward(x), 0, batch, cache, out=(wide, 2) if placed else None)
        kernels.check_kernel_status(DEV)
        got.append((wide[:, 2:2 + H * E] if placed else y).double().cpu())
        assert len(ran) == 1                                  # the first pass spelled them out, the second did not
        if placed:
            assert bool((wide[:, :2] == 3.0).all()) and bool((wide[:, 2 + H * E:] == 3.0).all())
    want = _oracle(part, t, x, cache, batch, E, sink)
    size = want.norm()
    assert all(float((y - want).norm() / size) <= 5 * 2.0 ** -9 for y in got) and float((got[0] - got[1]).norm() / size) <= 10 * 2.0 ** -9
    # no head, request or row stands out: the largest difference against the largest number
    assert float((got[0] - want).abs().max()) <= 2.0 ** -5 * float(want.abs().max())


def test_an_odd_place_among_the_outputs_stays_absorbed(monkeypatch):
    """The kernel's stores want pairs of bfloat16: an odd first column or width takes the other form, whatever pays."""
    from forge_b200 import kernels
    gen = torch.Generator().manual_seed(1)
    part, t = _part(64, None, False, True, gen)
    _, cache, batch = _step(part, gen)
    x = torch.randn(batch.num_tokens, W, generator=gen).to(torch.bfloat16).to(DEV)
    monkeypatch.setattr(kernels, "latent_expand_pays", lambda *a: True)
    monkeypatch.setattr(kernels, "expanded_attention", None)
    wide = torch.zeros(batch.num_tokens, H * 64 + 5, dtype=torch.bfloat16, device=DEV)
    part.mix(part.proj.forward(x), 0, batch, cache, out=(wide, 3))
    want = _oracle(part, t, x, cache, batch, 64, False)
    assert float((wide[:, 3:3 + H * 64].double().cpu() - want).norm() / want.norm()) <= 5 * 2.0 ** -9


@pytest.mark.parametrize("option", [{"window": 64}, {"out_gate": "channel"}])
def test_windows_and_gates_have_no_such_form(option):
    from forge_b200.config.base import PartSpec
    from forge_b200.parts import Runtime, build_part
    part = build_part("mixer", PartSpec("latent_attention", dict(
        hidden_size=W, num_heads=H, head_dim=D, rot_dim=R, v_head_dim=64, kv_rank=C, q_rank=None, scale=0.1, eps=1e-5,
        position=PartSpec("rope_pairs", {"head_dim": R, "rotary_dims": R, "theta": 10000.0}), **option)), Runtime(torch.device(DEV), torch.bfloat16))
    part.bind({n: torch.zeros(tuple(s.shape), dtype=torch.bfloat16, device=DEV) for n, s in part.tensor_specs().items()})
    assert part.w_kv is None
