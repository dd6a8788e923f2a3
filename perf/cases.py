"""Cases that time the framework: the work that a program has the engine do, through the entry points that such a program calls.

Two cases are whole models driven through ``ModelRunner`` (prompts in one step, then decode steps, logits kept); the others are one
part of a layer (a mixer or a feed-forward of the part registry) over the batch of one step, in the two forms that the engine itself
gives it: a step with prompt portions launches the part's kernels, a decode step (one new token for each request) replays a CUDA graph
that captured them.  Layer sizes are those of ``bench.py`` (widths 2048 and 4096, the shapes that its designs are measured at).

A case's requests are ragged: ``tokens`` new tokens are dealt out to ``requests`` requests unevenly, and the first request has ``cached``
tokens behind it, the last ones few or none.
"""
import math
from types import SimpleNamespace

import torch

from forge_b200.cache.storage import CacheStorage
from forge_b200.config import config_from_dict
from forge_b200.config.base import PartSpec
from forge_b200.engine import ModelRunner, StepEntry
from forge_b200.engine.batch import build_step_batch
from forge_b200.kernels import StepWorkspace
from forge_b200.parts import KVCacheSpec, Runtime, StateSpec, build_part
from forge_b200.weights import random_tensors

DEVICE, PAGE, EPS = "cuda:0", 64, 1e-5
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def listed():
    return [
        # serving a small LLaMA-shaped model: eight ragged prompts in one step, then eight decode steps of the whole batch
        {"name": "generate bf16", "part": "generate", "dtype": "bf16", "layers": 22, "width": 2048, "heads": 32, "kv_heads": 4, "dim": 64,
         "ff": 5632, "vocab": 32000, "requests": 8, "tokens": 1021, "steps": 8},
        # the same decoder computed in 32 bits, as someone does who checks a model's numbers: two prompts, six decode steps
        {"name": "generate fp32", "part": "generate", "dtype": "fp32", "layers": 4, "width": 2048, "heads": 32, "kv_heads": 4, "dim": 64,
         "ff": 5632, "vocab": 32000, "requests": 2, "tokens": 333, "steps": 6},
        # chunked prefill: portions of three prompts, two of them with cached tokens behind them, through a grouped-query attention layer
        {"name": "attention prompt", "part": "attention", "mode": "prompt", "dtype": "bf16", "width": 4096, "heads": 32, "kv_heads": 8, "dim": 128,
         "requests": 3, "tokens": 1500, "cached": 1000},
        # decode of 32 conversations of up to 4,096 tokens through the same layer
        {"name": "attention decode", "part": "attention", "mode": "decode", "dtype": "bf16", "width": 4096, "heads": 32, "kv_heads": 8, "dim": 128,
         "requests": 32, "tokens": 32, "cached": 4000},
        # the smallest call: one token of one request through a small model's gated feed-forward
        {"name": "feed-forward decode", "part": "dense", "mode": "decode", "dtype": "bf16", "width": 2048, "ff": 5632, "requests": 1, "tokens": 1,
         "cached": 100},
        # decode of a batch of eight through a routed feed-forward, and a prompt step through a smaller one
        {"name": "routed decode", "part": "routed", "mode": "decode", "dtype": "bf16", "width": 4096, "ff": 7168, "experts": 8, "top": 2,
         "requests": 8, "tokens": 8, "cached": 100},
        {"name": "routed prompt", "part": "routed", "mode": "prompt", "dtype": "bf16", "width": 2048, "ff": 2816, "experts": 8, "top": 2,
         "requests": 2, "tokens": 1501, "cached": 0},
        # attention over a cached latent: a prompt step of two requests, and decode of sixteen
        {"name": "latent prompt", "part": "latent", "mode": "prompt", "dtype": "bf16", "width": 4096, "heads": 32, "dim": 128, "requests": 2,
         "tokens": 1536, "cached": 700},
        {"name": "latent decode", "part": "latent", "mode": "decode", "dtype": "bf16", "width": 2048, "heads": 32, "dim": 64, "requests": 16,
         "tokens": 16, "cached": 2000},
        # differential attention over one long prompt
        {"name": "differential prompt", "part": "differential", "mode": "prompt", "dtype": "bf16", "width": 2048, "heads": 16, "kv_heads": 2,
         "dim": 64, "requests": 1, "tokens": 2048, "cached": 0},
        # the gated delta rule over portions of three prompts, and retention's single tokens of 64 requests
        {"name": "delta prompt", "part": "delta", "mode": "prompt", "dtype": "bf16", "width": 2048, "heads": 32, "kv_heads": 16, "dim": 64,
         "requests": 3, "tokens": 2001, "cached": 500},
        {"name": "retention decode", "part": "retention", "mode": "decode", "dtype": "bf16", "width": 4096, "heads": 64, "dim": 64, "requests": 64,
         "tokens": 64, "cached": 900},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    part = rng.choice(["attention", "differential", "latent", "delta", "retention", "dense", "routed", "generate"])
    if part == "generate":
        return {"part": part, "dtype": rng.choice(["bf16", "bf16", "fp32"]), "layers": rng.choice([2, 3, 4]), "width": 2048, "heads": 32,
                "kv_heads": 4, "dim": 64, "ff": 5632, "vocab": 32000, "requests": rng.randint(1, 6), "tokens": _log(rng, 12, 400),
                "steps": rng.randint(2, 8)}
    large = rng.random() < 0.5
    case = {"part": part, "mode": rng.choice(["prompt", "decode"]), "dtype": "bf16", "width": 4096 if large else 2048}
    if part in ("attention", "dense") and rng.random() < 0.25:
        case["dtype"] = "fp32"
    if part == "attention":
        case.update(heads=32, kv_heads=8 if large else 4, dim=128 if large else 64)
    elif part == "differential":
        case.update(heads=16, kv_heads=4 if large else 2, dim=128 if large else 64)
    elif part == "latent":
        case.update(heads=32, dim=128 if large else 64)
    elif part == "delta":
        case.update(heads=64 if large else 32, kv_heads=rng.choice([16, 32]), dim=64)
    elif part == "retention":
        case.update(heads=64 if large else 32, dim=64)
    elif part == "dense":
        case.update(ff=14336 if large else 5632)
    else:
        case.update(ff=7168 if large else 2816, experts=8, top=2)
    if case["mode"] == "decode":
        n = _log(rng, 1, 64)
        case.update(requests=n, tokens=n, cached=_log(rng, 40, 4000))
    else:
        case.update(requests=rng.randint(1, 4), tokens=_log(rng, 24, 512 if case["dtype"] == "fp32" else 1600), cached=rng.choice([0, _log(rng, 40, 1000)]))
    return case


# ------------------------------------------------------------------------------------------------------------ a case's inputs

def _requests(case):
    """[(tokens behind it, new tokens)] of every request."""
    n, total = case["requests"], case["tokens"]
    shares = [i + 1 for i in range(n)]
    new = [max(1, total * s // sum(shares)) for s in shares]
    new[-1] += total - sum(new)
    cached = [case.get("cached", 0) * (n - i) // n for i in range(n)]
    if case.get("mode") == "prompt" and n > 1:
        cached[-1] = 0                                       # a prompt that begins with this step
    return list(zip(cached, new))


def _part_spec(case):
    """(category, PartSpec) of the layer's part, as the configurations of ``bench.py`` make it."""
    W, D, H = case["width"], case.get("dim"), case.get("heads")
    kind = case["part"]
    if kind == "attention":
        return "mixer", PartSpec("attention", dict(hidden_size=W, num_heads=H, num_kv_heads=case["kv_heads"], head_dim=D,
                                                   position=PartSpec("rope", {"head_dim": D, "theta": 10000.0})))
    if kind == "differential":
        return "mixer", PartSpec("differential_attention", dict(
            hidden_size=W, num_heads=H, num_kv_heads=case["kv_heads"], head_dim=D, v_head_dim=2 * D, diff=0.5, eps=EPS, scale=D ** -0.5,
            position=PartSpec("rope_halves", {"head_dim": D, "rotary_dims": D // 2, "theta": 10000.0})))
    if kind == "latent":
        return "mixer", PartSpec("latent_attention", dict(
            hidden_size=W, num_heads=H, head_dim=D, rot_dim=D // 2, v_head_dim=D, kv_rank=4 * D, q_rank=3 * W // 4, scale=(1.5 * D) ** -0.5, eps=EPS,
            position=PartSpec("rope_pairs", {"head_dim": D // 2, "rotary_dims": D // 2, "theta": 10000.0})))
    if kind == "delta":
        return "mixer", PartSpec("gated_delta", dict(hidden_size=W, num_heads=H, num_qk_heads=case["kv_heads"], head_dim=D, taps=4, eps=EPS))
    if kind == "retention":
        return "mixer", PartSpec("retention", dict(hidden_size=W, num_heads=H, head_dim=D, decay=_decays(H), eps=EPS,
                                                   position=PartSpec("rope_halves", {"head_dim": D, "rotary_dims": D, "theta": 10000.0})))
    if kind == "dense":
        return "feed_forward", PartSpec("swiglu", dict(hidden_size=W, intermediate_size=case["ff"]))
    return "feed_forward", PartSpec("routed_experts", dict(hidden_size=W, intermediate_size=case["ff"], experts=case["experts"], top=case["top"]))


def _decays(heads):
    return [1.0 - 2.0 ** (-4.0 - 6.0 * n / max(1, heads - 1)) for n in range(heads)]


def _weights(specs, gen, dtype):
    """Random tensors of a part's specs: outputs of the size of their inputs."""
    out = {}
    for name, spec in specs.items():
        shape = tuple(spec.shape)
        t = torch.randn(shape, generator=gen, device=DEVICE)
        if spec.role == "norm":
            t = 1.0 + 0.1 * t
        elif spec.role == "filter":
            t = 0.3 * t
            t[:, -1] += 1.0
        elif spec.role == "lambda_part":
            t = 0.7 * t / shape[0] ** 0.25
        elif spec.role == "bias":
            t = 0.5 * t
        else:
            t = t * shape[-1] ** -0.5
        out[name] = t if spec.role == "norm" else t.to(dtype)
    return out


def _layer(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    rt = Runtime(torch.device(DEVICE), dtype)
    category, spec = _part_spec(case)
    part = build_part(category, spec, rt)
    s = SimpleNamespace(case=case, part=part, requests=_requests(case), tensors=_weights(part.tensor_specs(), gen, dtype))
    part.bind(s.tensors)
    W, T = case["width"], sum(n for _, n in s.requests)
    s.x = torch.randn(T, W, generator=gen, device=DEVICE).to(dtype)
    s.residual = 0.1 * torch.randn(T, W, generator=gen, device=DEVICE)
    cache_spec = part.cache_spec() if category == "mixer" else None
    s.cache = s.batch = None
    if cache_spec is not None:
        pages = sum(-(-(c + n) // PAGE) for c, n in s.requests) + 1
        store = CacheStorage([cache_spec], [None], PAGE, pages, len(s.requests), dtype, torch.device(DEVICE))
        s.cache = store.layers[0]
        for i, (c, _) in enumerate(s.requests):
            store.manager.admit(i)
            if c:
                store.manager.append(i, c)
        if isinstance(cache_spec, KVCacheSpec):
            s.cache.kv.copy_(torch.randn(s.cache.kv.shape, generator=gen, device=DEVICE, dtype=dtype))
        if isinstance(cache_spec, StateSpec):
            s.cache.state.copy_(0.3 * torch.randn(s.cache.state.shape, generator=gen, device=DEVICE))
            for i, (c, _) in enumerate(s.requests):
                if not c:
                    s.cache.state[store.manager.slot(i)].zero_()
        s.slots = [store.manager.slot(i) for i in range(len(s.requests))]
        entries = [StepEntry(i, [0] * n, []) for i, (_, n) in enumerate(s.requests)]
        s.batch = build_step_batch(entries, store.manager, torch.device(DEVICE), max(-(-(c + n) // PAGE) for c, n in s.requests))
        s.tables = {g: [store.manager.block_table(i, g) for i in range(len(s.requests))] for g in store.manager.groups}
        if case["mode"] == "decode":                        # as a decode step that a graph replays is described to its parts
            s.batch.decode_only = True
            s.batch.max_context = max(256, 1 << max(c for c, _ in s.requests).bit_length())
    return s


def _forward(s):
    if s.batch is not None:
        return s.part.forward(s.x, s.batch, s.cache, s.residual)
    return s.part.forward(s.x, s.residual)


def _kept(s):
    return [s.residual] + [t for t in (getattr(s.cache, "kv", None), getattr(s.cache, "state", None)) if t is not None]


def prepare(case, seed):
    if case["part"] == "generate":
        return _prepare_generate(case, seed)
    s = _layer(case, seed)
    s.graph = None
    if case["mode"] == "decode":
        kept = [t.clone() for t in _kept(s)]
        _forward(s)                                          # once by itself, as the engine does before it captures
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _forward(s)
        for t, old in zip(_kept(s), kept):
            t.copy_(old)
    else:
        s.workspace = StepWorkspace(DEVICE)                  # what the engine's steps cut their intermediates from
    return s


def run(s):
    if s.case["part"] == "generate":
        return _run_generate(s)
    if s.graph is not None:
        s.graph.replay()
    else:
        with s.workspace.step():
            _forward(s)
    out = {"residual": s.residual}
    if s.cache is not None and s.cache.kv is not None:
        out["cache"] = s.cache.kv
    if s.cache is not None and s.cache.state is not None:
        out["state"] = s.cache.state
    return out


# ------------------------------------------------------------------------------------------------------------ whole models

def _config(case):
    return config_from_dict(dict(architectures=["LlamaForCausalLM"], vocab_size=case["vocab"], hidden_size=case["width"],
                                 intermediate_size=case["ff"], num_hidden_layers=case["layers"], num_attention_heads=case["heads"],
                                 num_key_value_heads=case["kv_heads"], head_dim=case["dim"], rope_theta=10000.0, rms_norm_eps=EPS,
                                 attention_bias=False, tie_word_embeddings=False, max_position_embeddings=2048))


def _model_inputs(case, seed):
    tensors = random_tensors(_config(case), seed=seed, std=0.02, embed_std=0.5, dtype=DTYPES[case["dtype"]], device=DEVICE)
    gen = torch.Generator().manual_seed(seed)
    prompts = [torch.randint(0, case["vocab"], (n,), generator=gen).tolist() for _, n in _requests(case)]
    steps = torch.randint(0, case["vocab"], (case["steps"], case["requests"]), generator=gen).tolist()
    return tensors, prompts, steps


def _prepare_generate(case, seed):
    tensors, prompts, steps = _model_inputs(case, seed)
    room = sum(-(-(len(p) + case["steps"]) // PAGE) * PAGE for p in prompts)
    runner = ModelRunner(config=_config(case), tensors=tensors, dtype=DTYPES[case["dtype"]], device=DEVICE, page_size=PAGE, cache_tokens=room,
                         max_requests=case["requests"])
    return SimpleNamespace(case=case, runner=runner, prompts=prompts, steps=steps)


def _run_generate(s):
    r, ids = s.runner, list(range(len(s.prompts)))
    for i in ids:
        r.admit(i)
    logits = [r.step([StepEntry(i, p, [len(p) - 1]) for i, p in zip(ids, s.prompts)])]
    for tokens in s.steps:
        logits.append(r.step([StepEntry(i, [t], [0]) for i, t in zip(ids, tokens)]))
    for i in ids:
        r.release(i)
    return logits


# ------------------------------------------------------------------------------------------------------------ what a pass cannot do without

def _pairs(requests):
    """(token, key) pairs that causal attention sees."""
    return sum(n * c + n * (n + 1) // 2 for c, n in requests)


def _matrices(case):
    """(elements of the matrices that a token passes through, elements of those that the step reads)"""
    W, D, H, kind = case["width"], case.get("dim"), case.get("heads"), case["part"]
    if kind == "generate":
        layer = W * D * 2 * (case["heads"] + case["kv_heads"]) + 3 * W * case["ff"]
        return case["layers"] * layer, case["layers"] * layer
    if kind == "dense":
        return 3 * W * case["ff"], 3 * W * case["ff"]
    if kind == "routed":
        one = 3 * W * case["ff"]
        return case["top"] * one, min(case["experts"], case["top"] * case["tokens"]) * one
    if kind == "attention":
        n = 2 * W * D * (H + case["kv_heads"])
    elif kind == "differential":
        n = W * (4 * H * D + 4 * case["kv_heads"] * D)
    elif kind == "latent":
        Cq, C, R = 3 * W // 4, 4 * D, D // 2
        n = W * Cq + Cq * H * (D + R) + W * (C + R) + 2 * H * D * C + W * H * D
    elif kind == "delta":
        n = W * (2 * case["kv_heads"] * D + 2 * H * D + 2 * H) + W * H * D
    else:
        n = 5 * W * H * D
    return n, n


def work(case):
    reqs, W, kind = _requests(case), case["width"], case["part"]
    T, el = sum(n for _, n in reqs), 4 if case["dtype"] == "fp32" else 2
    through, read = _matrices(case)
    if kind == "generate":
        R, S, V = case["requests"], case["steps"], case["vocab"]
        after = [(n, S) for _, n in reqs]
        flops = 2 * through * (T + R * S) + 2 * W * V * R * (1 + S) + 4 * case["layers"] * case["heads"] * case["dim"] * (_pairs(reqs) + _pairs(after))
        row = 2 * case["layers"] * case["kv_heads"] * case["dim"] * el
        return {"bytes": (read + W * V) * el * (1 + S) + row * (2 * T + R * S + _pairs(after)) + R * (1 + S) * V * 4, "flops": flops}
    flops, size = 2 * through * T, read * el + T * W * (el + 8)
    cached = sum(c for c, _ in reqs)
    H, D = case.get("heads", 0), case.get("dim", 0)
    if kind == "attention":
        flops += 4 * H * D * _pairs(reqs)
        size += 2 * case["kv_heads"] * D * el * (cached + T)
    elif kind == "differential":
        flops += 12 * H * D * _pairs(reqs)                   # two maps of D channels, each over values of 2 D
        size += 4 * case["kv_heads"] * D * el * (cached + T)
    elif kind == "latent":
        flops += 2 * H * (D + D // 2 + D) * _pairs(reqs)
        size += (4 * D + D // 2) * el * (cached + T)
    elif kind == "delta":
        flops += 8 * T * H * D * D
        size += len(reqs) * 2 * 4 * H * D * D
    elif kind == "retention":
        flops += 4 * T * H * D * D
        size += len(reqs) * 2 * 4 * H * D * D
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """32-bit runs: about four times what sums in another order change.  16-bit activations between a part's products: a change of
    rounding before one of them moves its result by parts of 2^-9; a whole model adds that up over its layers."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 3e-4}
    if case["part"] == "generate":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 8e-3, "max": 0.1}


# ------------------------------------------------------------------------------------------------------------ the same in 64 bits

def _rms(x):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + EPS)


def _turn(x, positions, dims, neighbours=False):
    """Rotates the first ``dims`` channels of x [T, heads, D] by position: channel i with i + dims/2, or (``neighbours``) 2i with 2i + 1."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    a = (positions.double()[:, None] * 10000.0 ** (-2.0 * i / dims))[:, None, :]
    c, s = torch.cos(a), torch.sin(a)
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        turned = torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        turned = torch.cat([u * c - v * s, v * c + u * s], dim=-1)
    return torch.cat([turned, x[..., dims:]], dim=-1)


def _attend(q, k, v, c, scale):
    """q [n, H, D] at positions c .. c + n - 1; k [c + n, G, D], v [c + n, G, E] -> [n, H, E]."""
    n, share = q.shape[0], q.shape[1] // k.shape[1]
    hidden = torch.arange(c + n, device=q.device)[None, :] > c + torch.arange(n, device=q.device)[:, None]
    heads = []
    for h in range(q.shape[1]):
        p = torch.softmax((q[:, h] @ k[:, h // share].t() * scale).masked_fill(hidden, -math.inf), dim=-1)
        heads.append(p @ v[:, h // share])
    return torch.stack(heads, dim=1)


def _by_request(s):
    """(index, tokens behind, first and last token of the step) of every request."""
    at, out = 0, []
    for i, (c, n) in enumerate(s.requests):
        out.append((i, c, at, at + n))
        at += n
    return out


def _rows_of(table, positions):
    return torch.tensor([table[p // PAGE] for p in positions], device=DEVICE), torch.tensor([p % PAGE for p in positions], device=DEVICE)


def _exact_attention(s, w, x, positions):
    case = s.case
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    q, k, v = (x @ w[f"self_attn.{n}_proj.weight"].t() for n in "qkv")
    T = x.shape[0]
    q, k, v = _turn(q.view(T, H, D), positions, D), _turn(k.view(T, G, D), positions, D), v.view(T, G, D)
    kv, outs = s.cache.kv.double(), []
    for i, c, lo, hi in _by_request(s):
        page, row = _rows_of(s.tables[s.cache.group][i], range(c, c + hi - lo))
        kv[page, 0, :, row], kv[page, 1, :, row] = k[lo:hi], v[lo:hi]
        page, row = _rows_of(s.tables[s.cache.group][i], range(c + hi - lo))
        outs.append(_attend(q[lo:hi], kv[page, 0, :, row], kv[page, 1, :, row], c, D ** -0.5))
    return torch.cat(outs).reshape(T, H * D) @ w["self_attn.o_proj.weight"].t(), kv


def _exact_differential(s, w, x, positions):
    case = s.case
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    T = x.shape[0]
    q, k = (_turn((x @ w["mix." + n].t()).view(T, heads * 2, D), positions, D // 2) for n, heads in (("q", H), ("k", G)))
    v = (x @ w["mix.v"].t()).view(T, G, 2 * D)
    lam = math.exp(float(w["mix.lq1"] @ w["mix.lk1"])) - math.exp(float(w["mix.lq2"] @ w["mix.lk2"])) + 0.5
    kv, outs = s.cache.kv.double(), []
    flat, half = kv.view(kv.shape[0], -1), G * PAGE * 2 * D
    keys, values = (z.unflatten(1, (G, PAGE, 2 * D)) for z in (flat[:, :half], flat[:, half:]))
    for i, c, lo, hi in _by_request(s):
        page, row = _rows_of(s.tables[s.cache.group][i], range(c, c + hi - lo))
        keys[page, :, row], values[page, :, row] = k[lo:hi].reshape(-1, G, 2 * D), v[lo:hi]
        page, row = _rows_of(s.tables[s.cache.group][i], range(c + hi - lo))
        ks, vs, qs = keys[page, :, row], values[page, :, row], q[lo:hi].view(-1, H, 2, D)
        one, two = (_attend(qs[:, :, m], ks[..., m * D:(m + 1) * D], vs, c, D ** -0.5) for m in range(2))
        outs.append(_rms(one - lam * two) * 0.5)
    return torch.cat(outs).reshape(T, -1) @ w["mix.o"].t(), kv


def _exact_latent(s, w, x, positions):
    case = s.case
    H, D = case["heads"], case["dim"]
    R, C, T = D // 2, 4 * D, x.shape[0]
    q = ((_rms(x @ w["mix.dq"].t()) * w["mix.dq.norm"]) @ w["mix.uq"].t()).view(T, H, D + R)
    q_flat, q_rot = q[..., :D], _turn(q[..., D:], positions, R, neighbours=True)
    both = x @ w["mix.dkv"].t()
    new = torch.cat([_rms(both[:, :C]) * w["mix.dkv.norm"], _turn(both[:, None, C:], positions, R, neighbours=True)[:, 0]], dim=-1)
    kv, outs = s.cache.kv.double(), []
    rows = kv.view(-1, PAGE, C + R)
    for i, c, lo, hi in _by_request(s):
        page, row = _rows_of(s.tables[s.cache.group][i], range(c, c + hi - lo))
        rows[page, row] = new[lo:hi]
        page, row = _rows_of(s.tables[s.cache.group][i], range(c + hi - lo))
        seen = rows[page, row]
        k = torch.cat([(seen[:, :C] @ w["mix.uk"].t()).view(-1, H, D), seen[:, None, C:].expand(-1, H, R)], dim=-1)
        outs.append(_attend(torch.cat([q_flat, q_rot], dim=-1)[lo:hi], k, (seen[:, :C] @ w["mix.uv"].t()).view(-1, H, D), c, (1.5 * D) ** -0.5))
    return torch.cat(outs).reshape(T, H * D) @ w["mix.o"].t(), kv


def _exact_delta(s, w, x, positions):
    case = s.case
    N, M, K, taps = case["heads"], case["kv_heads"], case["dim"], 4
    T = x.shape[0]
    silu = torch.nn.functional.silu
    state = s.cache.state.double()
    raw = torch.cat([x @ w["mix." + n].t() for n in "qkv"], dim=1)
    filt = torch.cat([w[f"mix.{n}.conv"] for n in "qkv"], dim=0)
    beta = torch.sigmoid(x @ w["mix.b"].t())
    g = torch.exp(-torch.exp(w["mix.A_log"]) * torch.nn.functional.softplus(x @ w["mix.a"].t() + w["mix.dt_bias"]))
    unit = lambda z: z / torch.sqrt((z * z).sum(dim=-1, keepdim=True) + 1e-6)
    channels, off, outs = raw.shape[1], N * K * K, []
    for i, c, lo, hi in _by_request(s):
        row = state[s.slots[i]]
        S, ring = row[:off].view(N, K, K), row[off:off + taps * channels].view(taps, channels)     # the input of position p: row p % taps
        before = [ring[p % taps].clone() if p >= 0 else torch.zeros_like(ring[0]) for p in range(c - taps + 1, c)]
        line = torch.cat([torch.stack(before), raw[lo:hi]])
        mixed = silu(sum(line[j:j + hi - lo] * filt[:, j] for j in range(taps)))
        q, k = (unit(mixed[:, m * M * K:(m + 1) * M * K].view(-1, M, K)).repeat_interleave(N // M, dim=1) for m in range(2))
        q, v = q * K ** -0.5, mixed[:, 2 * M * K:].view(-1, N, K)
        for t in range(hi - lo):
            S.mul_(g[lo + t][:, None, None])
            u = beta[lo + t][:, None] * (v[t] - torch.einsum("nkv,nk->nv", S, k[t]))
            S.add_(k[t][:, :, None] * u[:, None, :])
            outs.append(torch.einsum("nkv,nk->nv", S, q[t]))
        for t in range(max(0, hi - lo - taps), hi - lo):
            ring[(c + t) % taps] = raw[lo + t]
    y = _rms(torch.stack(outs)) * w["mix.norm"] * silu((x @ w["mix.g"].t()).view(T, N, K))
    return y.reshape(T, N * K) @ w["mix.o"].t(), state


def _exact_retention(s, w, x, positions):
    case = s.case
    N, K, T = case["heads"], case["dim"], x.shape[0]
    state, outs = s.cache.state.double(), []
    decay = torch.tensor(_decays(N), dtype=torch.float64, device=DEVICE)[:, None, None]
    q, k, v = ((x @ w["mix." + n].t()).view(T, N, K) for n in "qkv")
    q, k = _turn(q, positions, K), _turn(k, positions, K) * K ** -0.5
    for i, c, lo, hi in _by_request(s):
        S = state[s.slots[i]].view(N, K, K)
        for t in range(lo, hi):
            S.mul_(decay).add_(k[t][:, :, None] * v[t][:, None, :])
            outs.append(torch.einsum("nkv,nk->nv", S, q[t]))
    y = _rms(torch.stack(outs)).reshape(T, N * K) * torch.nn.functional.silu(x @ w["mix.g"].t())
    return y @ w["mix.o"].t(), state


def _gated(x, gate, up, down):
    return (torch.nn.functional.silu(x @ gate.t()) * (x @ up.t())) @ down.t()


def _exact_routed(s, w, x):
    score, chosen = torch.sigmoid(x @ w["mlp.router"].t()).topk(s.case["top"], dim=-1)
    y = torch.zeros_like(x)
    for e in range(s.case["experts"]):
        t, k = (chosen == e).nonzero(as_tuple=True)
        y[t] += score[t, k][:, None] * _gated(x[t], *(w[f"mlp.e{e}.{n}"] for n in ("gate", "up", "down")))
    return y


def _exact_generate(case, seed):
    tensors, prompts, steps = _model_inputs(case, seed)
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    outs = [[] for _ in range(case["steps"] + 1)]
    for i, prompt in enumerate(prompts):
        ids = prompt + [t[i] for t in steps]
        T, positions = len(ids), torch.arange(len(ids), device=DEVICE)
        h = tensors["model.embed_tokens.weight"][torch.tensor(ids, device=DEVICE)].double()
        for n in range(case["layers"]):
            w = lambda name: tensors[f"model.layers.{n}.{name}.weight"].double()      # noqa: B023
            x = _rms(h) * w("input_layernorm")
            q, k = (_turn((x @ w(f"self_attn.{m}_proj").t()).view(T, heads, D), positions, D) for m, heads in (("q", H), ("k", G)))
            v = (x @ w("self_attn.v_proj").t()).view(T, G, D)
            h = h + _attend(q, k, v, 0, D ** -0.5).reshape(T, H * D) @ w("self_attn.o_proj").t()
            h = h + _gated(_rms(h) * w("post_attention_layernorm"), *(w(f"mlp.{m}_proj") for m in ("gate", "up", "down")))
        h = _rms(h[len(prompt) - 1:]) * tensors["model.norm.weight"].double()
        for o, row in zip(outs, h @ tensors["lm_head.weight"].double().t()):
            o.append(row)
    return [torch.stack(o) for o in outs]


def exact(case, seed):
    if case["part"] == "generate":
        return _exact_generate(case, seed)
    s = _layer(case, seed)
    w, x = {n: t.double() for n, t in s.tensors.items()}, s.x.double()
    if case["part"] == "dense":
        return {"residual": s.residual.double() + _gated(x, *(w[f"mlp.{m}_proj.weight"] for m in ("gate", "up", "down")))}
    if case["part"] == "routed":
        return {"residual": s.residual.double() + _exact_routed(s, w, x)}
    positions = torch.cat([torch.arange(c, c + n, device=DEVICE) for c, n in s.requests])
    forms = {"attention": _exact_attention, "differential": _exact_differential, "latent": _exact_latent, "delta": _exact_delta,
             "retention": _exact_retention}
    y, kept = forms[case["part"]](s, w, x, positions)
    return {"residual": s.residual.double() + y, "cache" if s.cache.kv is not None else "state": kept}
