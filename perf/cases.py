"""The work that users of this framework have it do, as cases whose speed and outputs can be compared.

A case is a request (or a batch of them) that goes through the public entry points:

  generate   start(prompt), then advance(steps): prefill and batch-1 decode, greedy or sampled
  score      append(tokens, want): a long prompt's logits at several places (evaluation, replay of given tokens)
  serve      several requests with prompts of different lengths on sessions that share weights, prefilled one by one,
             then advanced together through batch_advance_one (continuous batching)
  attention  paged grouped-query decode attention on device buffers (the allocation-free operator)

Models have the shapes of this repository's configurations and workloads, the largest cut in depth so that a model is
made in seconds.  Their weights come from a fixed seed and stay loaded, like a server's; a state is a fork with its own
cache.  Matrices are N(0, 1 / columns), those that write the residual stream scaled down by the depth, and each row of
the head leans towards the embedding of the token that precedes it in a fixed permutation of the vocabulary: the next
token is as clear as in a trained model, so that a stream of tokens does not hang on the last bit of a logit.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from nerva_b200 import ops, parallel_model, sandwich_model, synth
from nerva_b200.session import CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus, sampler_config

DEVICE = "cuda"
F64 = torch.float64
VOCAB = 151936


# ---------------------------------------------------------------- models ----
def _vuvolix():
    """1.7b widths of the vuvolix workload: 28 layer runs, a third of them second passes, window 1024."""
    spec = parallel_model.ParallelLayer(heads=16, kv_heads=8, qk_dim=128, v_dim=128, intermediate=6144, window=1024,
                                        score_scale=128 ** -0.5, rotary_dims=64, rotary_base=1e6,
                                        scaling={"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0})
    return parallel_model.ParallelConfig(name="vuvolix-1.7b", hidden=2048, vocab=VOCAB, rms_eps=1e-6,
                                         layer_specs=(spec,) * 19, embedding_scale=2048 ** 0.5, logit_softcap=30.0,
                                         loop_start=5, loop_stop=14, loop_times=2)


def _vamidra():
    """The same widths in the vamidra workload: attention and state-space layers in turn."""
    attention = sandwich_model.attention_layer(heads=16, kv_heads=8, qk_dim=128, v_dim=128, intermediate=6144,
                                               window=1024, keep_first=4, score_scale=128 ** -0.5, score_softcap=50.0)
    space = sandwich_model.StateSpaceLayer(heads=64, v_dim=64, state=128, groups=8, conv=4, norm_groups=8,
                                           intermediate=6144)
    return sandwich_model.SandwichConfig(name="vamidra-1.7b", hidden=2048, vocab=VOCAB, rms_eps=1e-5,
                                         layer_specs=tuple(space if i % 2 else attention for i in range(19)),
                                         logit_scale=0.5, loop_start=5, loop_stop=14, loop_times=2)


#: name -> (configuration, tokens of context a session has room for)
MODELS = {
    "tiny": (synth.TINY_QWEN3, 512),
    "dense": (dataclasses.replace(synth.QWEN3_8B, layers=8), 16384),
    "latent-moe": (dataclasses.replace(synth.DEEPSEEK_V2_LITE, layers=6), 2048),
    "moe": (synth.DecoderConfig("moe", layers=6, hidden=2048, heads=16, kv_heads=4, head_dim=128, intermediate=6144,
                                vocab=VOCAB, num_experts=64, top_k=8, moe_intermediate=768, norm_topk_prob=True), 2048),
    "vuvolix": (_vuvolix(), 8192),
    "vamidra": (_vamidra(), 8192),
}


def _runs(cfg):
    return getattr(cfg, "layer_runs", cfg.layers)


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _normal(gen, shape, std, mean=0.0):
    return (torch.randn(shape, generator=gen, device=DEVICE) * std + mean).to(torch.bfloat16)


def _next_token(cfg):
    """The permutation a model follows."""
    return torch.randperm(cfg.vocab, generator=_generator(99), device=DEVICE)


def _decoder_shapes(cfg, layer):
    """name -> shape of one layer of a DecoderConfig."""
    h, a, kv = cfg.hidden, cfg.attention_hidden, cfg.kv_hidden
    shapes = {"rms_attn": (h,), "rms_mlp": (h,)}
    if cfg.kv_lora_rank:
        shapes.update(w_q=(cfg.heads * (cfg.qk_nope_head_dim + cfg.qk_rope_head_dim), h),
                      w_kv_a=(cfg.kv_lora_rank + cfg.qk_rope_head_dim, h), kv_a_norm=(cfg.kv_lora_rank,),
                      w_kv_b=(cfg.heads * (cfg.qk_nope_head_dim + cfg.head_dim), cfg.kv_lora_rank))
    else:
        shapes.update(w_q=(a, h), w_k=(kv, h), w_v=(kv, h), q_norm=(cfg.head_dim,), k_norm=(cfg.head_dim,))
    shapes["w_o"] = (h, a)
    if cfg.num_experts and layer >= cfg.dense_layers:
        e, m, s = cfg.num_experts, cfg.moe_intermediate, cfg.shared_intermediate
        shapes.update(w_router=(e, h), w_expert_gate_up=(e, 2 * m, h), w_expert_down=(e, h, m))
        if s:
            shapes.update(w_shared_expert_gate=(s, h), w_shared_expert_up=(s, h), w_shared_expert_down=(h, s))
    else:
        i = cfg.intermediate
        shapes.update(w_gate=(i, h), w_up=(i, h), w_down=(h, i))
    return shapes


def _shapes(cfg):
    if not isinstance(cfg, synth.DecoderConfig):
        return cfg.tensor_shapes()
    shapes = {"embed": (cfg.vocab, cfg.hidden), "final.norm": (cfg.hidden,), "head": (cfg.vocab, cfg.hidden)}
    for layer in range(cfg.layers):
        shapes.update({f"l{layer}.{k}": v for k, v in _decoder_shapes(cfg, layer).items()})
    return shapes


def _weights(model):
    """name -> bf16 tensor on the GPU."""
    cfg = MODELS[model][0]
    gen, out = _generator(7), {}
    into_stream = ("w_o", "w_down", "w_expert_down", "w_shared_expert_down", "mix.o", "mlp.down")
    behind = ("norm1b", "norm2b")  # the norms whose outputs are added to the stream
    depth = (2 * _runs(cfg)) ** -0.5
    for name, shape in _shapes(cfg).items():
        if name == "embed":
            out[name] = _normal(gen, shape, 1.0 / getattr(cfg, "embedding_scale", 1.0))
        elif name == "head":
            scale = 1.0 / getattr(cfg, "logit_scale", 1.0)
            head = torch.randn(shape, generator=gen, device=DEVICE) * (scale * shape[1] ** -0.5)
            lean = 24.0 * scale / shape[1] * getattr(cfg, "embedding_scale", 1.0)
            head[_next_token(cfg)] += lean * out["embed"].float()
            out[name] = head.to(torch.bfloat16)
        elif name == "loop.step":
            out[name] = _normal(gen, shape, 0.1)
        elif name == "loop.in":
            both = torch.cat([0.9 * torch.eye(shape[0], device=DEVICE), 0.2 * torch.eye(shape[0], device=DEVICE)], dim=1)
            out[name] = (both + torch.randn(shape, generator=gen, device=DEVICE) * 0.2 * shape[1] ** -0.5).to(torch.bfloat16)
        elif name.endswith(".conv"):
            out[name] = _normal(gen, shape, 0.3)
        elif name.endswith(".conv.b"):
            out[name] = _normal(gen, shape, 0.1)
        elif name.endswith(".A_log"):  # decay rates from 1 to 16
            out[name] = torch.linspace(1.0, 16.0, shape[0], device=DEVICE).log().to(torch.bfloat16)
        elif name.endswith(".dt_bias"):  # steps from 0.001 to 0.1
            out[name] = torch.linspace(1e-3, 0.1, shape[0], device=DEVICE).expm1().log().to(torch.bfloat16)
        elif name.endswith("w_router"):
            out[name] = _normal(gen, shape, 2.0 * shape[1] ** -0.5)
        elif len(shape) == 1:
            out[name] = _normal(gen, shape, 0.1, 1.0)
            if name.endswith(behind):
                out[name] = (out[name].float() * depth).to(torch.bfloat16)
        else:
            out[name] = _normal(gen, shape, shape[-1] ** -0.5 * (depth if name.endswith(into_stream) else 1.0))
    return out


def _host(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16)


def _checkpoint(model):
    cfg = MODELS[model][0]
    weights = {name: _host(t) for name, t in _weights(model).items()}
    if not isinstance(cfg, synth.DecoderConfig):
        return parallel_model.ParallelCheckpoint(cfg, weights)
    checkpoint = synth.DenseCheckpoint(cfg, embeddings=weights["embed"].reshape(-1),
                                       final_norm=weights["final.norm"], lm_head=weights["head"].reshape(-1))
    for layer in range(cfg.layers):
        checkpoint.layers.append({k: weights[f"l{layer}.{k}"].reshape(-1) for k in _decoder_shapes(cfg, layer)})
    return checkpoint


_loaded = {}  # the model that is loaded: name -> its first session


def _root(model):
    if model not in _loaded:
        for session in _loaded.values():
            session.destroy()
        _loaded.clear()
        checkpoint = _checkpoint(model)
        torch.cuda.empty_cache()
        # packed steps ask for described weights; sparse models with ordinary attention come by pointers only
        described = not MODELS[model][0].num_experts
        session = CudaHfDecodeSequenceSession(checkpoint, MODELS[model][1], use_descriptors=described)
        if session.status != SmokeStatus.OK:
            raise RuntimeError(f"session create: {session.status} {session.error}")
        _loaded[model] = session
    return _loaded[model]


# ----------------------------------------------------------------- cases ----
def listed():
    return [
        # the smallest request: the tiny decoder that the tests and the CPU path use; launches and latency only
        {"name": "tiny chat", "kind": "generate", "model": "tiny", "prompt": 64, "steps": 32, "sampled": False},
        # a short question and a long answer on the headline model's layers: batch-1 decode, bound by the weights
        {"name": "dense decode", "kind": "generate", "model": "dense", "prompt": 33, "steps": 128, "sampled": False},
        # the headline workload's prompt with the sampler users ask for
        {"name": "dense chat sampled", "kind": "generate", "model": "dense", "prompt": 512, "steps": 64, "sampled": True},
        # a document and a few words about it: long prefill, decode over a long cache
        {"name": "dense long context", "kind": "generate", "model": "dense", "prompt": 12011, "steps": 32, "sampled": False},
        # scoring of given tokens: prefill alone, of a size that is no multiple of anything
        {"name": "dense score", "kind": "score", "model": "dense", "prompt": 3001, "places": 16},
        # a full continuous batch: 32 requests of up to 200 tokens
        {"name": "dense serve 32", "kind": "serve", "model": "dense", "prompt": 200, "steps": 48, "batch": 32},
        # latent attention with sparse and shared experts, its workload's prompt
        {"name": "latent moe chat", "kind": "generate", "model": "latent-moe", "prompt": 1024, "steps": 64, "sampled": False},
        # grouped-query attention with sparse experts
        {"name": "moe chat", "kind": "generate", "model": "moe", "prompt": 300, "steps": 100, "sampled": False},
        # parallel blocks with windowed attention, their workload's prompt
        {"name": "vuvolix chat", "kind": "generate", "model": "vuvolix", "prompt": 2048, "steps": 64, "sampled": False},
        # sandwich blocks, half of the layers state spaces
        {"name": "vamidra chat", "kind": "generate", "model": "vamidra", "prompt": 1500, "steps": 64, "sampled": False},
        # the attention operator: one sequence of a moderate length, and the long-context batch of the sweep
        {"name": "attention 1 x 8k", "kind": "attention", "batch": 1, "context": 8192, "heads": 32, "kv_heads": 8, "dim": 128},
        {"name": "attention 8 x 128k", "kind": "attention", "batch": 8, "context": 131072, "heads": 32, "kv_heads": 8, "dim": 128},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["generate", "generate", "generate", "score", "serve", "attention"])
    if kind == "attention":
        return {"kind": kind, "batch": rng.randint(1, 8), "context": _spread(rng, 1000, 131072),
                "heads": 32, "kv_heads": rng.choice([4, 8, 8, 16]), "dim": rng.choice([64, 128, 128])}
    if kind == "score":
        model = rng.choice(["dense", "dense", "latent-moe", "moe", "vuvolix", "vamidra"])
        return {"kind": kind, "model": model, "prompt": _spread(rng, 40, 900 if "moe" in model else 6000),
                "places": rng.randint(1, 24)}
    if kind == "serve":
        model = rng.choice(["tiny", "dense", "dense", "vuvolix", "vamidra"])
        return {"kind": kind, "model": model, "prompt": _spread(rng, 8, 300), "steps": _spread(rng, 8, 48),
                "batch": _spread(rng, 2, 32)}
    model = rng.choice(["tiny", "dense", "dense", "latent-moe", "moe", "vuvolix", "vamidra"])
    longest = {"tiny": 400, "dense": 12000, "latent-moe": 1024, "moe": 1024}.get(model, 6000)
    return {"kind": kind, "model": model, "prompt": _spread(rng, 2, longest), "steps": _spread(rng, 8, 100),
            "sampled": rng.random() < 0.3}


def _prompts(case, seed):
    """The requests' prompts; those of a batch are of different lengths, up to the case's."""
    cfg, rng = MODELS[case["model"]][0], np.random.default_rng(seed)
    longest = case["prompt"]
    lengths = [longest] + [int(rng.integers(max(1, longest // 4), longest + 1)) for _ in range(case.get("batch", 1) - 1)]
    return [rng.integers(0, cfg.vocab, n).astype(np.uint32) for n in lengths]


def prepare(case, seed):
    if case["kind"] == "attention":
        gen = _generator(seed)
        batch, pages, width = case["batch"], (case["context"] + 15) // 16, case["kv_heads"] * case["dim"]
        keys, values = (torch.empty((batch, pages * 16, width), dtype=torch.bfloat16, device=DEVICE) for _ in range(2))
        for t in (*keys, *values):
            t.normal_(generator=gen)
        return {"case": case, "keys": keys, "values": values,
                "q": torch.randn((batch, case["heads"] * case["dim"]), generator=gen, device=DEVICE),
                "table": torch.stack([torch.randperm(pages, generator=gen, device=DEVICE) for _ in range(batch)]).int(),
                "out": torch.empty((batch, case["heads"] * case["dim"]), device=DEVICE)}
    root = _root(case["model"])
    sessions = [root.fork_shared_weights() for _ in range(case.get("batch", 1))]
    for session in sessions:
        if session.status != SmokeStatus.OK:
            raise RuntimeError(f"session fork: {session.status} {session.error}")
    return {"case": case, "sessions": sessions, "prompts": _prompts(case, seed),
            "places": _places(case) if case["kind"] == "score" else None}


def _places(case):
    """Where a scored prompt's logits are wanted: spread over it, its last token always."""
    count = min(case["places"], case["prompt"])
    return [(i + 1) * case["prompt"] // count - 1 for i in range(count)]


def _start(session, prompt, sampler=None):
    summary, loop = CudaHfDecodeSequenceLoop.start(session, prompt, sampler=sampler)
    if loop is None:
        raise RuntimeError(f"session start: {summary.status} {summary.error}")
    return loop


def run(state):
    case = state["case"]
    if case["kind"] == "attention":
        ops.gqa_decode_attention_static_scratch(
            state["q"].data_ptr(), state["keys"].data_ptr(), state["values"].data_ptr(), state["table"].data_ptr(),
            state["out"].data_ptr(), case["batch"], case["context"], case["heads"], case["kv_heads"], case["dim"],
            stream=torch.cuda.current_stream().cuda_stream)
        return state["out"]
    sessions, prompts = state["sessions"], state["prompts"]
    if case["kind"] == "score":
        return sessions[0].append(prompts[0], want=state["places"], reset=True)
    if case["kind"] == "generate":
        sampler = sampler_config(temperature=0.7, top_p=0.9, top_k=50, seed=11) if case["sampled"] else None
        out = _start(sessions[0], prompts[0], sampler).advance(case["steps"])
        if out.status != SmokeStatus.OK:
            raise RuntimeError(f"session advance: {out.status} {out.error}")
        return {"tokens": np.asarray(out.tokens), "logits": sessions[0].read_logits()}
    # the token that a prompt's prefill has sampled is fetched first: the session then waits for its next step
    tokens = [[_start(session, prompt).advance(1).tokens[0] for session, prompt in zip(sessions, prompts)]]
    for _ in range(case["steps"]):
        out = CudaHfDecodeSequenceSession.batch_advance_one(sessions, target_block_tokens=32, min_block_tokens=1)
        if out.status != SmokeStatus.OK or out.observed_tokens != len(sessions):
            raise RuntimeError(f"batch advance: {out.status} {out.error}")
        tokens.append(out.tokens)
    return {"tokens": np.asarray(tokens), "logits": np.stack([s.read_logits() for s in sessions])}


# ------------------------------------------------------------------ work ----
def _elements(cfg):
    """(matrix elements that one token meets in all layer runs, all matrix elements of the layer runs)."""
    one = every = 0
    in_loop = range(getattr(cfg, "loop_start", 0), getattr(cfg, "loop_stop", 0))
    for name, shape in _shapes(cfg).items():
        if len(shape) < 2 or name in ("embed", "head", "loop.step"):
            continue
        n = math.prod(shape)
        if name == "loop.in":
            n *= cfg.loop_times
        elif int(name[1:name.index(".")]) in in_loop:
            n *= cfg.loop_times
        every += n
        one += n * cfg.top_k // cfg.num_experts if "w_expert" in name else n
    return one, every


def _attention_work(cfg, context):
    """(cache bytes, operations) of one token's attention over `context` positions, all layer runs."""
    if isinstance(cfg, synth.DecoderConfig):
        if cfg.kv_lora_rank:
            width = cfg.kv_lora_rank + cfg.qk_rope_head_dim
            return 2 * width * context * cfg.layers, 2 * cfg.heads * (width + cfg.kv_lora_rank) * context * cfg.layers
        return 4 * cfg.kv_hidden * context * cfg.layers, 4 * cfg.attention_hidden * context * cfg.layers
    total_bytes = flops = 0
    for i, s in enumerate(cfg.layer_specs):
        times = cfg.loop_times if cfg.loop_start <= i < cfg.loop_stop else 1
        if isinstance(s, sandwich_model.StateSpaceLayer):
            total_bytes += 8 * s.inner * s.state * times
            flops += 6 * s.inner * s.state * times
        else:
            seen = min(context, s.window + s.keep_first) if s.window else context
            total_bytes += 2 * s.kv_heads * (s.qk_dim + s.v_dim) * seen * times
            flops += 2 * s.heads * (s.qk_dim + s.v_dim) * seen * times
    return total_bytes, flops


def work(case):
    if case["kind"] == "attention":
        kv = case["batch"] * case["context"] * case["kv_heads"] * case["dim"]
        return {"bytes": 4 * kv + 8 * case["batch"] * case["heads"] * case["dim"],
                "flops": 4 * case["batch"] * case["context"] * case["heads"] * case["dim"]}
    cfg = MODELS[case["model"]][0]
    one, every = _elements(cfg)
    head = cfg.vocab * cfg.hidden
    prompt = case["prompt"]
    batch = case.get("batch", 1)
    lengths = [prompt] + [prompt * 5 // 8] * (batch - 1)  # a batch's other prompts: the mean
    # prompts: the matrices once per prompt (a short one does not reach every expert), the cache written once
    total_bytes = flops = 0
    for n in lengths:
        total_bytes += 2 * min(every, one * n)
        flops += 2 * one * n + sum(_attention_work(cfg, n // 2)[1:]) * n
    places = case.get("places", batch)
    total_bytes += 2 * head + 4 * places * cfg.vocab
    flops += 2 * head * places
    # decode: the matrices and the head once per step for the whole batch, each request's cache
    steps = case["steps"] - 1 if case["kind"] == "generate" else case.get("steps", 0)
    for n in lengths:
        cache, attention = _attention_work(cfg, n + steps // 2)
        total_bytes += steps * cache
        flops += steps * (attention + 2 * (one + head))
    total_bytes += steps * 2 * (min(every, one * batch) + head)
    return {"bytes": total_bytes, "flops": flops}


# ------------------------------------------------------------- exact values ----
def _rms(x, w=None, eps=1e-6):
    y = x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _layer_norm(x, w, eps):
    return _rms(x - x.mean(-1, keepdim=True), w, eps)


def _turned(x, angle, magnitude=1.0):
    """x [T, heads, dim]: pairs (i, i + n) of the first 2n dimensions turned by angle [T, n]."""
    n = angle.shape[1]
    c, s = (angle.cos() * magnitude)[:, None], (angle.sin() * magnitude)[:, None]
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], dim=-1)


def _angles(count, dims, base, scaling=None):
    plain = base ** (-torch.arange(0, dims, 2, dtype=F64, device=DEVICE) / dims)
    magnitude = 1.0
    if scaling:
        def dim_of(turns):
            return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low = max(math.floor(dim_of(scaling["fast"])), 0)
        high = min(math.ceil(dim_of(scaling["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=F64, device=DEVICE) - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        plain = plain / scaling["factor"] * ramp + plain * (1.0 - ramp)
        magnitude = 0.1 * math.log(scaling["factor"]) + 1.0
    return torch.arange(count, dtype=F64, device=DEVICE)[:, None] * plain, magnitude


def _attention(q, k, v, scale, window=0, keep_first=0, cap=0.0):
    """Causal attention; q [T, H, d], k [T, G, d], v [T, G, e]."""
    count, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty((count, heads, v.shape[2]), dtype=F64, device=DEVICE)
    key_at = torch.arange(count, device=DEVICE)
    for begin in range(0, count, 512):
        at = key_at[begin:begin + 512, None]
        see = key_at <= at
        if window:
            see = see & ((at - key_at < window) | (key_at < keep_first))
        for g in range(groups):
            mine = slice(g * heads // groups, (g + 1) * heads // groups)
            score = torch.einsum("thd,sd->hts", q[begin:begin + 512, mine], k[:, g]) * scale
            score = cap * torch.tanh(score / cap) if cap else score
            p = torch.softmax(score.masked_fill(~see, -torch.inf), dim=-1)
            out[begin:begin + 512, mine] = torch.einsum("hts,se->the", p, v[:, g])
    return out


def _experts(cfg, n, get):
    p = torch.softmax(n @ get("w_router").T, dim=-1)
    weight, chosen = torch.topk(p, cfg.top_k, dim=-1)
    if cfg.norm_topk_prob:
        weight = weight / weight.sum(-1, keepdim=True)
    y = torch.zeros_like(n)
    for e in range(cfg.num_experts):
        token, rank = torch.nonzero(chosen == e, as_tuple=True)
        if token.numel():
            gate, up = (n[token] @ get("w_expert_gate_up", e).T).chunk(2, dim=-1)
            y[token] += (torch.nn.functional.silu(gate) * up) @ get("w_expert_down", e).T * weight[token, rank, None]
    if cfg.shared_intermediate:
        gate, up = n @ get("w_shared_expert_gate").T, n @ get("w_shared_expert_up").T
        y += (torch.nn.functional.silu(gate) * up) @ get("w_shared_expert_down").T
    return y


def _decoder_stream(cfg, weights, tokens):
    count = len(tokens)
    x = weights["embed"][tokens].to(F64)
    for layer in range(cfg.layers):
        def get(name, index=None):
            t = weights[f"l{layer}.{name}"]
            return (t if index is None else t[index]).to(F64)
        n = _rms(x, get("rms_attn"), cfg.rms_eps)
        if cfg.kv_lora_rank:
            nope, rope, rank = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.kv_lora_rank
            angle, _ = _angles(count, rope, cfg.rope_theta)

            def paired(t):  # neighbours are a pair here
                return _turned(torch.cat([t[..., 0::2], t[..., 1::2]], dim=-1), angle)
            q = (n @ get("w_q").T).view(count, cfg.heads, nope + rope)
            kv = n @ get("w_kv_a").T
            b = (_rms(kv[:, :rank], get("kv_a_norm"), cfg.rms_eps) @ get("w_kv_b").T).view(count, cfg.heads, -1)
            q = torch.cat([q[..., :nope], paired(q[..., nope:])], dim=-1)
            k = torch.cat([b[..., :nope], paired(kv[:, None, rank:]).expand(-1, cfg.heads, -1)], dim=-1)
            a = _attention(q, k, b[..., nope:], (nope + rope) ** -0.5)
        else:
            angle, _ = _angles(count, cfg.head_dim, cfg.rope_theta)
            q = _rms((n @ get("w_q").T).view(count, cfg.heads, -1), get("q_norm"), cfg.rms_eps)
            k = _rms((n @ get("w_k").T).view(count, cfg.kv_heads, -1), get("k_norm"), cfg.rms_eps)
            v = (n @ get("w_v").T).view(count, cfg.kv_heads, -1)
            a = _attention(_turned(q, angle), _turned(k, angle), v, cfg.head_dim ** -0.5)
        x = x + a.reshape(count, -1) @ get("w_o").T
        n = _rms(x, get("rms_mlp"), cfg.rms_eps)
        if cfg.num_experts and layer >= cfg.dense_layers:
            x = x + _experts(cfg, n, get)
        else:
            x = x + (torch.nn.functional.silu(n @ get("w_gate").T) * (n @ get("w_up").T)) @ get("w_down").T
    return x


def _state_space(s, n, get, eps):
    count, inner, shared = len(n), s.inner, s.groups * s.state
    z, u, step = torch.split(n @ get("in").T, [inner, s.channels, s.heads], dim=1)
    taps = get("conv")
    mixed = get("conv.b").expand(count, -1).clone()
    for back in range(min(s.conv, count)):
        mixed[back:] += taps[:, s.conv - 1 - back] * u[:count - back]
    u = torch.nn.functional.silu(mixed)
    x = u[:, :inner].view(count, s.heads, s.v_dim)
    b, c = (t.view(count, s.groups, s.state).repeat_interleave(s.heads // s.groups, dim=1)
            for t in (u[:, inner:inner + shared], u[:, inner + shared:]))
    step = torch.nn.functional.softplus(step + get("dt_bias"))
    decay = torch.exp(-get("A_log").exp() * step)
    b = b * step[..., None]
    memory = torch.zeros((s.heads, s.state, s.v_dim), dtype=F64, device=DEVICE)
    y = torch.empty_like(x)
    for t in range(count):
        memory = memory * decay[t][:, None, None] + b[t][:, :, None] * x[t][:, None, :]
        y[t] = torch.bmm(c[t][:, None], memory)[:, 0]
    y = (y + x * get("D")[:, None]).view(count, inner) * torch.nn.functional.silu(z)
    y = _rms(y.view(count, s.norm_groups, -1), None, eps).view(count, inner) * get("norm")
    return y @ get("o").T


def _layered_stream(cfg, weights, tokens):
    """Parallel and sandwich blocks."""
    count, eps = len(tokens), cfg.rms_eps
    sandwich = isinstance(cfg, sandwich_model.SandwichConfig)
    first = x = weights["embed"][tokens].to(F64) * getattr(cfg, "embedding_scale", 1.0)
    inside = list(range(cfg.loop_start, cfg.loop_stop))
    runs = [(i, None) for i in range(cfg.loop_start)]
    runs += [(i, t if i == cfg.loop_start else None) for t in range(cfg.loop_times) for i in inside]
    runs += [(i, None) for i in range(cfg.loop_stop, cfg.layers)]
    for index, number in runs:
        s = cfg.layer_specs[index]

        def get(name):
            return weights[f"l{index}.{name}"].to(F64)
        if number is not None:
            if sandwich:
                x = torch.cat([x, first], dim=-1) @ weights["loop.in"].to(F64).T
            x = x + weights["loop.step"][number].to(F64)
        n = _layer_norm(x, get("norm1"), eps) if sandwich else _rms(x, get("norm1"), eps)
        if isinstance(s, sandwich_model.StateSpaceLayer):
            y = _state_space(s, n, lambda name: get("mix." + name), eps)
        else:
            q = (n @ get("mix.q").T).view(count, s.heads, s.qk_dim)
            k = (n @ get("mix.k").T).view(count, s.kv_heads, s.qk_dim)
            v = (n @ get("mix.v").T).view(count, s.kv_heads, s.v_dim)
            if s.rotary_dims:
                angle, magnitude = _angles(count, s.rotary_dims, s.rotary_base, s.scaling)
                q, k = _turned(q, angle, magnitude), _turned(k, angle, magnitude)
            if s.qk_norm:
                q, k = _rms(q, None, eps), _rms(k, None, eps)
            a = _attention(q, k, v, s.score_scale, s.window, s.keep_first, s.score_softcap)
            if s.head_gate:
                a = a * torch.sigmoid(n @ get("mix.g").T)[..., None]
            y = a.reshape(count, -1) @ get("mix.o").T
        if sandwich:
            x = x + _layer_norm(y, get("norm1b"), eps)
            n = _layer_norm(x, get("norm2"), eps)
            y = torch.nn.functional.gelu(n @ get("mlp.gate").T, approximate="tanh") * (n @ get("mlp.up").T)
            x = x + _layer_norm(y @ get("mlp.down").T, get("norm2b"), eps)
        else:
            y = y * get("ls1")
            x = x + y + (torch.nn.functional.silu(n @ get("mlp.gate").T) * (n @ get("mlp.up").T)) @ get("mlp.down").T * get("ls2")
    return x


def _logits(cfg, weights, tokens, places):
    tokens = torch.as_tensor(np.asarray(tokens).astype(np.int64), device=DEVICE)
    stream = (_decoder_stream if isinstance(cfg, synth.DecoderConfig) else _layered_stream)(cfg, weights, tokens)
    x, w = stream[places], weights["final.norm"].to(F64)
    x = _layer_norm(x, w, cfg.rms_eps) if isinstance(cfg, sandwich_model.SandwichConfig) else _rms(x, w, cfg.rms_eps)
    y = torch.cat([x @ part.to(F64).T for part in weights["head"].split(16384)], dim=-1)
    y = y * getattr(cfg, "logit_scale", 1.0)
    cap = getattr(cfg, "logit_softcap", 0.0)
    return cap * torch.tanh(y / cap) if cap else y


def exact(case, seed):
    if case["kind"] == "attention":
        s = prepare(case, seed)
        groups, dim, per = case["kv_heads"], case["dim"], case["heads"] // case["kv_heads"]
        out = []
        for b in range(case["batch"]):
            order = s["table"][b].long()
            k, v = (t[b].view(-1, 16, groups, dim)[order].reshape(-1, groups, dim)[:case["context"]] for t in (s["keys"], s["values"]))
            q = s["q"][b].to(F64).view(groups, per, dim)
            heads = []
            for g in range(groups):
                p = torch.softmax(q[g] @ k[:, g].to(F64).T * dim ** -0.5, dim=-1)
                heads.append(p @ v[:, g].to(F64))
            out.append(torch.stack(heads).reshape(-1))
        return torch.stack(out)
    cfg = MODELS[case["model"]][0]
    weights = _weights(case["model"])
    prompts = _prompts(case, seed)
    if case["kind"] == "score":
        return _logits(cfg, weights, prompts[0], _places(case))
    follow = _next_token(cfg).cpu().numpy()
    # the tokens that the model is built to say; the logits after a request's last step need those before it
    steps = case["steps"] - 1 if case["kind"] == "generate" else case["steps"]
    logits = []
    for prompt in prompts:
        tokens = list(prompt)
        for _ in range(steps):
            tokens.append(int(follow[tokens[-1]]))
        logits.append(_logits(cfg, weights, tokens, [len(tokens) - 1])[0])
    return {"tokens": None, "logits": logits[0] if case["kind"] == "generate" else torch.stack(logits)}


def tolerance(case):
    """About four times what was measured against exact(): 3.8e-6 for the operator (fp32 sums), 1.8e-3 to 3.2e-3 for
    logits (projection inputs, keys and values rounded to bf16).  Tokens are clear (see above): none may differ beyond
    a stray one."""
    if case["kind"] == "attention":
        return {"rel": 1.5e-5}
    return {"rel": 0.01, "differ": 0.01}
