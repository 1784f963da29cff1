"""The work this framework is measured on: steps of a serving engine on one GPU.

A step is what the engine launches again and again: a prompt step runs the decoder on the new tokens of some requests
(eagerly, keys and values going into the paged cache), a decode step runs it on one token of each running request (one
captured graph).  Models have the published sizes of the framework's presets with fewer layers, random weights, and
cache blocks scattered over the pool as they are after a while of serving.  Two further kinds stand for parts that these
models do not reach: a block-scaled e4m3 expert layer, and sampling with temperature, top-k and top-p.

Two things of trained weights matter to rounding and are kept: the residual stream is large beside what a layer adds to
it, and routers concentrate their choice, so that a near tie between the last chosen expert and the next moves little.
"""
import dataclasses
import math

import torch

from omni_npu_b200 import ops
from omni_npu_b200.attention.metadata import AttentionMetadata, set_forward_context
from omni_npu_b200.compilation.cuda_graph import CUDAGraphRunner
from omni_npu_b200.config import PRESETS
from omni_npu_b200.engine.llm import build_engine_config
from omni_npu_b200.layers.linear import Fp8BlockLinearMethod
from omni_npu_b200.layers.moe import FusedMoE
from omni_npu_b200.models.utils import random_init_
from omni_npu_b200.sample.sampler import Sampler
from omni_npu_b200.worker.worker import Worker

BLOCK = 16
LAYERS = {"llama-3-8b": 8, "qwen3-30b-a3b": 4, "deepseek-v2-lite": 4}
# longest decode context a graph is captured for: prompt + output + slack of the serving benchmark's workloads
MAX_LEN = {"llama-3-8b": 1296, "qwen3-30b-a3b": 4368, "deepseek-v2-lite": 2576}
EMBEDDING_GAIN, GATE_GAIN = 50.0, 3.0


def listed():
    return [
        # one user's chat turn on the dense model: the smallest step, bound by launches and weight streaming
        dict(name="dense_decode_1", kind="decode", model="llama-3-8b", seqs=1, ctx=611, spread=0),
        # the serving benchmark's full decode batch, contexts between prompt length and prompt + output
        dict(name="dense_decode_128", kind="decode", model="llama-3-8b", seqs=128, ctx=1280, spread=256),
        # the serving benchmark's prompt step: a full token budget of whole 1024-token prompts
        dict(name="dense_prompt_8x1024", kind="prompt", model="llama-3-8b", seqs=8, new=1024, spread=0, cached=0),
        # chunks of long prompts: uneven lengths, keys of earlier chunks already in the cache
        dict(name="dense_prompt_chunks", kind="prompt", model="llama-3-8b", seqs=5, new=731, spread=402, cached=3001),
        # a lightly loaded mixture-of-experts server: few rows per expert
        dict(name="moe_decode_16", kind="decode", model="qwen3-30b-a3b", seqs=16, ctx=2111, spread=600),
        # the same server at its full batch and long contexts
        dict(name="moe_decode_128", kind="decode", model="qwen3-30b-a3b", seqs=128, ctx=4352, spread=256),
        # its prompt step: two 4096-token prompts fill the token budget
        dict(name="moe_prompt_2x4096", kind="prompt", model="qwen3-30b-a3b", seqs=2, new=4096, spread=0, cached=0),
        # latent attention, full decode batch
        dict(name="latent_decode_128", kind="decode", model="deepseek-v2-lite", seqs=128, ctx=2560, spread=512),
        # latent attention, prompt step of 2048-token prompts
        dict(name="latent_prompt_4x2048", kind="prompt", model="deepseek-v2-lite", seqs=4, new=2048, spread=0, cached=0),
        # expert layer of a rank's share (32 of 256 experts) of the e4m3 checkpoint: a decode batch and a prompt chunk
        dict(name="fp8_experts_128", kind="experts", tokens=128),
        dict(name="fp8_experts_4096", kind="experts", tokens=4096),
        # a batch whose requests ask for temperature, top-k and top-p in the mixture that clients send
        dict(name="sample_128", kind="sample", rows=128, vocab=128256),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(sorted(LAYERS))
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "experts", "sample"])
    if kind == "decode":
        ctx = log(17, MAX_LEN[model] - 16)
        return dict(kind=kind, model=model, seqs=log(1, 128), ctx=ctx, spread=rng.randint(0, ctx // 2))
    if kind == "prompt":
        seqs = log(1, 8)
        new = log(16, (4096 if model == "qwen3-30b-a3b" else 2048) if seqs <= 2 else 8192 // (seqs + 1))
        cached = rng.choice([0, 0, log(16, 2048)])
        return dict(kind=kind, model=model, seqs=seqs, new=new, spread=rng.randint(0, new // 2), cached=cached)
    if kind == "experts":
        return dict(kind=kind, tokens=log(1, 4096))
    return dict(kind=kind, rows=log(1, 128), vocab=rng.choice([102400, 128256, 129280, 151936]))


# ------------------------------------------------------------------------------------------------------------- inputs
def _lengths(case):
    """(new tokens, cached tokens) of each sequence: between the stated length and ``spread`` less, evenly."""
    n, spread = case["seqs"], case["spread"]
    less = [(i * 7919) % n * spread // n for i in range(n)]
    if case["kind"] == "decode":
        return [1] * n, [max(0, case["ctx"] - 1 - d) for d in less]
    return [case["new"] - d for d in less], [max(0, case["cached"] - 3 * d) for d in less]


def _config(case, seed):
    mc = dataclasses.replace(PRESETS[case["model"]](), num_layers=LAYERS[case["model"]])
    new, cached = _lengths(case)
    longest = max(a + b for a, b in zip(new, cached))
    max_len = MAX_LEN[case["model"]] if case["kind"] == "decode" else longest
    return build_engine_config(mc, max_num_seqs=max(case["seqs"], 1), max_num_batched_tokens=max(sum(new), 256),
                               max_model_len=max_len, block_size=BLOCK, device="cuda", seed=seed,
                               num_gpu_blocks=sum(-(-(a + b) // BLOCK) for a, b in zip(new, cached)))


def _prepare_step(case, seed):
    cfg = _config(case, seed)
    worker = Worker(cfg, local_rank=0, rank=0)
    worker.init_device()
    worker.load_model()
    worker.initialize_from_config(cfg.cache.num_gpu_blocks)
    model, caches = worker.get_model(), worker.model_runner.kv_caches
    dev = worker.device
    g = torch.Generator(device=dev).manual_seed(seed)
    for name, p in model.named_parameters():
        if name.endswith(".gate.weight"):
            p.data.mul_(GATE_GAIN)
        elif name.endswith("embed_tokens.weight"):
            p.data.mul_(EMBEDDING_GAIN)
    # earlier tokens' rows, with the spread that projections of normed rows by these weights have
    # (the latent rows of the compressed cache are normed, their rotated part is not)
    std = 0.02 * math.sqrt(cfg.model.hidden_size)
    for c in caches:
        for t in (c if isinstance(c, (tuple, list)) else (c,)):
            t.normal_(0.0, 1.0 if cfg.model.use_mla else std, generator=g)

    new, cached = _lengths(case)
    lens = [a + b for a, b in zip(new, cached)]
    order = torch.randperm(cfg.cache.num_gpu_blocks, generator=g, device=dev).int()
    decode = case["kind"] == "decode"
    width = -(-(cfg.scheduler.max_model_len if decode else max(lens)) // BLOCK)
    tables = torch.zeros(len(new), width, dtype=torch.int32, device=dev)
    at = 0
    for i, n in enumerate(lens):
        nb = -(-n // BLOCK)
        tables[i, :nb] = order[at: at + nb]
        at += nb
    seq = torch.repeat_interleave(torch.arange(len(new)), torch.tensor(new))
    pos = torch.cat([torch.arange(b, a + b) for a, b in zip(new, cached)]).to(dev)
    seq = seq.to(dev)
    slots = tables[seq, pos // BLOCK].long() * BLOCK + pos % BLOCK
    cu = torch.tensor([0] + new).cumsum(0)
    ids = torch.randint(0, cfg.model.vocab_size, (sum(new),), generator=g, device=dev, dtype=torch.int32)
    md = AttentionMetadata(is_prefill=not decode, num_seqs=len(new), num_tokens=sum(new), max_q_len=max(new),
                           max_seq_len=cfg.scheduler.max_model_len if decode else max(lens), q_len=1 if decode else 0,
                           positions=pos.int(), slot_mapping=slots.int(), block_tables=tables,
                           seq_lens=torch.tensor(lens, dtype=torch.int32, device=dev), cu_q=cu.int().to(dev),
                           num_actual_tokens=sum(new), num_actual_seqs=len(new))
    if not decode:
        md.extra["seq_lens_host"] = lens
    state = dict(case=case, cfg=cfg, model=model, caches=caches, md=md, ids=ids, last=(cu[1:] - 1).to(dev), new=new,
                 lens=lens)
    if decode:
        with torch.inference_mode():
            state["graph"] = CUDAGraphRunner(lambda: _forward(state), dev)
            state["graph"].capture(warmup=2)
    return state


def _prepare_experts(case, seed):
    mc = PRESETS["deepseek-v3.2"]()
    dev = torch.device("cuda", 0)
    # process groups and buffers of a one-GPU engine
    worker = Worker(build_engine_config(PRESETS["tiny-llama"](), device="cuda", max_num_seqs=1, num_gpu_blocks=16))
    worker.init_device()
    layer = FusedMoE(32, mc.num_experts_per_tok, mc.hidden_size, mc.moe_intermediate_size, mc.dtype, dev,
                     mc.scoring_func, mc.norm_topk_prob, mc.routed_scaling_factor, mc.n_group, mc.topk_group,
                     mc.router_bias, mc.num_shared_experts, enable_expert_parallel=False, prefix="mlp",
                     max_tokens=case["tokens"], quant="fp8", shared_quant_factory=Fp8BlockLinearMethod)
    random_init_(layer, seed=seed)
    g = torch.Generator(device=dev).manual_seed(seed)
    for name, p in layer.named_parameters():
        if "scale" in name:      # of blocks whose largest value is three to four deviations of 0.02 wide weights
            p.data.uniform_(0.5e-3, 0.75e-3, generator=g)
        elif name.endswith("correction_bias"):
            p.data.normal_(0.0, 0.05, generator=g)
    for m in layer.modules():
        hook = getattr(m, "process_weights_after_loading", None)
        if callable(hook):
            hook()
    layer.init_ep_buffers()
    x = torch.randn(case["tokens"], mc.hidden_size, generator=g, device=dev, dtype=torch.bfloat16)
    state = dict(case=case, cfg=mc, layer=layer, x=x)
    if case["tokens"] <= 256:    # decode batches run as a captured graph
        with torch.inference_mode():
            state["graph"] = CUDAGraphRunner(lambda: layer(x), dev)
            state["graph"].capture(warmup=2)
    return state


def _prepare_sample(case, seed):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    n = case["rows"]
    # logits of a language model: a broad bulk and some tokens well above it
    logits = torch.randn(n, case["vocab"], generator=g, device=dev) * 2.0
    logits += (torch.rand(n, case["vocab"], generator=g, device=dev) < 1e-3) * 6.0
    row = torch.arange(n, device=dev)
    # a quarter each: greedy, temperature alone, with top-p, with top-k and top-p
    temperature = torch.where(row % 4 == 0, 0.0, 0.6 + 0.1 * (row % 5)).float()
    top_p = torch.where(row % 4 >= 2, 0.95 - 0.05 * (row % 3), 1.0).float()
    top_k = torch.where(row % 4 == 3, 20 + 10 * (row % 4), 0).int()
    seeds = torch.randint(0, 1 << 30, (n,), generator=g, device=dev)
    return dict(case=case, sampler=Sampler(None, dev), args=(logits, temperature, top_k, top_p, seeds))


def prepare(case, seed):
    return {"decode": _prepare_step, "prompt": _prepare_step, "experts": _prepare_experts,
            "sample": _prepare_sample}[case["kind"]](case, seed)


# --------------------------------------------------------------------------------------------------------------- pass
def _forward(state):
    with set_forward_context(state["md"], state["caches"], state["cfg"]):
        hidden = state["model"](state["ids"], state["md"].positions)
        if state["md"].is_prefill:
            hidden = hidden.index_select(0, state["last"])
        return state["model"].compute_logits(hidden)


@torch.inference_mode()
def run(state):
    kind = state["case"]["kind"]
    if kind == "sample":
        return {"tokens": state["sampler"](*state["args"])}
    if kind == "experts":
        return {"y": state["graph"].replay() if "graph" in state else state["layer"](state["x"])}
    logits = state["graph"].replay() if "graph" in state else _forward(state)
    return {"logits": logits, "caches": state["caches"]}


# ------------------------------------------------------------------------------------------------- what a pass amounts to
def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["rows"] * case["vocab"], "flops": 5.0 * case["rows"] * case["vocab"]}
    if case["kind"] == "experts":
        mc, t = PRESETS["deepseek-v3.2"](), case["tokens"]
        one = 3 * mc.hidden_size * mc.moe_intermediate_size
        live = 32 * (1 - (1 - mc.num_experts_per_tok / 32) ** t)
        return {"bytes": (live + 1) * one + 32 * mc.hidden_size * 2 + 4.0 * t * mc.hidden_size,
                "flops": 2.0 * t * (mc.num_experts_per_tok + 1) * one}
    mc = PRESETS[case["model"]]()
    new, cached = _lengths(case)
    layers, tokens, h = LAYERS[case["model"]], sum(new), mc.hidden_size
    pairs = sum(a * b + a * (a + 1) / 2 for a, b in zip(new, cached))       # (query, key) pairs that are not masked
    if mc.use_mla:
        qk, rope, v, n, lat = mc.qk_nope_head_dim, mc.qk_rope_head_dim, mc.v_head_dim, mc.num_heads, mc.kv_lora_rank
        attn = h * (n * (qk + rope) + lat + rope) + lat * n * (qk + v) + h * n * v
        row = lat + rope
        pair = 2.0 * n * (qk + rope + v) if case["kind"] == "prompt" else 2.0 * n * (2 * lat + rope)
    else:
        attn = h * mc.head_dim * 2 * (mc.num_heads + mc.num_kv_heads)
        row = 2 * mc.num_kv_heads * mc.head_dim
        pair = 4.0 * mc.num_heads * mc.head_dim
    read = used = 0.0                                                     # parameters read, and used per token
    for i in range(layers):
        if mc.layer_is_moe(i):
            one = 3 * h * mc.moe_intermediate_size
            live = mc.num_experts * (1 - (1 - mc.num_experts_per_tok / mc.num_experts) ** tokens)
            read += attn + h * mc.num_experts + one * (live + mc.num_shared_experts)
            used += attn + h * mc.num_experts + one * (mc.num_experts_per_tok + mc.num_shared_experts)
        else:
            read += attn + 3 * h * mc.intermediate_size
            used += attn + 3 * h * mc.intermediate_size
    head = mc.vocab_size * h
    seqs = case["seqs"]
    return {"bytes": 2.0 * (read + head + h * tokens + layers * row * (sum(cached) + tokens)) + 4.0 * seqs * mc.vocab_size,
            "flops": 2.0 * (tokens * used + seqs * head) + layers * pairs * pair}


def tolerance(case):
    if case["kind"] == "sample":       # a threshold that sums are compared with may fall between other tokens
        return {"differ": 0.01}
    if case["kind"] == "experts":      # a value that rounds to another e4m3 number moves by up to an eighth
        return {"rel": 0.02, "max": 0.5}
    return {"rel": 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _halves(x, pos, base, split):
    """Rotation of the last axis by position; ``split``: pairs are the two halves, else neighbours."""
    d = x.shape[-1]
    a = pos.double()[:, None] / base ** (torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    c, s = a.cos(), a.sin()
    while c.dim() < x.dim():
        c, s = c.unsqueeze(1), s.unsqueeze(1)
    u, v = (x[..., : d // 2], x[..., d // 2:]) if split else (x[..., 0::2], x[..., 1::2])
    p, q = u * c - v * s, v * c + u * s
    return torch.cat([p, q], -1) if split else torch.stack([p, q], -1).flatten(-2)


def _gate_up(w):
    """Rows of a stacked weight that lie in alternating groups of eight, as the two matrices."""
    r = torch.arange(w.shape[0], device=w.device)
    return w[(r // 8) % 2 == 0].double(), w[(r // 8) % 2 == 1].double()


def _mlp(x, gate, up, down):
    return (torch.nn.functional.silu(x @ gate.T) * (x @ up.T)) @ down.double().T


def _attend(q, k, v, first, scale):
    """q [n, heads, d], k / v [m, kv heads, .]; query i sees keys up to first + i."""
    n, heads, _ = q.shape
    group = heads // k.shape[1]
    out = []
    for h in range(0, heads, group):
        s = torch.einsum("nhd,md->hnm", q[:, h: h + group], k[:, h // group]) * scale
        if n > 1:
            hidden = torch.arange(k.shape[0], device=q.device)[None] > first + torch.arange(n, device=q.device)[:, None]
            s = s.masked_fill(hidden, -math.inf)
        out.append(torch.einsum("hnm,md->nhd", s.softmax(-1), v[:, h // group]))
    return torch.cat(out, 1)


def _choose(scores, k, renormalize):
    w, ids = scores.topk(k, -1)
    return (w / w.sum(-1, keepdim=True) if renormalize else w), ids


def _experts(x, w, ids, count, expert):
    out = torch.zeros_like(x)
    for e in range(count):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            out.index_add_(0, t, _mlp(x[t], *expert(e)) * w[t, j, None])
    return out


def _exact_step(state):
    mc, md, model = state["cfg"].model, state["md"], state["model"]
    pos, slot = md.positions.long(), md.slot_mapping.long()
    x = model.model.embed_tokens.weight[state["ids"].long()].double()
    cu = [0]
    for n in state["new"]:
        cu.append(cu[-1] + n)
    caches = []
    for i, layer in enumerate(model.model.layers):
        at, h = layer.self_attn, _norm(x, layer.input_layernorm.weight, mc.rms_norm_eps)
        own = state["caches"][i]
        t = x.shape[0]
        if mc.use_mla:
            n, nope, rope, lat = mc.num_heads, mc.qk_nope_head_dim, mc.qk_rope_head_dim, mc.kv_lora_rank
            q = (h @ at.q_proj.weight.double().T).view(t, n, nope + rope)
            q = torch.cat([q[..., :nope], _halves(q[..., nope:], pos, mc.rope_theta, False)], -1)
            kv = h @ at.kv_a_proj_with_mqa.weight.double().T
            row = torch.cat([_norm(kv[:, :lat], at.kv_a_layernorm.weight, mc.rms_norm_eps),
                             _halves(kv[:, lat:], pos, mc.rope_theta, False)], -1)
            cache = own.double()
            cache.view(-1, lat + rope)[slot] = row
            caches.append(cache)
            w_kv = at.kv_b_proj.weight.double()
        else:
            d, n, nk = mc.head_dim, mc.num_heads, mc.num_kv_heads
            qkv = (h @ at.qkv_proj.weight.double().T).view(t, n + 2 * nk, d)
            q, k, v = qkv[:, :n], qkv[:, n: n + nk], qkv[:, n + nk:]
            if mc.qk_norm:
                q, k = _norm(q, at.q_norm.weight, mc.rms_norm_eps), _norm(k, at.k_norm.weight, mc.rms_norm_eps)
            q, k = (_halves(z, pos, mc.rope_theta, True) for z in (q, k))
            cache = [z.double() for z in own]                              # [blocks, kv heads, tokens, d]
            for z, rows in zip(cache, (k, v)):
                z[slot // BLOCK, :, slot % BLOCK] = rows
            caches.append(tuple(cache))
        outs = []
        for s, length in enumerate(state["lens"]):
            blocks = md.block_tables[s, : -(-length // BLOCK)].long()
            qs, first = q[cu[s]: cu[s + 1]], length - state["new"][s]
            if mc.use_mla:
                rows = cache[blocks].flatten(0, 1)[:length]
                kv = (rows[:, :lat] @ w_kv.T).view(length, n, nope + mc.v_head_dim)
                ks = torch.cat([kv[..., :nope], rows[:, None, lat:].expand(-1, n, -1)], -1)
                outs.append(_attend(qs, ks, kv[..., nope:], first, (nope + rope) ** -0.5))
            else:
                ks, vs = (z[blocks].transpose(1, 2).flatten(0, 1)[:length] for z in cache)
                outs.append(_attend(qs, ks, vs, first, d ** -0.5))
        x = x + torch.cat(outs).flatten(1) @ at.o_proj.weight.double().T
        h = _norm(x, layer.post_attention_layernorm.weight, mc.rms_norm_eps)
        mlp = layer.mlp
        if mc.layer_is_moe(i):
            scores = (h @ mlp.gate.weight.double().T).softmax(-1)
            w, ids = _choose(scores, mc.num_experts_per_tok, mc.norm_topk_prob)
            x = x + _experts(h, w, ids, mc.num_experts, lambda e: (*_gate_up(mlp.w13[e]), mlp.w2[e]))
            mlp = mlp.shared_experts
        if mlp is not None:
            x = x + _mlp(h, *_gate_up(mlp.gate_up_proj.weight), mlp.down_proj.weight)
    x = _norm(x[state["last"]], model.model.norm.weight, mc.rms_norm_eps)
    return {"logits": x @ model.lm_head.weight[: mc.vocab_size].double().T, "caches": caches}


def _exact_experts(state):
    mc, layer, x = state["cfg"], state["layer"], state["x"].double()

    def full(w, scale):
        s = scale.double().repeat_interleave(128, 0).repeat_interleave(128, 1)
        return w.float().double() * s[: w.shape[0], : w.shape[1]]

    def expert(e):
        gate, up = _gate_up(layer.w13[e].float())
        half = layer.w13_scale[e].shape[0] // 2
        return full(gate, layer.w13_scale[e][:half]), full(up, layer.w13_scale[e][half:]), full(layer.w2[e], layer.w2_scale[e])

    score = (x @ layer.gate.weight.double().T).sigmoid()
    biased = score + layer.e_score_correction_bias.double()
    groups = biased.view(len(x), mc.n_group, -1).topk(2, -1).values.sum(-1).topk(mc.topk_group, -1).indices
    keep = torch.zeros(len(x), mc.n_group, dtype=torch.bool, device=x.device).scatter_(1, groups, True)
    biased = biased.masked_fill(~keep.repeat_interleave(32 // mc.n_group, 1), -math.inf)
    ids = biased.topk(mc.num_experts_per_tok, -1).indices
    w = score.gather(1, ids)
    y = _experts(x, w / w.sum(-1, keepdim=True) * mc.routed_scaling_factor, ids, 32, expert)
    shared = layer.shared_experts
    both = full(shared.gate_up_proj.weight, shared.gate_up_proj.weight_scale_inv)
    gate, up = both.chunk(2)
    return {"y": y + _mlp(x, gate, up, full(shared.down_proj.weight, shared.down_proj.weight_scale_inv))}


@torch.inference_mode()
def exact(case, seed):
    if case["kind"] == "sample":       # the draw is the framework's own: there is no such value
        return None
    state = prepare(case, seed)
    return _exact_experts(state) if case["kind"] == "experts" else _exact_step(state)
