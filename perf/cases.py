"""Generation workloads whose speed is followed: what they are, how one pass runs, what it should return.

A pass is one ``LLM.generate`` over a batch of new requests: the prompts are prefilled, ``new`` tokens are
generated for each, and the logits of the last step are collected for up to ``SCORED`` of the requests (what a
program that scores its answers does with ``score_positions`` / ``take_scores``). Models are this package's named
shapes with random weights; those whose bf16 weights would not fit a GPU three times over run with fewer of their
(equal) layers. Engines are set up as the benchmark of this repository sets them up: 8192 tokens a step at most, CUDA
graphs, asynchronous scheduling; prefix caching is off, as every pass stands for new prompts.

Weights are drawn so that the model is as sure of its next token as a trained one is: an untied lm_head whose row
``follow[t]`` looks along the embedding of ``t``, sublayers whose sum is shorter than the embedding, attention scores
and router logits of a spread of about two, slow decays in the recurrent layers.
"""
from __future__ import annotations

import dataclasses
import gc
import math
import random

import torch

from vllm_cpp_b200.config import EngineArgs, synthetic_config
from vllm_cpp_b200.engine import LLM, SamplingParams

SCORED = 8
BLOCK = 32                # tokens of a KV block
STEP_TOKENS = 8192        # most tokens of an engine step

# model -> layers that run (None: all of them)
MODELS = {"qwen3-0.6b": None, "llama-3.1-8b": None, "llama-3.1-8b+fp8": None, "qwen3-30b-a3b": 12,
          "qwen3.6-27b": 8, "deepseek-v2-lite": 12}


def _case(model, requests, low, high, new, sampled=False):
    return {"model": model, "requests": requests, "shortest": low, "longest": high, "new": new, "sampled": sampled}


def listed():
    c = {
        # a short question to a small model: launches and latency
        "small, one request": _case("qwen3-0.6b", 1, 40, 40, 24),
        # many users of a small model, drawn with temperature, top-k and top-p: the sampler's path
        "small, sampled": _case("qwen3-0.6b", 40, 30, 400, 16, True),
        # one user in a chat with the main dense model: time to first token, then single-row decode steps
        "dense, one request": _case("llama-3.1-8b", 1, 700, 700, 16),
        # a lightly loaded server, ragged prompts
        "dense, few requests": _case("llama-3.1-8b", 13, 60, 500, 24),
        # a fully loaded server: prefill in several steps mixed with decodes, then wide decode steps
        "dense, many requests": _case("llama-3.1-8b", 120, 100, 450, 20),
        # a document read once, a short answer: prefill attention and the widest products
        "dense, long prompt": _case("llama-3.1-8b", 1, 15501, 15501, 4),
        # the same dense model with fp8 weights and activations
        "fp8, some requests": _case("llama-3.1-8b+fp8", 32, 100, 600, 16),
        # routed experts: few rows (single experts' weights), and many
        "experts, few requests": _case("qwen3-30b-a3b", 3, 200, 900, 24),
        "experts, many requests": _case("qwen3-30b-a3b", 64, 100, 700, 16),
        # recurrent and attention layers with NVFP4 weights, as that shape is configured here
        "hybrid, some requests": _case("qwen3.6-27b", 9, 100, 1800, 16),
        # latent attention, shared and routed experts
        "latent, some requests": _case("deepseek-v2-lite", 21, 100, 1300, 16),
    }
    return [{"name": k, **v} for k, v in c.items()]


# most requests and most prompt tokens of a drawn case, about what the largest listed case costs or less
LIMITS = {"qwen3-0.6b": (160, 24000), "llama-3.1-8b": (120, 16000), "llama-3.1-8b+fp8": (120, 20000),
          "qwen3-30b-a3b": (120, 24000), "qwen3.6-27b": (32, 16000), "deepseek-v2-lite": (64, 20000)}


def draw(rng):
    """One more case: any model, from one request to many, prompts from a few tokens to many thousands."""
    model = rng.choice(sorted(MODELS))
    most, tokens = LIMITS[model]

    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    requests = spread(1, most)
    high = spread(8, max(9, tokens // requests))
    return _case(model, requests, max(1, min(high, spread(max(1, high // 8), high))), high, spread(1, 32),
                 rng.random() < 0.2)


# ------------------------------------------------------------------------------------------- inputs
def _config(case):
    cfg = synthetic_config(case["model"])
    layers = MODELS[case["model"]]
    if layers is not None:
        cfg.num_layers = layers
        if cfg.layer_types:
            cfg.layer_types = cfg.layer_types[:layers]
    return dataclasses.replace(cfg, tie_word_embeddings=False)


def _lengths(case):
    """Prompt lengths: the case's own, whatever the seed."""
    r = random.Random(case["requests"] * 1000003 + case["longest"] * 1009 + case["shortest"])
    n = [r.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]
    n[-1] = case["longest"]
    return n


def _scored(case):
    """The requests whose last logits are collected, spread over the batch."""
    n = case["requests"]
    return list(range(n)) if n <= SCORED else [i * (n - 1) // (SCORED - 1) for i in range(SCORED)]


def _prompts(case, seed):
    r = random.Random(seed)
    vocab = synthetic_config(case["model"]).vocab_size
    return [[r.randrange(vocab) for _ in range(n)] for n in _lengths(case)]


def _normal(shape, std, seed, where):
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + where)
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)


def _follow(cfg, seed):
    """follow[t]: the token that the model expects after t."""
    return torch.randperm(cfg.vocab_size, generator=torch.Generator(device="cuda").manual_seed(seed * 7919 + 1),
                          device="cuda")


def _embedding(cfg, seed):
    return _normal((cfg.vocab_size, cfg.hidden_size), 1.0, seed, 2)


def _head(cfg, seed):
    head = torch.empty((cfg.vocab_size, cfg.hidden_size), dtype=torch.bfloat16, device="cuda")
    head[_follow(cfg, seed)] = _embedding(cfg, seed) * cfg.hidden_size ** -0.5
    return head


def _share(cfg):
    """Length of the sublayers' sum against the embedding's. What rounding leaves of it is in every difference of two
    correct results: 8-bit activations leave ten times more than bf16 ones."""
    return 0.2 if cfg.quant == "fp8" else 0.5


def _layer(cfg, seed, l):
    """HF-named bf16 tensors of one decoder layer."""
    c, H, D = cfg, cfg.hidden_size, cfg.head_dim
    at = [16 + 64 * l]
    part = _share(c) * (2 * c.num_layers) ** -0.5          # what one sublayer adds, against an embedding of one

    def w(*shape, gain=1.0):
        at[0] += 1
        return _normal(shape, gain * shape[-1] ** -0.5, seed, at[0])

    def flat(n, value):
        return torch.full((n,), value - (1.0 if c.gemma_norm else 0.0), dtype=torch.bfloat16, device="cuda")

    t = {"input_layernorm.weight": flat(H, 1.0), "post_attention_layernorm.weight": flat(H, 1.0)}
    if c.is_hybrid and c.layer_types[l] == "linear_attention":
        hk, hv = c.linear_num_key_heads, c.linear_num_value_heads
        g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 16 + 64 * l)
        u = torch.rand((2, hv), generator=g, device="cuda")
        dt = torch.exp(math.log(1e-3) + u[0] * math.log(100.0))
        t.update({"linear_attn.in_proj_qkv.weight": w(2 * hk * 128 + hv * 128, H), "linear_attn.in_proj_z.weight": w(hv * 128, H),
                  "linear_attn.in_proj_b.weight": w(hv, H), "linear_attn.in_proj_a.weight": w(hv, H),
                  "linear_attn.conv1d.weight": w(2 * hk * 128 + hv * 128, 1, 4),
                  "linear_attn.A_log": torch.log(1 + 15 * u[1]), "linear_attn.dt_bias": torch.log(torch.expm1(dt)),
                  "linear_attn.norm.weight": torch.ones(128, dtype=torch.bfloat16, device="cuda"),
                  "linear_attn.out_proj.weight": w(H, hv * 128, gain=1.6 * part)})
    elif c.is_mla:
        heads, nope, rot, rank = c.num_heads, c.qk_nope_head_dim, c.qk_rope_head_dim, c.kv_lora_rank
        t.update({"self_attn.q_proj.weight": w(heads * (nope + rot), H, gain=1.3),
                  "self_attn.kv_a_proj_with_mqa.weight": w(rank + rot, H),
                  "self_attn.kv_a_layernorm.weight": flat(rank, 1.0),
                  "self_attn.kv_b_proj.weight": w(heads * (nope + c.v_head_dim), rank),
                  "self_attn.o_proj.weight": w(H, heads * c.v_head_dim, gain=4 * part)})
    else:
        gain = 1.0 if c.qk_norm else 1.4
        t.update({"self_attn.q_proj.weight": w(c.num_heads * D * (2 if c.attn_output_gate else 1), H, gain=gain),
                  "self_attn.k_proj.weight": w(c.num_kv_heads * D, H, gain=gain),
                  "self_attn.v_proj.weight": w(c.num_kv_heads * D, H),
                  "self_attn.o_proj.weight": w(H, c.num_heads * D, gain=4 * part)})
        if c.qk_norm:
            t.update({"self_attn.q_norm.weight": flat(D, 1.4), "self_attn.k_norm.weight": flat(D, 1.4)})
    if c.is_moe and l >= c.first_k_dense_replace:
        n, ff = c.num_experts, c.moe_intermediate_size
        t.update({"mlp.gate.weight": w(n, H, gain=2.0), "mlp.experts.gate_proj.weight": w(n, ff, H),
                  "mlp.experts.up_proj.weight": w(n, ff, H), "mlp.experts.down_proj.weight": w(n, H, ff, gain=2.0 * part)})
        if c.num_shared_experts:
            ff *= c.num_shared_experts
            t.update({"mlp.shared_experts.gate_proj.weight": w(ff, H), "mlp.shared_experts.up_proj.weight": w(ff, H),
                      "mlp.shared_experts.down_proj.weight": w(H, ff, gain=1.6 * part)})
    else:
        ff = c.intermediate_size
        t.update({"mlp.gate_proj.weight": w(ff, H), "mlp.up_proj.weight": w(ff, H),
                  "mlp.down_proj.weight": w(H, ff, gain=1.6 * part)})
    return t


def _checkpoint(cfg, seed):
    yield "model.embed_tokens.weight", _embedding(cfg, seed)
    for l in range(cfg.num_layers):
        for k, v in _layer(cfg, seed, l).items():
            yield f"model.layers.{l}.{k}", v
    yield "model.norm.weight", torch.full((cfg.hidden_size,), 0.0 if cfg.gemma_norm else 1.0, dtype=torch.bfloat16, device="cuda")
    yield "lm_head.weight", _head(cfg, seed)


class _Checkpoint(LLM):
    """An engine over the drawn checkpoint: its tensors are loaded where a model without files takes random weights."""

    def __init__(self, args, checkpoint):
        from vllm_cpp_b200.models import registry
        cls = registry.resolve(args.model_config.architecture)[1]
        own = cls.init_random
        cls.init_random = lambda model, seed=0, std=0.02: model.load_weights(checkpoint)
        try:
            super().__init__(args)
        finally:
            cls.init_random = own


def prepare(case, seed):
    """The engine with its weights loaded, and the batch's prompts."""
    gc.collect()          # an engine that was dropped gives its memory back
    cfg, new = _config(case), case["new"]
    lengths, requests = _lengths(case), case["requests"]
    llm = _Checkpoint(EngineArgs(model_config=cfg, block_size=BLOCK, num_blocks=16 + sum(-(-(n + new) // BLOCK) + 1 for n in lengths),
                                 max_model_len=max(lengths) + new + 8, max_num_seqs=requests, max_num_batched_tokens=STEP_TOKENS,
                                 enable_prefix_caching=False, async_scheduling=True, max_score_rows=SCORED),
                      _checkpoint(cfg, seed))
    params = SamplingParams(max_tokens=new, ignore_eos=True, **(
        {"temperature": 0.8, "top_k": 50, "top_p": 0.95, "seed": 1234 + seed % 1000} if case["sampled"] else {"temperature": 0.0}))
    return {"llm": llm, "prompts": _prompts(case, seed), "params": params, "scored": _scored(case), "new": new, "batch": 0}


def run(state):
    """Generates for the whole batch. -> token ids [requests, new], last logits [scored, vocabulary]."""
    llm, prompts = state["llm"], state["prompts"]
    state["batch"] += 1
    names = [f"{state['batch']}.{i}" for i in range(len(prompts))]
    for i in state["scored"]:
        llm.score_positions(names[i], [len(prompts[i]) + state["new"] - 2])
    for name, p in zip(names, prompts):
        llm.add_request(p, state["params"], request_id=name)
    tokens = {}
    while llm.has_unfinished_requests():
        for out in llm.step():
            if out.finished:
                tokens[out.request_id] = out.outputs[0].token_ids
    scores = llm.take_scores()
    return {"tokens": torch.tensor([tokens[n] for n in names]),
            "logits": torch.stack([scores[names[i]][0][1] for i in state["scored"]])}


# ------------------------------------------------------------------------------------------- cost
def work(case):
    """Every step of a request reads the weights that it needs and the keys and values before it; the prompts need
    their products and causal attention once. Weights are counted once for the prefill and once for every further
    token of the batch."""
    c, lengths, new, requests = _config(case), _lengths(case), case["new"], case["requests"]
    H, each = c.hidden_size, {"llama-3.1-8b+fp8": 1.0, "qwen3.6-27b": 0.5625}.get(case["model"], 2.0)
    ff = 3 * H * c.moe_intermediate_size if c.is_moe else 0
    tokens, last = sum(lengths), new - 1
    rows = [requests] * last
    pairs = sum(n * (n + 1) // 2 + sum(n + j for j in range(1, new)) for n in lengths)
    held = sum(sum(n + j for j in range(1, new)) for n in lengths)      # cached positions that decode steps read
    every = flops = moved = 0.0
    for l in range(c.num_layers):
        if c.is_hybrid and c.layer_types[l] == "linear_attention":
            hk, hv = c.linear_num_key_heads, c.linear_num_value_heads
            mix = H * (2 * hk * 128 + 3 * hv * 128 + 2 * hv)
            flops += 2 * 3 * hv * 128 * 128 * (tokens + requests * last)
            moved += 2 * hv * 128 * 128 * 4 * requests * last
        elif c.is_mla:
            nope, rot, rank, v = c.qk_nope_head_dim, c.qk_rope_head_dim, c.kv_lora_rank, c.v_head_dim
            mix = H * (c.num_heads * (nope + rot) + rank + rot + c.num_heads * v) + rank * c.num_heads * (nope + v)
            flops += 2 * c.num_heads * (nope + rot + v) * pairs
            moved += 2 * (rank + rot) * (held + tokens)
        else:
            mix = H * c.head_dim * (c.num_heads * (3 if c.attn_output_gate else 2) + 2 * c.num_kv_heads)
            flops += 4 * c.num_heads * c.head_dim * pairs
            moved += 4 * c.num_kv_heads * c.head_dim * (held + tokens)
        if c.is_moe and l >= c.first_k_dense_replace:
            k, n, s = c.num_experts_per_tok, c.num_experts, c.num_shared_experts
            every += 2 * (mix + s * ff + n * H)
            flops += 2 * (mix + (k + s) * ff + n * H) * (tokens + requests * last)
            moved += 2 * ff * sum(n * (1 - (1 - k / n) ** r) for r in [tokens] + rows)
        else:
            every += each * (mix + 3 * H * c.intermediate_size)
            flops += 2 * (mix + 3 * H * c.intermediate_size) * (tokens + requests * last)
    flops += 2 * H * c.vocab_size * requests * new
    return {"bytes": moved + (every + 2 * H * c.vocab_size) * new, "flops": flops}


def tolerance(case):
    """16-bit streams through 8 to 32 layers. The same prompts in steps of other sizes, so by other kernels and in another
    order of the sums, gave logits that differ by 0.007 (hybrid) to 0.016 (dense) and 0.019 (fp8), about as much as each
    of them differs from 64 bits, and 0.1 at most at one value. The tokens are far from ties."""
    return {"rel": 0.03, "max": 0.3}


# ------------------------------------------------------------------------------------------- 64 bits
def _grid4(w):
    """The NVFP4 values of a weight: e2m1 times an e4m3 scale for every 16 and one 32-bit scale."""
    x = w.float()
    g = x.abs().max() / (448.0 * 6.0)
    b = x.reshape(x.shape[0], -1, 16)
    s = ((b.abs().amax(-1) / 6.0 / g).to(torch.float8_e4m3fn).float() * g)[..., None]
    q = b / s.clamp_min(1e-30)
    grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device=w.device)
    near = grid[torch.bucketize(q.abs(), (grid[1:] + grid[:-1]) / 2)]
    return (torch.copysign(near, q).double() * s.double()).reshape(w.shape)


def _grid8(w):
    """The e4m3 values of a weight with one scale a row."""
    s = (w.float().abs().amax(1, keepdim=True) / 448.0)
    return (w.float() / s).to(torch.float8_e4m3fn).double() * s.double()


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _frequencies(cfg):
    """Inverse frequencies of the rotated dimensions and the factor on the attention scores."""
    r = cfg.rope
    dims = r.rotary_dim or cfg.head_dim
    inv = r.theta ** (-torch.arange(0, dims, 2, dtype=torch.float64) / dims)
    if r.scaling_type == "llama3":
        turns = r.original_max_position * inv / (2 * math.pi)
        keep = ((turns - r.low_freq_factor) / (r.high_freq_factor - r.low_freq_factor)).clamp(0, 1)
        return inv * (keep + (1 - keep) / r.factor), 1.0
    if r.scaling_type == "deepseek_yarn":
        def dim(turns):
            return dims * math.log(r.original_max_position / (turns * 2 * math.pi)) / (2 * math.log(r.theta))
        low, high = max(math.floor(dim(r.beta_fast)), 0), min(math.ceil(dim(r.beta_slow)), dims - 1)
        slow = ((torch.arange(dims // 2, dtype=torch.float64) - low) / max(high - low, 1e-3)).clamp(0, 1)
        return inv * (1 - slow + slow / r.factor), (0.1 * r.mscale_all_dim * math.log(r.factor) + 1.0) ** 2
    return inv, 1.0


def _rotate(x, inv, neox):
    """x [tokens, heads, dims] at positions 0.."""
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * inv.to(x.device)
    cos, sin, n = a.cos()[:, None], a.sin()[:, None], 2 * inv.numel()
    y = x.clone()
    p, q = (x[..., : n // 2], x[..., n // 2: n]) if neox else (x[..., 0:n:2], x[..., 1:n:2])
    first, second = p * cos - q * sin, q * cos + p * sin
    if neox:
        y[..., : n // 2], y[..., n // 2: n] = first, second
    else:
        y[..., 0:n:2], y[..., 1:n:2] = first, second
    return y


def _attend(q, k, v, scale):
    """Causal attention of [tokens, heads, dims], query heads in groups over the key heads."""
    n, heads, rep = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    out = torch.empty(n, heads, v.shape[2], dtype=torch.float64, device=q.device)
    step = max(64, min(n, (1 << 27) // n))
    for h in range(heads):
        kh, vh = k[:, h // rep], v[:, h // rep]
        for i in range(0, n, step):
            s = q[i:i + step, h] @ kh[: i + step].t() * scale
            rows = torch.arange(i, min(i + step, n), device=q.device)[:, None]
            s.masked_fill_(torch.arange(s.shape[1], device=q.device)[None] > rows, -math.inf)
            out[i:i + step, h] = torch.softmax(s, -1) @ vh[: i + step]
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _unit(x, t, prefix):
    return (_silu(x @ t[prefix + "gate_proj.weight"].t()) * (x @ t[prefix + "up_proj.weight"].t())) @ t[prefix + "down_proj.weight"].t()


def _experts(cfg, x, t):
    p = torch.softmax(x @ t["mlp.gate.weight"].double().t(), -1)
    w, ids = p.topk(cfg.num_experts_per_tok, -1)
    if cfg.norm_topk_prob:
        w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        at, k = (ids == e).nonzero(as_tuple=True)
        if at.numel():
            one = {n: t[f"mlp.experts.{n}"][e].double() for n in ("gate_proj.weight", "up_proj.weight", "down_proj.weight")}
            out.index_add_(0, at, _unit(x[at], one, "") * w[at, k, None])
    if cfg.num_shared_experts:
        out += _unit(x, {k: v.double() for k, v in t.items() if "shared" in k}, "mlp.shared_experts.")
    return out


def _recurrent(cfg, x, t, spans):
    """Gated delta rule over every sequence, token by token; sequences side by side, the short ones padded."""
    hk, hv, longest = cfg.linear_num_key_heads, cfg.linear_num_value_heads, max(e - b for b, e in spans)
    mixed = x @ t["linear_attn.in_proj_qkv.weight"].t()
    conv, seq = t["linear_attn.conv1d.weight"][:, 0].double(), torch.zeros(len(spans), longest, mixed.shape[1], dtype=torch.float64, device=x.device)
    gates = torch.zeros(2, len(spans), longest, hv, dtype=torch.float64, device=x.device)
    b, a = torch.sigmoid(x @ t["linear_attn.in_proj_b.weight"].t()), x @ t["linear_attn.in_proj_a.weight"].t()
    decay = torch.exp(-torch.exp(t["linear_attn.A_log"].double()) * torch.nn.functional.softplus(a + t["linear_attn.dt_bias"].double()))
    for i, (lo, hi) in enumerate(spans):
        past = torch.cat([torch.zeros(3, mixed.shape[1], dtype=torch.float64, device=x.device), mixed[lo:hi]])
        seq[i, : hi - lo] = _silu(sum(past[j: j + hi - lo] * conv[:, j] for j in range(4)))
        gates[0, i, : hi - lo], gates[1, i, : hi - lo] = b[lo:hi], decay[lo:hi]
    q, k, v = seq.split([hk * 128, hk * 128, hv * 128], -1)

    def heads(y):
        y = y.reshape(len(spans), longest, hk, 128)
        return (y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(hv // hk, 2)

    q, k, v = heads(q) * 128 ** -0.5, heads(k), v.reshape(len(spans), longest, hv, 128)
    state, out = torch.zeros(len(spans), hv, 128, 128, dtype=torch.float64, device=x.device), torch.empty_like(v)
    for j in range(longest):
        state *= gates[1, :, j, :, None, None]
        gap = (v[:, j] - (state @ k[:, j, :, :, None])[..., 0]) * gates[0, :, j, :, None]
        state += gap[..., None] * k[:, j, :, None]
        out[:, j] = (state @ q[:, j, :, :, None])[..., 0]
    core = torch.cat([out[i, : hi - lo] for i, (lo, hi) in enumerate(spans)])
    z = (x @ t["linear_attn.in_proj_z.weight"].t()).reshape(-1, hv, 128)
    core = _rms(core, t["linear_attn.norm.weight"].double(), cfg.rms_norm_eps) * _silu(z)
    return core.reshape(-1, hv * 128) @ t["linear_attn.out_proj.weight"].t()


def _attention(cfg, x, t, spans, inv, factor):
    c, n, D = cfg, x.shape[0], cfg.head_dim
    one = 1.0 if c.gemma_norm else 0.0
    gate = None
    q, w_o = x @ t["self_attn.q_proj.weight"].t(), t["self_attn.o_proj.weight"]
    if c.is_mla:
        nope, rank = c.qk_nope_head_dim, c.kv_lora_rank
        q = q.reshape(n, c.num_heads, -1)
        a = x @ t["self_attn.kv_a_proj_with_mqa.weight"].t()
        up = (_rms(a[:, :rank], t["self_attn.kv_a_layernorm.weight"].double(), c.rms_norm_eps) @ t["self_attn.kv_b_proj.weight"].t())
        up, own = up.reshape(n, c.num_heads, -1), a[:, None, rank:]
        v, scale = up[..., nope:], q.shape[-1] ** -0.5 * factor
    else:
        q = q.reshape(n, c.num_heads, -1)
        q, gate = (q[..., :D], q[..., D:]) if c.attn_output_gate else (q, None)
        k = (x @ t["self_attn.k_proj.weight"].t()).reshape(n, c.num_kv_heads, D)
        v, scale = (x @ t["self_attn.v_proj.weight"].t()).reshape(n, c.num_kv_heads, D), D ** -0.5 * factor
        if c.qk_norm:
            q = _rms(q, t["self_attn.q_norm.weight"].double() + one, c.rms_norm_eps)
            k = _rms(k, t["self_attn.k_norm.weight"].double() + one, c.rms_norm_eps)
    out = []
    for lo, hi in spans:
        if c.is_mla:
            qs = torch.cat([q[lo:hi, :, :nope], _rotate(q[lo:hi, :, nope:], inv, False)], -1)
            ks = torch.cat([up[lo:hi, :, :nope], _rotate(own[lo:hi], inv, False).expand(-1, c.num_heads, -1)], -1)
        else:
            qs, ks = _rotate(q[lo:hi], inv, c.rope.neox), _rotate(k[lo:hi], inv, c.rope.neox)
        out.append(_attend(qs, ks, v[lo:hi], scale))
    out = torch.cat(out)
    if gate is not None:
        out = out * torch.sigmoid(gate)
    return out.reshape(n, -1) @ w_o.t()


def exact(case, seed):
    """The last logits of the scored requests in 64 bits (weights as the case stores them), every request continued
    with the tokens that the model expects. None where that takes too long."""
    cfg, prompts, new = _config(case), _prompts(case, seed), case["new"]
    follow, texts = _follow(cfg, seed).tolist(), []
    for i in _scored(case):
        text = list(prompts[i])
        for _ in range(new - 1):
            text.append(follow[text[-1]])
        texts.append(text)
    if max(map(len, texts)) > 16000 or sum(map(len, texts)) > 24000:
        return None
    ends = torch.tensor([len(t) for t in texts]).cumsum(0).tolist()
    spans = [(e - len(t), e) for e, t in zip(ends, texts)]
    if cfg.quant == "fp8":
        grid = _grid8
    elif cfg.quant == "nvfp4":
        grid = _grid4
    else:
        grid = torch.Tensor.double
    one, (inv, factor) = 1.0 if cfg.gemma_norm else 0.0, _frequencies(cfg)
    x = _embedding(cfg, seed)[torch.tensor([t for text in texts for t in text], device="cuda")].double()
    for l in range(cfg.num_layers):
        t, groups = _layer(cfg, seed, l), []
        # tensors that the engine stores as one matrix share that matrix's scale
        groups = [("self_attn.q_proj.weight", "self_attn.k_proj.weight", "self_attn.v_proj.weight"), ("mlp.gate_proj.weight", "mlp.up_proj.weight"),
                  tuple(f"linear_attn.in_proj_{p}.weight" for p in ("qkv", "z", "b", "a"))]
        for g in groups + [(k,) for k in t if k.endswith("proj.weight") or "kv_a_proj" in k]:
            if all(k in t for k in g) and t[g[0]].dim() == 2 and t[g[0]].dtype != torch.float64:
                for k, part in zip(g, grid(torch.cat([t[k] for k in g])).split([t[k].shape[0] for k in g])):
                    t[k] = part
        y = _rms(x, t["input_layernorm.weight"].double() + one, cfg.rms_norm_eps)
        recurrent = cfg.is_hybrid and cfg.layer_types[l] == "linear_attention"
        x = x + (_recurrent(cfg, y, t, spans) if recurrent else _attention(cfg, y, t, spans, inv, factor))
        y = _rms(x, t["post_attention_layernorm.weight"].double() + one, cfg.rms_norm_eps)
        if "mlp.gate.weight" in t:
            x = x + _experts(cfg, y, t)
        else:
            x = x + torch.cat([_unit(part, t, "mlp.") for part in y.split(4096)])
        del t
    x = _rms(x[torch.tensor(ends, device="cuda") - 1], 1.0, cfg.rms_norm_eps)
    head = _head(cfg, seed)
    return {"tokens": None, "logits": torch.cat([x @ part.double().t() for part in head.split(16384)], 1)}
