"""What this framework is measured on: requests served by ``LLM.generate``, single steps of the op-by-op model families, the
state-space mixers and the sampler, with float64 restatements of what they compute.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a program holds before
the call, ``run`` is one pass through the public entry points, ``work`` is what a pass cannot do without and ``exact`` is its
result in float64.

Weights are random with the spreads of initialised checkpoints (0.02, or the inverse root of the fan-in). Served models carry
embeddings of unit size and an output head that is the embedding rolled by a few rows, so that every token has one clear
successor: greedy and sampled decoding then give the same tokens whatever order a sum is taken in, as confident trained models do.
"""

import math
import random

import numpy as np
import torch
import torch.nn.functional as F

PAGE = 128
DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # Llama-3.1-8B shapes through LLM.generate, all 32 layers.
        # One user in a chat: a prompt of a few hundred tokens, then decode steps of a single row (latency of small launches).
        dict(name="chat", kind="generate", seqs=1, prompt=331, new=24, sampled=False),
        # A full batch, as the serving benchmark decodes (64 in flight): short ragged prompts, then greedy decode steps.
        dict(name="batch", kind="generate", seqs=64, prompt=7040, new=24, sampled=False),
        # Requests with temperature, top-k and top-p (steps that sample take no captured graph), an odd number of them.
        dict(name="sampled", kind="generate", seqs=13, prompt=3000, new=12, sampled=True),
        # A long document, answered in a few tokens: prefill with attention over the whole prompt.
        dict(name="document", kind="generate", seqs=1, prompt=12001, new=2, sampled=False),
        # The feed-forward of a Llama-3.3-70B layer with block-scaled fp8 weights, on the rows of a prefill step.
        dict(name="fp8-mlp", kind="mlp", tokens=2050),
        # DeepSeek-V3 shapes (128 heads, latent cache, 256 fp8 experts top-8 and a shared one): a dense and an expert layer.
        # A decode step of a batch with about a thousand tokens of context each (replays its captured graph).
        dict(name="latent-decode", kind="deepseek", seqs=48, tokens=48, context=1100),
        # A prefill step of ragged prompts, one of them continuing a cached prefix.
        dict(name="latent-prefill", kind="deepseek", seqs=3, tokens=2100, context=700),
        # Gotunex at width 2048 (delta rule and latent attention beside dense and routed feed-forwards): four prompts ...
        dict(name="delta-prefill", kind="gotunex", seqs=4, tokens=8192, context=0),
        # ... and a decode step of 64 sequences (recurrent states and latent cache).
        dict(name="delta-decode", kind="gotunex", seqs=64, tokens=64, context=2048),
        # The state-space mixers on packed prompts: Mamba-1 (selective scan) and Mamba-2 (one decay per head).
        dict(name="mamba1", kind="mamba1", seqs=3, tokens=4099, hidden=2048),
        dict(name="mamba2", kind="mamba2", seqs=2, tokens=4096, hidden=2560),
        # The sampler alone on the logits of a batch: rows with top-k, top-p and min-p in the usual ranges.
        dict(name="sampler", kind="sampler", seqs=64),
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["generate"] * 4 + ["mlp", "deepseek", "deepseek", "gotunex", "gotunex", "mamba1", "mamba2", "sampler"])
    if kind == "generate":
        seqs = rng.choice([1, _spread(rng, 1, 64), _spread(rng, 1, 64)])
        prompt = max(_spread(rng, 64, 11000), 24 * seqs)
        if 0 < prompt % 1024 < 256:          # the scheduler would split such a prompt batch over two steps
            prompt += 256 - prompt % 1024
        return dict(kind=kind, seqs=seqs, prompt=prompt, new=rng.randint(2, 24), sampled=rng.random() < 0.3)
    if kind in ("deepseek", "gotunex"):
        top = dict(deepseek=2100, gotunex=8192)[kind]
        if rng.random() < 0.5:
            seqs = _spread(rng, 1, 64)
            return dict(kind=kind, seqs=seqs, tokens=seqs, context=_spread(rng, 16, 2048 if kind == "gotunex" else 1400))
        seqs = rng.randint(1, 4)
        return dict(kind=kind, seqs=seqs, tokens=_spread(rng, 64, top), context=rng.choice([0, _spread(rng, 16, 700)]) if kind == "deepseek" else 0)
    if kind == "sampler":
        return dict(kind=kind, seqs=_spread(rng, 1, 64))
    if kind == "mlp":
        return dict(kind=kind, tokens=_spread(rng, 1, 2050))
    return dict(kind=kind, seqs=rng.randint(1, 4), tokens=_spread(rng, 64, 4099), hidden=2048 if kind == "mamba1" else 2560)


def _ragged(total, n, least=1):
    """n lengths of at least ``least`` that add up to ``total``: the same ones for the same arguments."""
    r = random.Random(total * 1009 + n)
    share = [0.3 + r.random() for _ in range(n)]
    free = total - least * n
    lens = [least + int(free * s / sum(share)) for s in share]
    lens[0] += total - sum(lens)
    return lens


class _Rand:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return torch.randn(*shape, device=DEV, dtype=dtype, generator=self.g).mul_(std)

    def around_one(self, n, dtype=torch.bfloat16):
        return (1.0 + 0.1 * torch.randn(n, device=DEV, generator=self.g)).to(dtype)

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, device=DEV, generator=self.g)

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), device=DEV, generator=self.g)


# ---------------------------------------------------------------------------------------------- LLM.generate
ROLL = 7          # the successor of token t is t + ROLL


def _llama_config():
    from modular_b200.models.llama3 import Llama3Config

    return Llama3Config.llama31_8b()


def _llama_weights(cfg, seed):
    from modular_b200.models.llama3 import LayerWeights, Llama3Weights

    r = _Rand(seed)
    H, I, deep = cfg.hidden_size, cfg.intermediate_size, 0.02 / math.sqrt(2 * cfg.num_hidden_layers)
    embed = r.normal(cfg.vocab_size, H)
    layers = [LayerWeights(attn_norm=r.around_one(H), wqkv=r.normal(cfg.q_dim + 2 * cfg.kv_dim, H, std=0.02),
                           wo=r.normal(H, cfg.q_dim, std=deep), mlp_norm=r.around_one(H), wgu=r.normal(2 * I, H, std=0.02),
                           wd=r.normal(H, I, std=deep)) for _ in range(cfg.num_hidden_layers)]
    return Llama3Weights(embed, layers, r.around_one(H), torch.roll(embed, ROLL, 0).mul_(0.02))


def _prompts(case, seed, vocab):
    lens = _ragged(case["prompt"], case["seqs"], 16)
    ids = np.random.default_rng(int(seed)).integers(0, vocab, size=case["prompt"])
    return np.split(ids, np.cumsum(lens)[:-1])


def _prepare_generate(case, seed):
    from modular_b200.entrypoints.llm import LLM
    from modular_b200.pipelines.context import SamplingParams

    cfg = _llama_config()
    prompts = _prompts(case, seed, cfg.vocab_size)
    longest, new = max(len(p) for p in prompts), case["new"]
    llm = LLM(cfg, _llama_weights(cfg, seed), device=DEV, dtype=torch.bfloat16, max_length=longest + new + 8,
              max_batch_size=case["seqs"], max_batch_input_tokens=-(-case["prompt"] // 1024) * 1024, page_size=PAGE,
              num_kv_pages=sum(-(-(len(p) + new + 2) // PAGE) + 1 for p in prompts) + 2, enable_prefix_caching=False,
              graph_batch_sizes=[case["seqs"]])
    params = [SamplingParams(temperature=0.0, max_new_tokens=new, ignore_eos=True) if not case["sampled"] else
              SamplingParams(temperature=0.7 + 0.1 * (i % 4), top_k=(-1, 40, -1)[i % 3], top_p=(0.95, 0.9, 1.0)[i % 3],
                             min_p=(0.0, 0.0, 0.05)[i % 3], seed=i, max_new_tokens=new, ignore_eos=True)
              for i in range(case["seqs"])]
    return dict(kind="generate", llm=llm, prompts=prompts, params=params)


def _run_generate(state):
    recs = state["llm"].generate(state["prompts"], state["params"])
    # the tokens of every request and the logits that gave the last ones
    return {"tokens": np.array([r.tokens for r in recs], dtype=np.int64), "logits": state["llm"].model.logits_buf[: len(recs)]}


def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _llama3_angles(cfg, n):
    s = cfg.rope_scaling
    inv = 1.0 / cfg.rope_theta ** (torch.arange(0, cfg.head_dim, 2, dtype=F64, device=DEV) / cfg.head_dim)
    wave, old = 2 * math.pi / inv, s["original_max_position_embeddings"]
    smooth = ((old / wave - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
    inv = (1 - smooth) * inv / s["factor"] + smooth * inv
    return torch.arange(n, dtype=F64, device=DEV).unsqueeze(1) * inv


def _rotate(x, ang, interleaved=False):
    """x [T, heads, d], ang [T, d / 2]"""
    c, s = torch.cos(ang).unsqueeze(1), torch.sin(ang).unsqueeze(1)
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((a * c - b * s, b * c + a * s), -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _attend(q, k, v, scale, first, sink=None):
    """One head: q [n, d] at positions first .. over k [m, d], v [m, dv], causal; in slices of queries."""
    out = []
    for a in range(0, q.shape[0], 2048):
        s = (q[a: a + 2048] @ k.t()) * scale
        at = torch.arange(a, a + s.shape[0], device=s.device).unsqueeze(1) + first
        s = s.masked_fill(torch.arange(k.shape[0], device=s.device) > at, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink.expand(s.shape[0], 1)), 1)
        out.append(torch.softmax(s, -1)[:, : k.shape[0]] @ v)
    return torch.cat(out)


def _exact_generate(case, seed):
    cfg = _llama_config()
    if case["prompt"] + case["seqs"] * case["new"] > 14000:
        return None
    w = _llama_weights(cfg, seed)
    new, seqs = case["new"], []
    for p in _prompts(case, seed, cfg.vocab_size):
        seqs.append(np.concatenate((p, (p[-1] + ROLL * np.arange(1, new)) % cfg.vocab_size)))     # the last token is not fed back
    lens = [len(s) for s in seqs]
    x = w.embed[torch.from_numpy(np.concatenate(seqs)).to(DEV)].double()
    ang = torch.cat([_llama3_angles(cfg, n) for n in lens])
    nq, nk, d, eps = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.rms_norm_eps
    for l in w.layers:
        qkv = (_rms(x, l.attn_norm, eps) @ l.wqkv.double().t()).view(-1, nq + 2 * nk, d)
        qk = _rotate(qkv[:, : nq + nk], ang)
        a = torch.empty_like(qk[:, :nq])
        at = 0
        for n in lens:
            for g in range(nk):
                k, v, each = qk[at: at + n, nq + g], qkv[at: at + n, nq + nk + g], nq // nk
                if n <= 1024:                 # the query heads of a group at once
                    s = qk[at: at + n, g * each: (g + 1) * each].transpose(0, 1) @ k.t() * d ** -0.5
                    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), -math.inf)
                    a[at: at + n, g * each: (g + 1) * each] = (torch.softmax(s, -1) @ v).transpose(0, 1)
                    continue
                for h in range(g * each, (g + 1) * each):
                    a[at: at + n, h] = _attend(qk[at: at + n, h], k, v, d ** -0.5, 0)
            at += n
        x = x + a.reshape(-1, nq * d) @ l.wo.double().t()
        gate, up = (_rms(x, l.mlp_norm, eps) @ l.wgu.double().t()).chunk(2, -1)
        x = x + (F.silu(gate) * up) @ l.wd.double().t()
    ends = np.cumsum(lens)
    rows = torch.from_numpy(np.concatenate([np.arange(e - new, e) for e in ends])).to(DEV)
    logits = _rms(x[rows], w.final_norm, eps) @ w.lm_head.double().t()
    logits = logits.view(case["seqs"], new, -1)
    return {"tokens": logits.argmax(-1), "logits": logits[:, -1]}


def _work_generate(case):
    cfg, T, n, B = _llama_config(), case["prompt"], case["new"], case["seqs"]
    H, I, V, L = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, cfg.num_hidden_layers
    per_layer = H * (cfg.q_dim + 2 * cfg.kv_dim) + H * cfg.q_dim + 3 * H * I
    lens = _ragged(T, B, 16)
    seen = sum(a * (a + 1) / 2 + (n - 1) * a + n * (n - 1) / 2 for a in lens)         # pairs of query and key
    read = sum((n - 1) * a + n * (n - 1) / 2 for a in lens)                           # cached tokens read by decode steps
    kv = 2 * cfg.kv_dim * 2 * L
    weights = 2 * (per_layer * L + V * H)
    return {"bytes": n * weights + kv * (T + B * (n - 1) + read) + n * B * V * 4,
            "flops": 2 * per_layer * L * (T + B * (n - 1)) + 4 * cfg.q_dim * L * seen + 2 * n * B * H * V}


# ---------------------------------------------------------------------------------------------- fp8 feed-forward
WIDTH, INNER = 8192, 28672


def _fp8(r, std, *shape):
    """Block-scaled fp8 values of standard deviation ``std`` in all."""
    q = r.normal(*shape, std=100.0).clamp_(-448, 448).to(torch.float8_e4m3fn)
    return q, r.uniform(0.008 * std, 0.012 * std, *shape[:-2], -(-shape[-2] // 128), -(-shape[-1] // 128))


def _unblocked(q, s):
    return q.double() * s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)


def _mlp_inputs(case, seed):
    r = _Rand(seed)
    return _fp8(r, 0.02, 2 * INNER, WIDTH), _fp8(r, 0.02, WIDTH, INNER), r.normal(case["tokens"], WIDTH), r.normal(case["tokens"], WIDTH)


def _prepare_mlp(case, seed):
    from modular_b200.nn.layers import MLP, Linear

    (gu, gu_s), (down, down_s), x, h = _mlp_inputs(case, seed)
    return dict(kind="mlp", mlp=MLP(Linear(gu, weight_scale=gu_s), Linear(down, weight_scale=down_s)), x=x, h=h)


def _run_mlp(s):
    return {"h": s["mlp"](s["x"], residual=s["h"])}


def _exact_mlp(case, seed):
    gu, down, x, h = _mlp_inputs(case, seed)
    gate, up = (x.double() @ _unblocked(*gu).t()).chunk(2, -1)
    return {"h": h.double() + (F.silu(gate) * up) @ _unblocked(*down).t()}


# ---------------------------------------------------------------------------------------------- steps of paged models
def _layout(case, page=PAGE):
    """Step tensors of a packed batch whose sequences bring ``tokens`` in all and have up to ``context`` cached ones."""
    B, T, ctx = case["seqs"], case["tokens"], case["context"]
    decode = B == T
    q = [1] * B if decode else _ragged(T, B, 1)
    r = random.Random(T * 31 + ctx)
    if decode:
        past = [max(1, int(ctx * (0.6 + 0.4 * r.random()))) for _ in range(B)]
    else:
        past = [0] * (B - 1) + [ctx]                # the last prompt continues a cached prefix
    kv = [a + b for a, b in zip(q, past)]
    need = [-(-n // page) for n in kv]
    order = list(range(1, sum(need) + 1))           # page 0 is the null page
    r.shuffle(order)
    table = torch.zeros(B, max(need), dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = torch.tensor(order[at: at + n], dtype=torch.int32)
        at += n
    pos = torch.cat([torch.arange(p, n) for p, n in zip(past, kv)])
    seq = torch.cat([torch.full((n,), i) for i, n in enumerate(q)])
    slots = table[seq, pos // page].long() * page + pos % page
    start = torch.tensor([0] + q[:-1]).cumsum(0)
    i32 = lambda t: t.to(device=DEV, dtype=torch.int32)
    step = dict(positions=i32(pos), slots=slots.to(DEV), block_table=table.to(DEV), q_start=i32(start), q_len=i32(torch.tensor(q)),
                kv_len=i32(torch.tensor(kv)), logit_rows=i32(start + torch.tensor(q) - 1))
    return step, q, past, sum(need) + 1


def _cached(kv_plane, table_row, n):
    """The first n rows of a sequence in a paged plane [pages, page, width], in float64."""
    return kv_plane[table_row.long()].reshape(-1, kv_plane.shape[-1])[:n].double()


def _deepseek_config():
    from modular_b200.models.deepseek_v3 import DeepseekV3Config

    cfg = DeepseekV3Config.deepseek_v3()
    cfg.num_hidden_layers, cfg.first_k_dense_replace = 2, 1
    return cfg


def _deepseek_weights(cfg, seed):
    from modular_b200.models.deepseek_v3 import DeepseekV3Weights, DSLayer
    from modular_b200.nn.moe import Fp8ExpertWeights, MoE

    r = _Rand(seed)
    H, h, I, E = cfg.hidden_size, cfg.num_attention_heads, cfg.moe_intermediate_size, cfg.n_routed_experts
    layers = []
    for i in range(cfg.num_hidden_layers):
        l = DSLayer(r.around_one(H), r.normal(cfg.q_lora_rank, H, std=0.02), r.around_one(cfg.q_lora_rank),
                    r.normal(h * cfg.qk_head_dim, cfg.q_lora_rank, std=0.02), r.normal(cfg.latent_dim, H, std=0.02),
                    r.around_one(cfg.kv_lora_rank), r.normal(h, cfg.kv_lora_rank, cfg.qk_nope_head_dim, std=0.02),
                    r.normal(h, cfg.v_head_dim, cfg.kv_lora_rank, std=0.02), r.normal(H, h * cfg.v_head_dim, std=0.02), r.around_one(H))
        if cfg.is_moe_layer(i):
            gate, bias = r.normal(E, H, std=0.02).float(), r.normal(E, std=0.1, dtype=torch.float32)
            gu, down = _fp8(r, 0.02, E, 2 * I, H), _fp8(r, 0.01, E, H, I)      # output projections are scaled down with depth
            l.moe = MoE(cfg.moe_config(), gate, Fp8ExpertWeights(*gu), Fp8ExpertWeights(*down), bias,
                        r.normal(2 * I * cfg.n_shared_experts, H, std=0.02), r.normal(H, I * cfg.n_shared_experts, std=0.01))
        else:
            l.wgu, l.wd = r.normal(2 * cfg.intermediate_size, H, std=0.02), r.normal(H, cfg.intermediate_size, std=0.02)
        layers.append(l)
    return DeepseekV3Weights(cfg, r.normal(cfg.vocab_size, H), layers, r.around_one(H), r.normal(cfg.vocab_size, H, std=0.02)), r


def _deepseek_inputs(case, seed):
    cfg = _deepseek_config()
    w, r = _deepseek_weights(cfg, seed)
    step, q, past, pages = _layout(case)
    # cached latents have unit size (they are normed), cached rotated keys are of the same order
    kv = r.normal(pages, 1, cfg.num_hidden_layers, 1, PAGE, cfg.latent_dim)
    step["tokens"] = r.ids(case["tokens"], cfg.vocab_size)
    return cfg, w, step, q, past, kv


def _prepare_deepseek(case, seed):
    from modular_b200.models.deepseek_v3 import DeepseekV3Model

    cfg, w, step, q, past, kv = _deepseek_inputs(case, seed)
    model = DeepseekV3Model(cfg, w, kv, max_tokens=max(case["tokens"], 64), max_seqs=max(case["seqs"], 1), max_position=4096)
    if case["seqs"] == case["tokens"]:
        model.capture_decode_graphs([case["seqs"]])
    return dict(kind="deepseek", model=model, step=step, kv=kv)


def _run_deepseek(state):
    return {"logits": state["model"].forward_tensors(**state["step"]), "cache": state["kv"]}


def _yarn_angles(cfg, pos):
    rs, d = cfg.rope_scaling, cfg.qk_rope_head_dim
    inv = 1.0 / cfg.rope_theta ** (torch.arange(0, d, 2, dtype=F64, device=DEV) / d)
    edge = lambda n: d * math.log(rs["original_max_position_embeddings"] / (n * 2 * math.pi)) / (2 * math.log(cfg.rope_theta))
    lo, hi = max(math.floor(edge(rs["beta_fast"])), 0), min(math.ceil(edge(rs["beta_slow"])), d - 1)
    ramp = ((torch.arange(d // 2, dtype=F64, device=DEV) - lo) / (hi - lo)).clamp(0, 1)
    return pos.double().unsqueeze(1) * (inv / rs["factor"] * ramp + inv * (1 - ramp))


def _exact_deepseek(case, seed):
    cfg, w, st, qlen, past, kv = _deepseek_inputs(case, seed)
    h, N, R, eps, m = cfg.num_attention_heads, cfg.qk_nope_head_dim, cfg.kv_lora_rank, cfg.rms_norm_eps, cfg.moe_config()
    scale = cfg.qk_head_dim ** -0.5 * (0.1 * math.log(cfg.rope_scaling["factor"]) + 1.0) ** 2
    ang = _yarn_angles(cfg, st["positions"])
    cache = kv.double()
    flat = cache.view(-1, cfg.num_hidden_layers, PAGE, cfg.latent_dim)
    x = w.embed[st["tokens"]].double()
    ffn = lambda z, gu, down: (lambda g, u: (F.silu(g) * u) @ down.double().t())(*(z @ gu.double().t()).chunk(2, -1))
    for li, l in enumerate(w.layers):
        xn = _rms(x, l.attn_norm, eps)
        q = (_rms(xn @ l.q_a.double().t(), l.q_a_norm, eps) @ l.q_b.double().t()).view(-1, h, cfg.qk_head_dim)
        a = xn @ l.kv_a.double().t()
        row = torch.cat((_rms(a[:, :R], l.kv_a_norm, eps), _rotate(a[:, None, R:], ang, True)[:, 0]), 1)
        flat[st["slots"] // PAGE, li, st["slots"] % PAGE] = row
        q_lat = torch.cat((torch.einsum("thn,hrn->thr", q[..., :N], l.w_uk.double()), _rotate(q[..., N:], ang, True)), -1)
        o = torch.empty(x.shape[0], h, R, dtype=F64, device=DEV)
        at = 0
        for i, n in enumerate(qlen):
            keys = _cached(flat[:, li], st["block_table"][i], past[i] + n)
            for j in ([slice(None)] if n == 1 else range(h)):
                if n == 1:
                    p = torch.softmax(q_lat[at] @ keys.t() * scale, -1)
                    o[at] = p @ keys[:, :R]
                else:
                    o[at: at + n, j] = _attend(q_lat[at: at + n, j], keys, keys[:, :R], scale, past[i])
            at += n
        x = x + torch.einsum("thr,hvr->thv", o, l.w_uv.double()).reshape(x.shape[0], -1) @ l.wo.double().t()
        xn = _rms(x, l.mlp_norm, eps)
        if l.moe is None:
            x = x + ffn(xn, l.wgu, l.wd)
            continue
        e = l.moe
        score = torch.sigmoid(xn @ e.gate.double().t())
        choice = score + e.bias.double()
        group = choice.view(-1, m.n_group, m.n_routed_experts // m.n_group)
        kept = torch.zeros_like(group[..., 0], dtype=torch.bool).scatter_(1, group.topk(2, -1).values.sum(-1).topk(m.topk_group, -1).indices, True)
        ids = choice.masked_fill(~kept.repeat_interleave(group.shape[2], 1), -math.inf).topk(m.num_experts_per_tok, -1).indices
        p = score.gather(1, ids)
        p = p / p.sum(-1, keepdim=True) * m.routed_scaling_factor
        y = ffn(xn, e.shared_gate_up, e.shared_down)
        for j in range(m.n_routed_experts):
            tok, at = torch.nonzero(ids == j, as_tuple=True)
            if tok.numel():
                y.index_add_(0, tok, ffn(xn[tok], _unblocked(e.w_gate_up.q[j], e.w_gate_up.scale[j]), _unblocked(e.w_down.q[j], e.w_down.scale[j])) * p[tok, at, None])
        x = x + y
    x = _rms(x[st["logit_rows"].long()], w.final_norm, eps)
    return {"logits": x @ w.lm_head.double().t(), "cache": cache}


def _pairs(case):
    _, q, past, _ = _layout(case)
    return sum(n * p + n * (n + 1) / 2 for n, p in zip(q, past)), sum(n + p for n, p in zip(q, past))


def _work_deepseek(case):
    cfg, T, B = _deepseek_config(), case["tokens"], case["seqs"]
    H, h, R, I, k, E = cfg.hidden_size, cfg.num_attention_heads, cfg.kv_lora_rank, cfg.moe_intermediate_size, cfg.num_experts_per_tok, cfg.n_routed_experts
    att = H * (cfg.q_lora_rank + cfg.latent_dim) + cfg.q_lora_rank * h * cfg.qk_head_dim + h * (cfg.qk_nope_head_dim + cfg.v_head_dim) * R + h * cfg.v_head_dim * H
    used = E * (1 - (1 - k / E) ** T)                        # experts that get at least one of T tokens
    pairs, keys = _pairs(case)
    weights = 2 * (2 * att + 3 * H * cfg.intermediate_size + 3 * H * I + H * E + cfg.vocab_size * H) + used * 3 * H * I
    # a query and a key meet in the narrower form: 192 + 128 wide per head after projecting the latents up once
    wide = min(cfg.qk_head_dim + cfg.v_head_dim + 0.0, 2 * R + cfg.qk_rope_head_dim) if T > B else 2 * R + cfg.qk_rope_head_dim
    return {"bytes": weights + 2 * 2 * cfg.latent_dim * keys + 4 * B * cfg.vocab_size,
            "flops": 2 * T * (2 * att + 3 * H * cfg.intermediate_size + 3 * H * I * (k + 1) + H * E) + 2 * 2 * h * wide * pairs + 2 * B * H * cfg.vocab_size}


# ---------------------------------------------------------------------------------------------- Gotunex
def _gotunex_config():
    from modular_b200.models.gotunex import GotunexConfig

    att = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=1536, scale=192 ** -0.5, rot=dict(base=10000.0, dims=64))
    delta = dict(heads=16, kv_heads=16, dim=128, vdim=128, conv=4)
    return GotunexConfig.build(2048, 102400, "dDDA", att, delta, 10944, 1408, 64, 6)


def _gotunex_tensors(cfg, r):
    sd = {}
    for name, shape in cfg.tensor_shapes().items():
        leaf = name.rsplit(".", 1)[-1]
        if leaf == "table":
            experts = cfg.layers[int(name.split(".")[0][1:])]["mlp"]["router"]["experts"]
            t = r.uniform(0, 1, shape[0], experts).topk(shape[1], dim=-1).indices.int()
        elif leaf == "A_log":
            t = r.uniform(-2.0, 0.0, *shape).bfloat16()
        elif leaf == "dt_bias":
            t = r.normal(*shape).sub_(3.0)
        elif "norm" in leaf:
            t = r.around_one(shape[0])
        elif leaf == "sink" or name == "embed":
            t = r.normal(*shape)
        else:
            t = r.normal(*shape, std=shape[-1] ** -0.5)
        sd[name] = t
    return sd


def _gotunex_inputs(case, seed):
    cfg, r = _gotunex_config(), _Rand(seed)
    sd = _gotunex_tensors(cfg, r)
    step, q, past, pages = _layout(case)
    kv = r.normal(pages, 1, len(cfg.cache_layers), 1, PAGE, cfg.cache_width)
    # states of running sequences: values of order v / sqrt(dim), raw inputs of the short convolutions
    state = {n: r.normal(case["seqs"], *shape, std=0.05 if n.endswith("delta") else 1.0, dtype=dt) for n, shape, dt in cfg.state_specs()}
    step["tokens"] = r.ids(case["tokens"], cfg.vocab_size)
    step["state_slot"] = torch.arange(case["seqs"], dtype=torch.int32, device=DEV).flip(0).contiguous()
    return cfg, sd, step, q, past, kv, state


def _prepare_gotunex(case, seed):
    from modular_b200.models.gotunex import GotunexModel, GotunexWeights

    cfg, sd, step, q, past, kv, state = _gotunex_inputs(case, seed)
    model = GotunexModel(cfg, GotunexWeights.from_state_dict(cfg, sd, DEV, torch.bfloat16), kv, max_tokens=max(case["tokens"], 64),
                         max_seqs=case["seqs"], max_position=4096, state=state)
    if case["seqs"] == case["tokens"]:
        model.capture_decode_graphs([case["seqs"]])
    return dict(kind="gotunex", model=model, step=step, kv=kv, state=state)


def _run_gotunex(state):
    return {"logits": state["model"].forward_tensors(**state["step"]), "cache": state["kv"], **state["state"]}


def _exact_gotunex(case, seed):
    cfg, sd, st, qlen, past, kv, state = _gotunex_inputs(case, seed)
    eps, dbl = cfg.rms_norm_eps, lambda n: sd[n].double()
    cache, state = kv.double(), {k: v.double() for k, v in state.items()}
    x = dbl("embed")[st["tokens"]]
    plane, T = 0, x.shape[0]
    spans, at = [], 0
    for n in qlen:
        spans.append(slice(at, at + n))
        at += n
    slot = st["state_slot"].tolist()
    for i, l in enumerate(cfg.layers):
        m, p, q_ = l["mixer"], f"l{i}.mix.", f"l{i}.mlp."
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        n1, n2 = _rms(x, sd[f"l{i}.norm1"], eps), _rms(x, sd[f"l{i}.norm2"], eps)
        if l["type"] == "latent_attention":
            R, r_ = m["kv_rank"], m["rot_dim"]
            ang = st["positions"].double().unsqueeze(1) * m["rot"]["base"] ** (-torch.arange(0, r_, 2, dtype=F64, device=DEV) / r_)
            a = n1 @ dbl(p + "dkv").t()
            view = cache[:, 0, plane, 0]
            view[st["slots"] // PAGE, st["slots"] % PAGE] = torch.cat((_rms(a[:, :R], sd[p + "dkv.norm"], eps), _rotate(a[:, None, R:], ang)[:, 0]), 1)
            q = (_rms(n1 @ dbl(p + "dq").t(), sd[p + "dq.norm"], eps) @ dbl(p + "uq").t()).view(T, H, d + r_)
            q = torch.cat((q[..., :d], _rotate(q[..., d:], ang)), -1)
            uk, uv, o = dbl(p + "uk").view(H, d, R), dbl(p + "uv").view(H, dv, R), torch.empty(T, H, dv, dtype=F64, device=DEV)
            for s, span in enumerate(spans):
                rows = _cached(view, st["block_table"][s], past[s] + qlen[s])
                for h in range(H):
                    o[span, h] = _attend(q[span, h], torch.cat((rows[:, :R] @ uk[h].t(), rows[:, R:]), 1), rows[:, :R] @ uv[h].t(),
                                         m["scale"], past[s], dbl(p + "sink")[h])
            y = (o.reshape(T, H * dv) * torch.sigmoid(n1 @ dbl(p + "g").t())) @ dbl(p + "o").t()
            plane += 1
        else:
            raw = torch.cat([n1 @ dbl(p + n).t() for n in "qkv"], 1)
            taps = torch.cat([dbl(p + n + ".conv") for n in "qkv"])
            beta = torch.sigmoid(n1 @ dbl(p + "b").t())
            g = torch.exp(-dbl(p + "A_log").exp().view(1, H, 1) * F.softplus(((n1 @ dbl(p + "a1").t()) @ dbl(p + "a2").t()
                                                                             + dbl(p + "dt_bias")).view(T, H, d)))
            o = torch.empty(T, H, dv, dtype=F64, device=DEV)
            S_all, conv = state[f"l{i}.delta"], state[f"l{i}.conv"]
            W = taps.shape[1]
            # sequences of one token run side by side, longer ones one after the other
            groups = [list(range(len(qlen)))] if T == len(qlen) else [[s] for s in range(len(qlen))]
            for seqs in groups:
                n, slots = qlen[seqs[0]], [slot[s] for s in seqs]
                rows = torch.stack([raw[spans[s]] for s in seqs])                               # [B, n, C]
                keep = torch.tensor([float(past[s] > 0) for s in seqs], dtype=F64, device=DEV)
                full = torch.cat((conv[slots].transpose(1, 2) * keep.view(-1, 1, 1), rows), 1)
                conv[slots] = full[:, full.shape[1] - (W - 1):].transpose(1, 2)
                c = F.silu(sum(full[:, j: j + n] * taps[:, j] for j in range(W)))
                q, k, v = (t.reshape(len(seqs), n, H, -1) for t in c.split([H * d, H * d, H * dv], -1))
                unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
                q, k = unit(q) / d ** 0.5, unit(k)
                gs, bs = torch.stack([g[spans[s]] for s in seqs]), torch.stack([beta[spans[s]] for s in seqs])
                S = S_all[slots] * keep.view(-1, 1, 1, 1)                                        # [B, H, dv, d]
                for t in range(n):
                    S = S * gs[:, t].unsqueeze(2)
                    u = bs[:, t].unsqueeze(-1) * (v[:, t] - (S @ k[:, t].unsqueeze(-1)).squeeze(-1))
                    S = S + u.unsqueeze(-1) * k[:, t].unsqueeze(2)
                    out = (S @ q[:, t].unsqueeze(-1)).squeeze(-1)
                    for b, s in enumerate(seqs):
                        o[spans[s].start + t] = out[b]
                S_all[slots] = S
            o = _rms(o, sd[p + "norm"], eps).reshape(T, -1) * torch.sigmoid((n1 @ dbl(p + "g1").t()) @ dbl(p + "g2").t())
            y = o @ dbl(p + "o").t()
        if l["mlp"]["kind"] == "dense":
            x = x + y + F.gelu(n2 @ dbl(q_ + "up").t(), approximate="tanh") @ dbl(q_ + "down").t()
            continue
        ids, top = sd[q_ + "table"][st["tokens"]], l["mlp"]["router"]["top"]
        x = x + y
        for e in range(l["mlp"]["router"]["experts"]):
            tok = torch.nonzero(ids == e, as_tuple=True)[0]
            if tok.numel():
                z = n2[tok]
                x.index_add_(0, tok, (F.silu(z @ dbl(f"{q_}e{e}.gate").t()) * (z @ dbl(f"{q_}e{e}.up").t())) @ dbl(f"{q_}e{e}.down").t() / top)
    logits = _rms(x[st["logit_rows"].long()], sd["final.norm"], eps) @ dbl("head").t()
    return {"logits": logits, "cache": cache, **state}


def _work_gotunex(case):
    cfg, T, B = _gotunex_config(), case["tokens"], case["seqs"]
    W, V = cfg.hidden_size, cfg.vocab_size
    pairs, keys = _pairs(case)
    bytes_, flops = V * W * 2 + B * V * 4.0, 2.0 * B * W * V
    for l in cfg.layers:
        m = l["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if l["type"] == "latent_attention":
            n = W * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + 2 * H * dv) + m["q_rank"] * H * (d + m["rot_dim"]) + m["kv_rank"] * H * (d + dv)
            bytes_ += 2 * cfg.cache_width * keys
            wide = d + m["rot_dim"] + dv if T > B else 2 * m["kv_rank"] + m["rot_dim"]
            flops += 2 * H * wide * pairs
        else:
            n = W * (2 * H * d + 2 * H * dv + 2 * d + H) + d * H * (d + dv)
            state = H * d * dv * 4 + (2 * H * d + H * dv) * (m["conv"] - 1) * 4
            bytes_ += B * state * (2 if T == B else 1)
            flops += 7 * T * H * d * dv
        bytes_ += 2 * n
        flops += 2 * T * n
        ff = l["mlp"]
        if ff["kind"] == "dense":
            bytes_ += 2 * 2 * W * ff["ff"]
            flops += 2 * T * 2 * W * ff["ff"]
        else:
            E, k, n = ff["router"]["experts"], ff["router"]["top"], 3 * W * ff["expert"]["ff"]
            bytes_ += 2 * n * E * (1 - (1 - k / E) ** T)
            flops += 2 * T * k * n
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------------------------- state-space mixers
def _mixer_inputs(case, seed):
    from modular_b200.nn.state_space import Mamba2Mixer, MambaMixer

    r, H, T = _Rand(seed), case["hidden"], case["tokens"]
    one = case["kind"] == "mamba1"
    with torch.no_grad():
        if one:
            m = MambaMixer(H, 2 * H, d_state=16, dtype=torch.bfloat16, device=DEV)
            for w in (m.in_proj, m.x_proj, m.dt_proj, m.out_proj):
                w.weight.copy_(r.normal(*w.weight.shape, std=w.weight.shape[1] ** -0.5))
            step = m.dt_proj.bias
        else:
            m = Mamba2Mixer(H, 2 * H // 64, 64, d_state=128, dtype=torch.bfloat16, device=DEV)
            for w in (m.in_proj, m.out_proj):
                w.weight.copy_(r.normal(*w.weight.shape, std=w.weight.shape[1] ** -0.5))
            m.A_log.copy_(torch.log(r.uniform(1, 16, m.H)))
            m.norm_w.copy_(r.around_one(m.d_inner))
            step = m.dt_bias
        m.conv_w.copy_(r.normal(*m.conv_w.shape, std=0.3))
        m.conv_b.copy_(r.normal(*m.conv_b.shape, std=0.1))
        m.D.copy_(r.around_one(m.D.shape[0]))
        dt = torch.exp(r.uniform(math.log(1e-3), math.log(0.1), *step.shape))          # step sizes as these models start with
        step.copy_(dt + torch.log(-torch.expm1(-dt)))
    lens = _ragged(T, case["seqs"])
    h = r.normal(T, H)
    conv, ssm = m.alloc_state(case["seqs"])
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return m, h, lens, i32([0] + list(np.cumsum(lens))), (conv, ssm), i32(list(range(case["seqs"]))), i32([0] * case["seqs"])


def _prepare_mixer(case, seed):
    m, h, _, cu, state, idx, init = _mixer_inputs(case, seed)
    return dict(kind=case["kind"], mixer=m, h=h, cu=cu, state=state, idx=idx, init=init)


def _run_mixer(s):
    return {"y": s["mixer"](s["h"], s["cu"], s["state"], s["idx"], s["init"]), "conv": s["state"][0], "ssm": s["state"][1]}


@torch.no_grad()
def _exact_mixer(case, seed):
    m, h, lens, _, (conv, ssm), _, _ = _mixer_inputs(case, seed)
    one, D = case["kind"] == "mamba1", m.d_inner
    conv, ssm = conv.double(), ssm.double()
    proj = h.double() @ m.in_proj.weight.double().t()
    x_all, z = (proj[:, :D], proj[:, D:]) if one else (proj[:, D: D + m.conv_dim], proj[:, :D])
    w, at, y = m.conv_w.double(), 0, torch.empty(h.shape[0], D, dtype=F64, device=DEV)
    A = -torch.exp(m.A_log.double())
    for s, n in enumerate(lens):
        raw = F.pad(x_all[at: at + n], (0, 0, m.d_conv - 1, 0))
        conv[s] = raw[n:].t()
        x = F.silu(sum(raw[j: j + n] * w[:, j] for j in range(m.d_conv)) + m.conv_b.double())
        if one:
            dbc = x @ m.x_proj.weight.double().t()
            dt = F.softplus(dbc[:, : m.dt_rank] @ m.dt_proj.weight.double().t() + m.dt_proj.bias.double())
            B, C = dbc[:, m.dt_rank:].split(m.d_state, -1)
            S = ssm[s]
            for t in range(n):
                S = torch.exp(dt[t, :, None] * A) * S + (dt[t] * x[t])[:, None] * B[t]
                y[at + t] = S @ C[t]
            y[at: at + n] = (y[at: at + n] + m.D.double() * x) * F.silu(z[at: at + n])
        else:
            dt = F.softplus(proj[at: at + n, D + m.conv_dim:] + m.dt_bias.double())
            xs = x[:, :D].view(n, m.H, m.P)
            B, C = (t.view(n, m.G, m.N).repeat_interleave(m.H // m.G, 1) for t in x[:, D:].split(m.G * m.N, -1))
            S, out = ssm[s], y.view(-1, m.H, m.P)
            for t in range(n):
                S = torch.exp(dt[t] * A).view(-1, 1, 1) * S + (dt[t, :, None] * xs[t]).unsqueeze(-1) * B[t].unsqueeze(1)
                out[at + t] = (S @ C[t].unsqueeze(-1)).squeeze(-1) + m.D.double()[:, None] * xs[t]
        ssm[s] = S
        at += n
    if not one:
        y = _rms(y * F.silu(z), m.norm_w, m.eps)
    return {"y": y @ m.out_proj.weight.double().t(), "conv": conv, "ssm": ssm}


def _work_mixer(case):
    H, T, B = case["hidden"], case["tokens"], case["seqs"]
    D = 2 * H
    if case["kind"] == "mamba1":
        rank = (H + 15) // 16
        weights, state, scan = 3 * H * D + D * (2 * rank + 32), D * (16 + 3), 6 * D * 16
    else:
        weights, state, scan = H * (2 * D + 256 + D // 64) + D * H, D * 128 + 3 * (D + 256), 5 * D * 128
    return {"bytes": 2 * weights + 4 * T * H + 4 * B * state, "flops": 2 * T * weights + T * scan}


# ---------------------------------------------------------------------------------------------- sampler
VOCAB = 128256


def _prepare_sampler(case, seed):
    r, n = _Rand(seed), case["seqs"]
    pick = lambda *v: torch.tensor([v[i % len(v)] for i in range(n)], device=DEV)
    # logits of a language model: a broad bulk and a few tokens that stand out
    logits = r.normal(n, VOCAB, std=2.0, dtype=torch.float32)
    lead = torch.randint(0, VOCAB, (n, 40), device=DEV, generator=r.g)
    logits.scatter_add_(1, lead, r.uniform(4.0, 12.0, n, 40))
    return dict(kind="sampler", logits=logits, temperature=pick(0.7, 1.0, 0.8, 0.6), top_k=pick(0, 50, 0, 20, 0).to(torch.int32),
                top_p=pick(0.9, 0.95, 1.0), min_p=pick(0.0, 0.0, 0.05, 0.0, 0.0),
                seeds=torch.randint(0, 1 << 62, (n,), device=DEV, generator=r.g))


def _run_sampler(s):
    from modular_b200 import ops

    return {"tokens": ops.sample(s["logits"], s["temperature"], s["top_k"], s["top_p"], s["min_p"], s["seeds"], step=3)}


# ---------------------------------------------------------------------------------------------- the interface
_PREPARE = dict(generate=_prepare_generate, mlp=_prepare_mlp, deepseek=_prepare_deepseek, gotunex=_prepare_gotunex, mamba1=_prepare_mixer, mamba2=_prepare_mixer,
                sampler=_prepare_sampler)
_RUN = dict(generate=_run_generate, mlp=_run_mlp, deepseek=_run_deepseek, gotunex=_run_gotunex, mamba1=_run_mixer, mamba2=_run_mixer, sampler=_run_sampler)
_WORK = dict(generate=_work_generate, deepseek=_work_deepseek, gotunex=_work_gotunex, mamba1=_work_mixer, mamba2=_work_mixer)
_EXACT = dict(generate=_exact_generate, mlp=_exact_mlp, deepseek=_exact_deepseek, gotunex=_exact_gotunex, mamba1=_exact_mixer, mamba2=_exact_mixer)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def work(case):
    if case["kind"] == "sampler":
        return {"bytes": case["seqs"] * (VOCAB * 4 + 36), "flops": 0}
    if case["kind"] == "mlp":
        return {"bytes": 3 * WIDTH * INNER + 6 * case["tokens"] * WIDTH, "flops": 6 * case["tokens"] * WIDTH * INNER}
    return _WORK[case["kind"]](case)


def exact(case, seed):
    """``run``'s answer in float64; None for the sampler (a draw from its own random stream has no such value)."""
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None


def tolerance(case):
    """About four times what separates the start of the measurements from ``exact``. Served models: 32 layers of bf16; fp8 products: operands
    of three bits; DeepSeek-V3: fp8 experts, and a close choice of experts may fall the other way."""
    return {"generate": {"rel": 0.08, "differ": 0.01}, "mlp": {"rel": 0.1}, "deepseek": {"rel": 0.06}, "gotunex": {"rel": 0.025},
            "mamba1": {"rel": 0.02}, "mamba2": {"rel": 0.02}, "sampler": {"differ": 0.05}}[case["kind"]]
