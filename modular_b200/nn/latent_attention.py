"""Latent attention: queries and keys / values go through low-rank latents, and the cache keeps one row per token
(the normed key/value latent and a rotated key part that all heads share).

Runs in the absorbed form (``q_lat = W_uk^T q`` per head, attention over the cached rows, ``o = W_uv o_lat`` per head); long
prompts of the usual sizes project the rows up to keys and values per head instead (:func:`prompt_plan`). Options: rotate-half or interleaved rotary pairs, a sliding window, a learned sink per head (a
score without key or value in the softmax denominator), a sigmoid output gate per value column or per head, and reading
another layer's cache rows (a layer without a key/value projection of its own).

Column layouts are padded for the kernels, with zeros: per head ``[dim -> multiple of 64 | rot_dim -> 64]`` for queries,
``[kv_rank -> a kernel size | rot_dim -> 64]`` for cache rows, vdim -> multiple of 8.

Kernels: ``attention_tc.cu`` (projected prompts), ``mla_tc.cu`` (tcgen05: 512-wide latents, multiples of 128 heads), ``mla.cu`` (other sizes in bf16),
``mla_ragged.cu`` (fp32 and anything wider); CPU tensors take the PyTorch form.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from .. import ops
from .._native import lib as _lib
from .delta_rule import gemm_k, pad_to, up8

_LATENT_SIZES = (64, 128, 192, 256, 384, 512)     # widths the tensor-core kernels are built for
_SPLIT_WS: dict = {}
_SPLIT_WS_BYTES = 64 << 20


def up64(n: int) -> int:
    return (n + 63) // 64 * 64


def latent_pad(kv_rank: int) -> int:
    return next((n for n in _LATENT_SIZES if kv_rank <= n), up64(kv_rank))


def rot_pad(rot_dim: int) -> int:
    return 64 if rot_dim <= 64 else up8(rot_dim)


@dataclass
class LatentAttentionConfig:
    heads: int
    dim: int                 # unrotated query / key width per head
    rot_dim: int             # width of the rotated part
    rot_dims: int            # how many of its values rotate (the first ones)
    vdim: int
    kv_rank: int
    q_rank: int
    scale: float
    rope_base: float
    eps: float
    own_cache: bool = True   # False: the layer reads another layer's cache rows
    interleaved: bool = False
    window: int = 0          # keys a query sees, itself included (0: all before it)
    sink: bool = True
    head_gate: bool = False  # the output gate is one number per head, applied inside the attention kernels

    @property
    def head_width(self) -> int:
        return up64(self.dim) + rot_pad(self.rot_dim)

    @property
    def projects(self) -> bool:
        """Whether prompts may run on projected keys and values (bf16 on the GPU)."""
        return up64(self.dim) == self.vdim_pad == 128 and rot_pad(self.rot_dim) == 64

    def prompt_scratch_bytes(self, T: int) -> int:
        return prompt_scratch_bytes(self.heads, latent_pad(self.kv_rank), T, self.projects)

    @property
    def cache_width(self) -> int:
        return latent_pad(self.kv_rank) + rot_pad(self.rot_dim)

    @property
    def vdim_pad(self) -> int:
        return up8(self.vdim)


def _split_ws(device) -> torch.Tensor:
    idx = device.index or 0
    if idx not in _SPLIT_WS:
        _SPLIT_WS[idx] = torch.empty(_SPLIT_WS_BYTES // 4, dtype=torch.float32, device=device)
    return _SPLIT_WS[idx]


def pad_heads(w: torch.Tensor, heads: int, rows: int, rows_pad: int) -> torch.Tensor:
    """[heads * rows, K] -> [heads * rows_pad, K] with zero rows after every head."""
    K = w.shape[1]
    if rows == rows_pad:
        return w
    out = torch.zeros(heads, rows_pad, K, dtype=w.dtype, device=w.device)
    out[:, :rows] = w.view(heads, rows, K)
    return out.view(heads * rows_pad, K)


class LatentAttention:
    """Weights of one mixer. ``w_in``: the projections that read the layer input, stacked ``[dq | dkv | g]`` (one GEMM)."""

    def __init__(self, cfg: LatentAttentionConfig, t: dict, width_pad: int, device, dtype):
        """``t``: the mixer's tensors by their short names (``dq``, ``dq.norm``, ``uk``, ``sink``, ...)."""
        c = self.cfg = cfg
        put = lambda x, dt=dtype: x.to(device=device, dtype=dt).contiguous()
        H, d, r, vp, Rp = c.heads, c.dim, c.rot_dim, c.vdim_pad, latent_pad(c.kv_rank)
        self.q_pad = gemm_k(c.q_rank)
        parts = [pad_to(t["dq"], self.q_pad, width_pad)]
        self.kv_off, at = -1, self.q_pad
        if c.own_cache:
            n = c.kv_rank + r
            parts.append(pad_to(t["dkv"], up8(n), width_pad))
            self.kv_off, at = at, at + up8(n)
        self.g_off = at
        parts.append(pad_to(t["g"], up8(H), width_pad) if c.head_gate else pad_to(pad_heads(t["g"], H, c.vdim, vp), H * vp, width_pad))
        self.w_in = put(torch.cat(parts))
        self.q_norm = put(t["dq.norm"])
        self.kv_norm = put(t["dkv.norm"]) if c.own_cache else None
        uq = t["uq"].view(H, d + r, c.q_rank)
        new = lambda *s: torch.zeros(*s, dtype=uq.dtype, device=uq.device)
        q = new(H, c.head_width, self.q_pad)
        q[:, :d, : c.q_rank] = uq[:, :d]
        q[:, up64(d): up64(d) + r, : c.q_rank] = uq[:, d:]
        self.w_uq = put(q.view(H * c.head_width, self.q_pad))
        uk = new(H, Rp, up64(d))
        uk[:, : c.kv_rank, :d] = t["uk"].view(H, d, c.kv_rank).transpose(1, 2)
        self.w_uk = put(uk)                                          # [h, latent, dim]: queries into latent space
        uv = new(H, vp, Rp)
        uv[:, : c.vdim, : c.kv_rank] = t["uv"].view(H, c.vdim, c.kv_rank)
        self.w_uv = put(uv)                                          # [h, vdim, latent]: latent outputs to values
        # prompts project latents up to keys and values where the sizes are those of the kernel
        self.projects = c.projects and self.w_uk.is_cuda and dtype == torch.bfloat16
        self.sink = put(t["sink"], torch.float32) if c.sink else None
        self.w_o = put(pad_to(pad_heads(t["o"].t().contiguous(), H, c.vdim, vp).t(), width_pad, gemm_k(H * vp)))

    def __call__(self, x, lin, cache, cos_sin, positions, slots, block_table, q_start, q_len, kv_len, one_token: bool,
                 plan: Optional["PromptPlan"] = None):
        """x [T, width] -> [T, width]; ``cache`` [pages, page, >= cache_width] is this layer's (or the shared) plane.
        ``plan``: :func:`prompt_plan` of the step for this layer's window."""
        c, T = self.cfg, x.shape[0]
        H, dp, Dp, Rp = c.heads, up64(c.dim), rot_pad(c.rot_dim), latent_pad(c.kv_rank)
        px = lin(x, self.w_in)
        c_q = torch.empty(T, self.q_pad, dtype=x.dtype, device=x.device)
        latent_post_down(self, px, c_q, positions, cos_sin, slots, cache)
        q = lin(c_q, self.w_uq)                                      # [T, h * (dim | rotated)]
        rotate_heads(q[:, dp:], H, c.head_width, c.rot_dims, c.interleaved, positions, cos_sin)
        q_rope = q.view(T, H, c.head_width)[:, :, dp:]
        gate = px[:, self.g_off: self.g_off + H] if c.head_gate else None
        width = H * c.vdim_pad
        o = torch.empty(T, self.w_o.shape[1], dtype=x.dtype, device=x.device)
        if o.shape[1] != width:
            o[:, width:].zero_()
        if plan is not None and self.projects:
            prompt_attention(plan, q.view(T, H, c.head_width)[:, :, :dp], q_rope, stacked_up(self.w_uk, self.w_uv), cache, block_table, q_start,
                             q_len, kv_len, o, c.scale, self.sink, c.window, gate)
        else:
            q_lat = torch.empty(T, H * Rp, dtype=x.dtype, device=x.device)
            ops.batched_linear_heads(q, self.w_uk, q_lat, c.head_width, Rp)
            o_lat = latent_attention(q_lat.view(T, H, Rp), q_rope, cache, block_table, q_start, q_len, kv_len, c.scale, self.sink,
                                     one_token, c.window, gate)
            ops.batched_linear_heads(o_lat.view(T, H * Rp), self.w_uv, o, Rp, c.vdim_pad)
        if not c.head_gate:
            ops.sigmoid_gate(o, px[:, self.g_off:], width)
        return lin(o, self.w_o)


# ------------------------------------------------------------------ prompts: projected keys and values
PROMPT_ROWS = 16384          # most cache rows of a step whose keys and values are projected (128 heads: 1 GiB of them)
_PER_ROW, _PER_PAIR = 256 * 512, (512 + 64 + 512) - (128 + 64 + 128)


@dataclass
class PromptPlan:
    """Work of a prompt step in the projected form: ``rows`` cache rows, those of sequence s from row ``kv_start[s]`` of
    ``scratch`` rows on (a multiple of 64, the keys of a tile: no tile reads another sequence's rows, whose values a
    product with a probability of zero would let through if they are not finite), and the query tiles of 128 tokens."""
    rows: int
    scratch: int
    kv_start: torch.Tensor
    tile_seq: torch.Tensor
    tile_q0: torch.Tensor


def prompt_scratch_bytes(heads: int, latent: int, T: int, dims_fit: bool = True) -> int:
    """Most scratch of a layer in a prompt step of ``T`` tokens: keys and values, gathered rows, stacked weights."""
    if T < 256 or not dims_fit:
        return 0
    return 2 * (PROMPT_ROWS * (2 * heads * 128 + latent + 64) + 2 * heads * 128 * latent)


def prompt_tiles(q_len, kv_len, window: int = 0):
    """(rows, first scratch row of every sequence and the end, tiles' sequences, tiles' first queries) of a step with these
    lengths, or None where the absorbed form is better. A query and a key meet in 320 products a head instead of 1088, but every
    cache row costs 256 x 512 a head first. ``pairs`` are the queries' keys (no more than ``window`` of them each), so the
    products are equal at a ratio of 1; measured at 16, 64 and 128 heads, the projected form takes 0.77 of the time and less from
    a ratio of 0.4 on (256 queries without a cache 39 against 51 us at 16 heads, 46 against 111 at 128), about the same at 0.2 to
    0.35, and more below (300 queries after 15000 cached rows, window 512, ratio 0.06: 135 against 81 and 660 against 269 us)."""
    pairs = 0
    for n, k in zip(q_len, kv_len):
        first, w = k - n, window or k
        short = max(0, min(k, w) - first)                    # queries that see fewer than ``w`` keys
        pairs += short * first + short * (short + 1) // 2 + (n - short) * w
    rows = sum(kv_len)
    if 5 * pairs * _PER_PAIR <= 2 * rows * _PER_ROW:
        return None
    start, seq, q0 = [0], [], []
    for s, (n, k) in enumerate(zip(q_len, kv_len)):
        start.append(start[-1] + -(-k // 64) * 64)
        for t in range(0, n, 128):
            seq.append(s)
            q0.append(t)
    return (rows, start, seq, q0) if start[-1] <= PROMPT_ROWS else None


def prompt_plans(windows, T: int, q_len, kv_len, lengths=None) -> dict:
    """The plan of a step for layers of each window (0: none), where their latents are better projected up to keys and values per
    head. Steps below 256 tokens, captured steps and rows beyond the scratch limit stay absorbed. ``lengths``: (q_len, kv_len) on
    the host; without it both are read back, which waits for all that is queued."""
    if not windows or not q_len.is_cuda or T < 256 or T == q_len.numel() or torch.cuda.is_current_stream_capturing():
        return {}
    if lengths is None:
        lengths = torch.stack((q_len.int(), kv_len.int())).tolist()
    out = {}
    for w in set(windows):
        tiles = prompt_tiles(*lengths, w)
        if tiles is None:
            continue
        rows, start, seq, q0 = tiles
        B, n = len(start) - 1, len(seq)
        # from pinned memory: a copy out of pageable memory would wait for the stream
        buf = torch.tensor(start[:B] + seq + q0, dtype=torch.int32).pin_memory().to(q_len.device, non_blocking=True)
        out[w] = PromptPlan(rows, start[B], buf[:B], buf[B: B + n], buf[B + n:])
    return out


def prompt_plan(T: int, q_len, kv_len, window: int = 0, lengths=None) -> Optional[PromptPlan]:
    """:func:`prompt_plans` of one window."""
    return prompt_plans((window,), T, q_len, kv_len, lengths).get(window)


def stacked_up(w_uk: torch.Tensor, w_uv: torch.Tensor) -> torch.Tensor:
    """[heads * 128 | heads * 128, latent] from ``w_uk`` [heads, latent, 128] and ``w_uv`` [heads, 128, latent]: scratch of one
    layer's step, so that it is never older than the weights."""
    h, R = w_uk.shape[:2]
    if w_uk.is_cuda and w_uk.dtype == torch.bfloat16 and R % 64 == 0 and w_uk.shape[2] == 128:
        out = torch.empty(2 * h * 128, R, dtype=w_uk.dtype, device=w_uk.device)
        _lib().latent_stack(w_uk.contiguous(), w_uv.contiguous(), out)
        return out
    return torch.cat((w_uk.transpose(1, 2).reshape(-1, R), w_uv.reshape(-1, R))).contiguous()


def prompt_attention(plan: PromptPlan, q, q_rope, w_up, cache, block_table, q_start, q_len, kv_len, out, scale, sink=None, window=0, gate=None):
    """q [T, h, 128], q_rope [T, h, 64] (rotated, any strides), cache [pages, page, latent + 64]; out [T, h * 128 ..]."""
    R, L = w_up.shape[1], _lib()
    c = torch.empty(plan.scratch, R, dtype=q.dtype, device=q.device)
    k_rope = torch.empty(plan.scratch, 64, dtype=q.dtype, device=q.device)
    L.latent_gather(cache, block_table, plan.kv_start, kv_len, c, k_rope)
    L.latent_prefill(q, q_rope, ops.linear(c, w_up), k_rope, plan.kv_start, q_start, q_len, kv_len, plan.tile_seq, plan.tile_q0, out, scale,
                     sink=sink, window=window, gate=gate)


def latent_post_down(m: LatentAttention, px, c_q, positions, cos_sin, slots, cache):
    """Query latent normed into ``c_q``; key/value latent normed and its rotated part stored in the tokens' cache rows."""
    c = m.cfg
    Rp, Dp = latent_pad(c.kv_rank), rot_pad(c.rot_dim)
    if px.is_cuda:
        _lib().latent_post_down(px, c.q_rank, m.q_norm, c_q, m.kv_off, c.kv_rank, Rp, m.kv_norm, c.rot_dim, Dp, c.rot_dims,
                                c.interleaved, c.eps, positions, cos_sin, slots, cache if c.own_cache else None)
        return
    rms = lambda t, w: t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + c.eps) * w.float()
    c_q.zero_()
    c_q[:, : c.q_rank] = rms(px[:, : c.q_rank].float(), m.q_norm).to(c_q.dtype)
    if not c.own_cache:
        return
    kv = px[:, m.kv_off: m.kv_off + c.kv_rank + c.rot_dim].float()
    rows = torch.zeros(px.shape[0], Rp + Dp)
    rows[:, : c.kv_rank] = rms(kv[:, : c.kv_rank], m.kv_norm)
    rows[:, Rp: Rp + c.rot_dim] = kv[:, c.kv_rank:]
    rotate_heads(rows[:, Rp:], 1, Dp, c.rot_dims, c.interleaved, positions, cos_sin)
    page = cache.shape[1]
    ok = slots >= 0
    cache[slots[ok] // page, slots[ok] % page, : Rp + Dp] = rows[ok].to(cache.dtype)


def rotate_heads(x, heads, head_stride, dims, interleaved, positions, cos_sin):
    """In place: the first ``dims`` values of every head of ``x`` (head i starts at column ``i * head_stride``)."""
    if x.is_cuda:
        _lib().rotate_heads(x, heads, head_stride, dims, interleaved, positions, cos_sin)
        return
    cs = cos_sin[positions.long()]
    cos, sin = cs[:, : dims // 2], cs[:, dims // 2:]
    for h in range(heads):
        part = x[:, h * head_stride: h * head_stride + dims]
        part.copy_(ops.reference.apply_rope(part.unsqueeze(1), cos, sin, interleaved).squeeze(1))


def latent_attention(q_lat, q_rope, cache, block_table, q_start, q_len, kv_len, scale, sink=None, one_token=False, window=0, gate=None):
    """Absorbed attention over paged latent rows; returns [T, h, latent]. ``gate`` [T, h]: heads are multiplied by its sigmoid."""
    if q_lat.is_cuda:
        out = torch.empty_like(q_lat)
        if q_lat.dtype == torch.bfloat16:
            ops.ensure_mla_split_workspace(q_lat.device)
        _lib().latent_attention(q_lat, q_rope, cache, block_table, q_start, q_len, kv_len, out, scale, sink, one_token,
                                _split_ws(q_lat.device), window=window, gate=gate)
        return out
    T, H, Rp = q_lat.shape
    LD, page = Rp + q_rope.shape[2], cache.shape[1]
    out = torch.zeros_like(q_lat)
    q = torch.cat([q_lat, q_rope], -1).float()
    for s in range(q_len.numel()):
        t0, n, kl = int(q_start[s]), int(q_len[s]), int(kv_len[s])
        k = cache[block_table[s, : (kl + page - 1) // page].long()].reshape(-1, cache.shape[2])[:kl, :LD].float()
        sc = torch.einsum("qhd,kd->hqk", q[t0: t0 + n], k) * scale
        dist = torch.arange(n).unsqueeze(1) + (kl - n) - torch.arange(kl).unsqueeze(0)
        sc = sc.masked_fill((dist < 0) | (dist >= (window or kl)), float("-inf"))
        if sink is not None:
            sc = torch.cat([sc, sink.view(H, 1, 1).expand(H, n, 1)], -1)
        p = torch.softmax(sc, -1)[..., :kl]
        o = torch.einsum("hqk,kd->qhd", p, k[:, :Rp])
        if gate is not None:
            o = o * torch.sigmoid(gate[t0: t0 + n].float()).unsqueeze(2)
        out[t0: t0 + n] = o.to(out.dtype)
    return out
