// Gated delta rule with a decay per key channel or per head, for ragged batches. Per head, with a state S [dim, vdim] in
// fp32:
//   S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// q, k and v pass a short causal convolution and silu first, q and k are unit vectors per head, and o is RMS-normed over
// vdim, scaled by a weight and gated.
//
//   delta_prep_kernel   one warp per (token, piece): convolution + silu of q, k, v (inputs before the step come from the
//                       sequence's convolution state), unit norms, decays g = exp(-exp(A_log) softplus(z + dt_bias)),
//                       beta, k . q. Everything leaves in fp32.
//   delta_scan_kernel   columns of S are independent, so a warp owns 8 or 16 of them: eight lanes share the rows of a
//                       column (each 4 * RL4 of them, in registers), four lane groups hold two or four columns each. A
//                       token costs one pass of decay, two dot products per column reduced together over eight lanes
//                       (o = (gS)^T q + u (k . q) needs no second reduction), and the rank-one update. Token rows are
//                       staged through shared memory with cp.async. The state is read once and written once per launch,
//                       [slot, head, column, row]; sequences of one token are a decode step, for which one CTA owns a
//                       whole head and also applies the output norm and gate. The convolution state is advanced at the
//                       end of this kernel, after every read of it by the first one.
//   head_out_kernel     output norm and gate for longer sequences, one warp per (token, head)
//
// Steps of few tokens, fp32 runs, one decay per head and other widths go token by token. What bounds that is the chain of a token, 650 cycles of
// shared-memory reads, two dot products and three shuffles; bf16 prompts with 128 rows run in chunks (below).
#include <cuda_runtime.h>

#include "../common/api.h"
#include "../common/launch.h"
#include "../common/scalar.cuh"

namespace mb {
namespace delta {

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// two fp32 lanes per 64-bit register: one instruction for two multiply-adds, each rounded like fmaf
struct __align__(16) u64x2 { uint64_t x, y; };
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float sum4(uint64_t a, uint64_t b) {
  float x, y;
  uint64_t c;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(c));
  return x + y;
}

// silu of a convolution output: fp32 runs take the accurate exponential, 16-bit runs the fast one
template <typename T>
__device__ __forceinline__ float conv_act(float z) {
  if constexpr (sizeof(T) == 4) return siluf(z);
  return __fdividef(z, 1.f + __expf(-z));
}

__device__ __forceinline__ float softplusf(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

// factor of the output gate: fp32 runs take the accurate exponential, 16-bit runs (the result is rounded) the fast one
template <typename T>
__device__ __forceinline__ float gate_of(float z, int silu, float mult) {
  if constexpr (sizeof(T) == 4) return mult * (silu ? siluf(z) : sigmoidf(z));
  return __fdividef(silu ? mult * z : mult, 1.f + __expf(-z));
}

// units of the preparation that make decays and step sizes: one per head, or 32 heads together with one decay per head
__device__ __host__ __forceinline__ int decay_units(const MbDelta& p) { return p.z ? p.heads : (p.heads + 31) / 32; }
template <typename T>
__device__ __forceinline__ void head_decay(const MbDelta& p, const T* row, int t, int h) {
  if (h >= p.heads) return;
  const size_t i = static_cast<size_t>(t) * p.heads + h;
  p.g[i] = expf(-expf(p.A_log[h]) * softplusf(ldf(row + p.a_off + h) + p.dt_bias[h]));
  p.beta[i] = sigmoidf(ldf(row + p.b_off + h));
}

template <typename T>
__global__ void __launch_bounds__(256) delta_prep_kernel(const MbDelta p) {
  const int t = blockIdx.x, lane = threadIdx.x & 31;
  const int unit = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int KH = p.kv_heads, H = p.heads, D = p.dim, V = p.vdim, DP = p.dim_pad;
  const int qkC = KH * D, vC = H * V, C = 2 * qkC + vC, W = p.taps;
  const int v_units = (vC + 127) / 128, G = decay_units(p);
  if (unit >= KH + G + v_units) return;
  int s = t;
  if (!p.one_token) {
    int lo = 0, hi = p.B - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.q_start[mid] <= t) lo = mid; else hi = mid - 1;
    }
    s = lo;
  }
  const int off = t - p.q_start[s];
  if (off < 0 || off >= p.q_len[s]) return;      // a row of no sequence
  const T* row = static_cast<const T*>(p.x) + static_cast<size_t>(t) * p.ldx;
  const int slot = p.state_idx[s];
  const float* hist = (slot >= 0 && W > 1 && p.kv_len[s] > p.q_len[s])
                          ? p.conv_state + static_cast<size_t>(slot) * C * (W - 1) : nullptr;
  // channel `ch` of the convolution state, read from column `col` of the projection rows
  auto conv_silu = [&](int ch, int col) {
    const T* w = static_cast<const T*>(p.conv_w) + static_cast<size_t>(ch) * W;
    float acc = 0.f;
    for (int j = 0; j < W; ++j) {
      const int src = off - (W - 1) + j;
      float xv = 0.f;
      if (src >= 0) xv = ldf(row - static_cast<ptrdiff_t>(W - 1 - j) * p.ldx + col);
      else if (hist) xv = hist[static_cast<size_t>(ch) * (W - 1) + (W - 1 + src)];
      acc = fmaf(ldf(w + j), xv, acc);
    }
    return siluf(acc);
  };
  if (unit < KH) {
    float* qo = p.q + (static_cast<size_t>(t) * KH + unit) * DP;
    float* ko = p.k + (static_cast<size_t>(t) * KH + unit) * DP;
    float qq = 0.f, kk = 0.f, kq = 0.f;
    for (int c = lane; c < D; c += 32) {
      const float a = conv_silu(unit * D + c, p.q_off + unit * D + c);
      const float b = conv_silu(qkC + unit * D + c, p.k_off + unit * D + c);
      qq = fmaf(a, a, qq); kk = fmaf(b, b, kk); kq = fmaf(a, b, kq);
      qo[c] = a; ko[c] = b;                        // rescaled below by the same lane
    }
    qq = warp_allsum(qq); kk = warp_allsum(kk); kq = warp_allsum(kq);
    const float iq = 1.f / sqrtf(qq + 1e-6f) / sqrtf(static_cast<float>(D)), ik = 1.f / sqrtf(kk + 1e-6f);
    for (int c = lane; c < DP; c += 32) {
      qo[c] = c < D ? qo[c] * iq : 0.f;
      ko[c] = c < D ? ko[c] * ik : 0.f;
    }
    if (lane == 0) p.kq[static_cast<size_t>(t) * KH + unit] = kq * iq * ik;
  } else if (unit < KH + G && !p.z) {
    head_decay(p, row, t, (unit - KH) * 32 + lane);
  } else if (unit < KH + G) {
    const int h = unit - KH;
    const float a = expf(p.A_log[h]);
    const float* z = p.z + static_cast<size_t>(t) * p.ldz + h * D;
    float* go = p.g + (static_cast<size_t>(t) * H + h) * DP;
    for (int c = lane; c < DP; c += 32) go[c] = c < D ? expf(-a * softplusf(z[c] + p.dt_bias[h * D + c])) : 0.f;
    if (lane == 0) p.beta[static_cast<size_t>(t) * H + h] = sigmoidf(ldf(row + p.b_off + h));
  } else {
    const int c0 = (unit - KH - G) * 128;
    for (int c = c0 + lane; c < min(c0 + 128, vC); c += 32)
      p.v[static_cast<size_t>(t) * vC + c] = conv_silu(2 * qkC + c, p.v_off + c);
  }
}

// The same for key widths up to 128 (a multiple of 4) and W taps known at compile time: a lane owns four neighbouring
// channels, keeps its taps and the convolution window in registers and walks `tile` consecutive tokens.
template <int W>
struct ConvLane {
  float w[W][4];
  float4 win[W];                    // the last W - 1 inputs in win[1..]
  template <typename T>
  __device__ __forceinline__ void taps(const T* p) {     // [4 channels, W]
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int j = 0; j < W; ++j) w[j][c] = ldf(p + c * W + j);
  }
  // inputs before token `off` of its sequence: rows of the step, then the state (`hist` [4 channels, W - 1] or none)
  template <typename T>
  __device__ __forceinline__ void start(const T* x, int ldx, int off, const float* hist) {
#pragma unroll
    for (int j = 0; j < W - 1; ++j) {
      const int src = off - (W - 1) + j;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (src >= 0) {
        v = ld4(x - static_cast<ptrdiff_t>(W - 1 - j) * ldx);
      } else if (hist) {
        const float* h = hist + (W - 1 + src);
        v = make_float4(h[0], h[W - 1], h[2 * (W - 1)], h[3 * (W - 1)]);
      }
      win[j + 1] = v;
    }
  }
  template <typename T>
  __device__ __forceinline__ float4 step(float4 x) {
#pragma unroll
    for (int j = 0; j < W - 1; ++j) win[j] = win[j + 1];
    win[W - 1] = x;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      a.x = fmaf(w[j][0], win[j].x, a.x); a.y = fmaf(w[j][1], win[j].y, a.y);
      a.z = fmaf(w[j][2], win[j].z, a.z); a.w = fmaf(w[j][3], win[j].w, a.w);
    }
    return make_float4(conv_act<T>(a.x), conv_act<T>(a.y), conv_act<T>(a.z), conv_act<T>(a.w));
  }
};

template <typename T, int W>
__global__ void __launch_bounds__(256) delta_prep_fast_kernel(const MbDelta p, int tile) {
  const int lane = threadIdx.x & 31;
  const int unit = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int KH = p.kv_heads, H = p.heads, D = p.dim, V = p.vdim, DP = p.dim_pad;
  const int qkC = KH * D, vC = H * V, C = 2 * qkC + vC;
  const int G = decay_units(p);
  if (unit >= KH + G + (vC + 127) / 128) return;
  const int tb = blockIdx.x * tile, te = min(tb + tile, p.T);
  int s = tb;
  if (!p.one_token) {
    int lo = 0, hi = p.B - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.q_start[mid] <= tb) lo = mid; else hi = mid - 1;
    }
    s = lo;
  }
  const bool is_qk = unit < KH, is_g = !is_qk && unit < KH + G;
  const int c = lane * 4;
  const int v0 = is_qk || is_g ? 0 : (unit - KH - G) * 128;
  const bool on = is_qk || is_g ? c < D : v0 + c < vC;
  const T* w = static_cast<const T*>(p.conv_w);
  const T* xq = static_cast<const T*>(p.x) + (is_qk ? p.q_off + unit * D + c : p.v_off + v0 + c);
  const T* xk = static_cast<const T*>(p.x) + p.k_off + unit * D + c;
  const int ch_a = is_qk ? unit * D + c : 2 * qkC + v0 + c, ch_b = qkC + unit * D + c;
  ConvLane<W> ca, cb;
  if (on && !is_g) ca.taps(w + static_cast<size_t>(ch_a) * W);
  if (on && is_qk) cb.taps(w + static_cast<size_t>(ch_b) * W);
  const bool chan_g = is_g && p.z;
  const float a_log = chan_g ? expf(p.A_log[unit - KH]) : 0.f;
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (chan_g && on) bias = *reinterpret_cast<const float4*>(p.dt_bias + (unit - KH) * D + c);
  const float scale = 1.f / sqrtf(static_cast<float>(D));
  float4 fut_a = make_float4(0.f, 0.f, 0.f, 0.f), fut_b = fut_a;
  if (on && !is_g) fut_a = ld4(xq + static_cast<size_t>(tb) * p.ldx);
  if (on && is_qk) fut_b = ld4(xk + static_cast<size_t>(tb) * p.ldx);
  int end = 0;                       // first token behind the current sequence
  for (int t = tb; t < te; ++t) {
    if (t >= end) {                  // a new sequence (or the first token of the tile)
      if (t > tb) ++s;
      while (s < p.B && p.q_start[s] + p.q_len[s] <= t) ++s;
      if (s >= p.B || p.q_start[s] > t) return;      // rows of no sequence
      end = p.q_start[s] + p.q_len[s];
      if (!is_g && on) {
        const int off = t - p.q_start[s], slot = p.state_idx[s];
        const float* hist = (slot >= 0 && W > 1 && p.kv_len[s] > p.q_len[s])
                                ? p.conv_state + static_cast<size_t>(slot) * C * (W - 1) : nullptr;
        ca.start(xq + static_cast<size_t>(t) * p.ldx, p.ldx, off, hist ? hist + static_cast<size_t>(ch_a) * (W - 1) : nullptr);
        if (is_qk)
          cb.start(xk + static_cast<size_t>(t) * p.ldx, p.ldx, off, hist ? hist + static_cast<size_t>(ch_b) * (W - 1) : nullptr);
      }
    }
    const size_t row = static_cast<size_t>(t) * p.ldx;
    const float4 nxt_a = fut_a, nxt_b = fut_b;
    if (on && t + 1 < te) {          // the next token's inputs travel while this one is worked on
      if (!is_g) fut_a = ld4(xq + row + p.ldx);
      if (is_qk) fut_b = ld4(xk + row + p.ldx);
    }
    if (is_qk) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f), k = q;
      if (on) { q = ca.template step<T>(nxt_a); k = cb.template step<T>(nxt_b); }
      float qq = q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w, kk = k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
      float kq = q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w;
      qq = warp_allsum(qq); kk = warp_allsum(kk); kq = warp_allsum(kq);
      const float iq = scale / sqrtf(qq + 1e-6f), ik = 1.f / sqrtf(kk + 1e-6f);
      const size_t o = (static_cast<size_t>(t) * KH + unit) * DP + c;
      if (c < DP) {
        *reinterpret_cast<float4*>(p.q + o) = make_float4(q.x * iq, q.y * iq, q.z * iq, q.w * iq);
        *reinterpret_cast<float4*>(p.k + o) = make_float4(k.x * ik, k.y * ik, k.z * ik, k.w * ik);
      }
      if (lane == 0) p.kq[static_cast<size_t>(t) * KH + unit] = kq * iq * ik;
    } else if (is_g && !chan_g) {
      head_decay(p, static_cast<const T*>(p.x) + row, t, (unit - KH) * 32 + lane);
    } else if (is_g) {
      const int h = unit - KH;
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on) {
        const float4 z = *reinterpret_cast<const float4*>(p.z + static_cast<size_t>(t) * p.ldz + h * D + c);
        g = make_float4(expf(-a_log * softplusf(z.x + bias.x)), expf(-a_log * softplusf(z.y + bias.y)),
                        expf(-a_log * softplusf(z.z + bias.z)), expf(-a_log * softplusf(z.w + bias.w)));
      }
      if (c < DP) *reinterpret_cast<float4*>(p.g + (static_cast<size_t>(t) * H + h) * DP + c) = g;
      if (lane == 0) p.beta[static_cast<size_t>(t) * H + h] = sigmoidf(ldf(static_cast<const T*>(p.x) + row + p.b_off + h));
    } else if (on) {
      *reinterpret_cast<float4*>(p.v + static_cast<size_t>(t) * vC + v0 + c) = ca.template step<T>(nxt_a);
    }
  }
}

// the last taps - 1 convolution inputs of a sequence of n rows from t0; share `part` of `parts` of the channels. The caller
// passes what it has read: loads of their own at the end of a decode step's scan cost 1.3 us of 39.
template <typename T>
__device__ __forceinline__ void keep_conv_inputs(const MbDelta& p, int n, int t0, int slot, bool resume, int part, int parts) {
  const int W = p.taps, KH = p.kv_heads, H = p.heads, V = p.vdim;
  if (n > 0 && slot >= 0 && W > 1) {
    const int qkC = KH * p.dim, C = 2 * qkC + H * V;
    for (int c = part * blockDim.x + threadIdx.x; c < C; c += parts * blockDim.x) {
      const int col = c < qkC ? p.q_off + c : c < 2 * qkC ? p.k_off + (c - qkC) : p.v_off + (c - 2 * qkC);
      float* cs = p.conv_state + (static_cast<size_t>(slot) * C + c) * (W - 1);
      // ascending order only overwrites entries that have been read: entry i comes from entry i + n
      for (int i = 0; i < W - 1; ++i) {
        const int src = n - (W - 1) + i;           // position within the step
        float x = 0.f;
        if (src >= 0) x = ldf(static_cast<const T*>(p.x) + static_cast<size_t>(t0 + src) * p.ldx + col);
        else if (resume) x = cs[W - 1 + src];
        cs[i] = x;
      }
    }
  }
}

template <typename T, int RL4, int NC, int MAXT, bool FUSE, bool HEADG>
__global__ void __launch_bounds__(MAXT) delta_scan_kernel(const MbDelta p, int col_blocks, int chunk) {
  constexpr int DP = 32 * RL4, NP = HEADG ? 2 : 3, NS = HEADG ? 4 : 2;     // fp32 vectors and scalars per token
  extern __shared__ __align__(16) float sm[];
  __shared__ float red[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rg = lane & 7, cg = lane >> 3;
  const int KH = p.kv_heads, H = p.heads, V = p.vdim;
  const int h = blockIdx.x / col_blocks, cols = (blockDim.x >> 5) * 4 * NC, cbase = (blockIdx.x % col_blocks) * cols;
  const int kh = h / (H / KH), s = blockIdx.y;
  const int t0 = p.q_start[s], n = p.q_len[s], slot = p.state_idx[s];
  const bool resume = slot >= 0 && p.kv_len[s] > n;
  if (n > 0) {
    const int row_floats = NP * DP + cols;         // q | k | (g) | v columns, then beta, k . q (and g) per token
    const int stage_floats = chunk * (row_floats + NS);
    float* so = sm + 2 * stage_floats;             // FUSE: outputs of one token
    auto fetch = [&](int c0, float* dst) {         // every thread walks the tokens of its piece of the row
      const int m = min(chunk, n - c0);
      const size_t t = static_cast<size_t>(t0 + c0);
      for (int pc = tid; pc < NP * DP / 4; pc += blockDim.x) {
        const int which = pc / (DP / 4), c = (pc % (DP / 4)) * 4;
        const float* src = which == 0 ? p.q + (t * KH + kh) * DP : which == 1 ? p.k + (t * KH + kh) * DP : p.g + (t * H + h) * DP;
        src += c;
        const int step = (which == 2 ? H : KH) * DP;
        float* d = dst + pc * 4;
        for (int j = 0; j < m; ++j, src += step, d += row_floats) cp_async16(d, src);
      }
      if (tid < cols && cbase + tid < V) {
        const float* src = p.v + (t * H + h) * V + cbase + tid;
        float* d = dst + NP * DP + tid;
        for (int j = 0; j < m; ++j, src += H * V, d += row_floats) cp_async4(d, src);
      }
      float* sc = dst + chunk * row_floats;
      for (int i = tid; i < NS * m; i += blockDim.x) {
        const int k = i % NS;
        if (k < 3) cp_async4(sc + i, k == 1 ? p.kq + (t + i / NS) * KH + kh : (k == 0 ? p.beta : p.g) + (t + i / NS) * H + h);
      }
      cp_async_commit();
    };
    fetch(0, sm);
    const int col0 = cbase + (warp * 4 + cg) * NC;
    float* st = p.state + ((static_cast<size_t>(slot >= 0 ? slot : 0) * H + h) * V + col0) * DP;
    u64x2 S[NC][RL4];                              // four rows per entry, two packed fp32 pairs
#pragma unroll
    for (int i = 0; i < RL4; ++i)
#pragma unroll
      for (int c = 0; c < NC; ++c)
        S[c][i] = (resume && col0 + c < V) ? *reinterpret_cast<const u64x2*>(st + c * DP + (i * 8 + rg) * 4) : u64x2{0ull, 0ull};
    // which reduced value this lane ends up with: column `mine` of its group, key product or query product
    const bool b4 = (lane & 4) != 0, b2 = (lane & 2) != 0, b1 = (lane & 1) != 0;
    const int mine = NC == 4 ? (b4 ? 2 : 0) + (b2 ? 1 : 0) : (b4 ? 1 : 0);
    const bool is_q = NC == 4 ? b1 : b2;
    const int my_col = (warp * 4 + cg) * NC + mine;
    float* optr = p.o + (static_cast<size_t>(t0) * H + h) * V + cbase + my_col;
    const bool holds_o = NC == 4 ? b1 : (lane & 3) == 2;
    const bool writes = holds_o && cbase + my_col < V;
    for (int c0 = 0, it = 0; c0 < n; c0 += chunk, ++it) {
      const int m = min(chunk, n - c0);
      const float* buf = sm + (it & 1) * stage_floats;
      if (c0 + chunk < n) { fetch(c0 + chunk, sm + ((it + 1) & 1) * stage_floats); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
      __syncthreads();
      const float* sc = buf + chunk * row_floats;
#pragma unroll 2
      for (int j = 0; j < m; ++j) {
        const float* rowp = buf + j * row_floats;
        u64x2 kr[RL4];
        uint64_t a[NC][2], b[NC][2], gh = 0ull;
        if (HEADG) gh = pack2(sc[NS * j + 2], sc[NS * j + 2]);
#pragma unroll
        for (int c = 0; c < NC; ++c) a[c][0] = a[c][1] = b[c][0] = b[c][1] = 0ull;
#pragma unroll
        for (int i = 0; i < RL4; ++i) {
          const int r = (i * 8 + rg) * 4;
          const u64x2 q4 = *reinterpret_cast<const u64x2*>(rowp + r);
          const u64x2 k4 = *reinterpret_cast<const u64x2*>(rowp + DP + r);
          const u64x2 g4 = HEADG ? u64x2{gh, gh} : *reinterpret_cast<const u64x2*>(rowp + 2 * DP + r);
          kr[i] = k4;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            S[c][i].x = mul2(S[c][i].x, g4.x); S[c][i].y = mul2(S[c][i].y, g4.y);
            a[c][0] = fma2(S[c][i].x, k4.x, a[c][0]); a[c][1] = fma2(S[c][i].y, k4.y, a[c][1]);
            b[c][0] = fma2(S[c][i].x, q4.x, b[c][0]); b[c][1] = fma2(S[c][i].y, q4.y, b[c][1]);
          }
        }
        float A[NC], Bq[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) { A[c] = sum4(a[c][0], a[c][1]); Bq[c] = sum4(b[c][0], b[c][1]); }
        // partial sums over the eight row lanes: every exchange halves the values a lane still carries
        float r;
        if (NC == 4) {
          float a2[2], q2[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            a2[c] = (b4 ? A[NC / 2 + c] : A[c]) + __shfl_xor_sync(0xffffffffu, b4 ? A[c] : A[NC / 2 + c], 4);
            q2[c] = (b4 ? Bq[NC / 2 + c] : Bq[c]) + __shfl_xor_sync(0xffffffffu, b4 ? Bq[c] : Bq[NC / 2 + c], 4);
          }
          const float a1 = (b2 ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? a2[0] : a2[1], 2);
          const float q1 = (b2 ? q2[1] : q2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? q2[0] : q2[1], 2);
          r = (b1 ? q1 : a1) + __shfl_xor_sync(0xffffffffu, b1 ? a1 : q1, 1);
        } else {
          const float a1 = (b4 ? A[1] : A[0]) + __shfl_xor_sync(0xffffffffu, b4 ? A[0] : A[1], 4);
          const float q1 = (b4 ? Bq[1] : Bq[0]) + __shfl_xor_sync(0xffffffffu, b4 ? Bq[0] : Bq[1], 4);
          r = (b2 ? q1 : a1) + __shfl_xor_sync(0xffffffffu, b2 ? a1 : q1, 2);
          r += __shfl_xor_sync(0xffffffffu, r, 1);
        }
        const float beta = sc[NS * j], kq = sc[NS * j + 1];
        const float vv = rowp[NP * DP + my_col];
        const float u = beta * (vv - r);           // meaningful in the lanes that hold a key product
        float uc[NC], u_mine = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          uc[c] = __shfl_sync(0xffffffffu, u, (lane & 24) | (NC == 4 ? (c >> 1) * 4 + (c & 1) * 2 : c * 4));
          u_mine = mine == c ? uc[c] : u_mine;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const uint64_t up = pack2(uc[c], uc[c]);
#pragma unroll
          for (int i = 0; i < RL4; ++i) { S[c][i].x = fma2(kr[i].x, up, S[c][i].x); S[c][i].y = fma2(kr[i].y, up, S[c][i].y); }
        }
        const float o = fmaf(u_mine, kq, r);       // in the lanes that hold a query product
        if (FUSE) {
          if (holds_o) so[my_col] = cbase + my_col < V ? o : 0.f;
        } else {
          if (writes) *optr = o;
          optr += H * V;
        }
        if (FUSE) {                                // one CTA holds the whole head (cbase = 0)
          __syncthreads();
          float ss = 0.f;
          for (int c = tid; c < V; c += blockDim.x) ss = fmaf(so[c], so[c], ss);
          ss = warp_allsum(ss);
          if (lane == 0) red[warp] = ss;
          __syncthreads();
          float tot = 0.f;
          for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) tot += red[i];
          const float inv = 1.f / sqrtf(tot / static_cast<float>(V) + p.eps);
          const size_t t = static_cast<size_t>(t0 + c0 + j);
          for (int c = tid; c < V; c += blockDim.x) {
            const float gate = gate_of<T>(ldf(static_cast<const T*>(p.gate) + t * p.ld_gate + h * V + c), p.gate_silu, p.out_mult);
            stf(static_cast<T*>(p.out) + t * p.ld_out + h * V + c, so[c] * inv * ldf(static_cast<const T*>(p.norm_w) + c) * gate);
          }
          __syncthreads();
        }
      }
      __syncthreads();                             // the stage is free again
    }
    if (slot >= 0) {
#pragma unroll
      for (int i = 0; i < RL4; ++i)
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (col0 + c < V) *reinterpret_cast<u64x2*>(st + c * DP + (i * 8 + rg) * 4) = S[c][i];
    }
  }
  keep_conv_inputs<T>(p, n, t0, slot, resume, blockIdx.x, gridDim.x);
}

template <typename T>
__global__ void __launch_bounds__(256) head_out_kernel(const MbHeadOut p) {
  const int V = p.vdim, lane = threadIdx.x & 31;
  const long long unit = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= static_cast<long long>(p.T) * p.heads) return;
  const size_t t = static_cast<size_t>(unit / p.heads);
  const int h = static_cast<int>(unit % p.heads);
  const float* o = p.o + unit * V;
  const T *gate = static_cast<const T*>(p.gate) + t * p.ld_gate + h * V, *w = static_cast<const T*>(p.norm_w) + h * p.w_stride;
  T* out = static_cast<T*>(p.out) + t * p.ld_out + h * V;
  float ss = 0.f;
  if (V <= 256 && V % 4 == 0 && p.ld_gate % 4 == 0 && p.ld_out % 4 == 0 &&
      ((reinterpret_cast<uintptr_t>(p.o) | reinterpret_cast<uintptr_t>(p.gate) | reinterpret_cast<uintptr_t>(p.norm_w) |
        reinterpret_cast<uintptr_t>(p.out)) & 15) == 0) {     // the head stays in registers
    float4 x[2], g[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (lane + 32 * i) * 4;
      x[i] = c < V ? *reinterpret_cast<const float4*>(o + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[i] = c < V ? ld4(gate + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      ss += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
    }
    const float inv = 1.f / sqrtf(warp_allsum(ss) / static_cast<float>(p.n) + p.eps);
    auto f = [&](float z) { return gate_of<T>(z, p.gate_silu, p.mult) * inv; };
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (lane + 32 * i) * 4;
      if (c >= V) continue;
      const float4 a = ld4(w + c);
      st4(out + c, make_float4(x[i].x * a.x * f(g[i].x), x[i].y * a.y * f(g[i].y), x[i].z * a.z * f(g[i].z), x[i].w * a.w * f(g[i].w)));
    }
    return;
  }
  for (int c = lane; c < V; c += 32) ss = fmaf(o[c], o[c], ss);
  const float inv = 1.f / sqrtf(warp_allsum(ss) / static_cast<float>(p.n) + p.eps);
  for (int c = lane; c < V; c += 32) stf(out + c, o[c] * inv * ldf(w + c) * gate_of<T>(ldf(gate + c), p.gate_silu, p.mult));
}

template <typename T>
static int head_out(const MbHeadOut& p, cudaStream_t stream) {
  const long long units = static_cast<long long>(p.T) * p.heads;
  return launch_plain(head_out_kernel<T>, dim3(static_cast<unsigned>((units + 7) / 8)), dim3(256), 0, stream, p) == cudaSuccess
             ? MB_OK : MB_ERR_LAUNCH;
}

template <typename T, int RL4, int NC, bool HEADG>
static int scan_launch(const MbDelta& p, int warps, bool fuse, cudaStream_t stream) {
  constexpr int MAXT = RL4 <= 8 ? 512 : 256;
  const int cols = warps * 4 * NC, col_blocks = (p.vdim + cols - 1) / cols;
  const int per_token = ((HEADG ? 2 : 3) * 32 * RL4 + cols + (HEADG ? 4 : 2)) * 4;
  // tokens per stage: even, so that the second stage stays 16-byte aligned (a one-token step has no second stage)
  int chunk = p.one_token ? 1 : 40 * 1024 / (2 * per_token);
  if (!p.one_token) chunk = chunk > 16 ? 16 : chunk < 2 ? 2 : chunk & ~1;
  const size_t smem = static_cast<size_t>(2) * chunk * per_token + (fuse ? cols * 4 : 0) + 16;
  const dim3 grid(p.heads * col_blocks, p.B);
  if (fuse)
    return launch_plain(delta_scan_kernel<T, RL4, NC, MAXT, true, HEADG>, grid, dim3(warps * 32), smem, stream, p, col_blocks, chunk) ==
                   cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
  if (launch_plain(delta_scan_kernel<T, RL4, NC, MAXT, false, HEADG>, grid, dim3(warps * 32), smem, stream, p, col_blocks, chunk) !=
      cudaSuccess)
    return MB_ERR_LAUNCH;
  const MbHeadOut o = {p.o, p.out, p.ld_out, p.gate, p.ld_gate, p.norm_w, p.T, p.heads, p.vdim, p.vdim, p.gate_silu, p.eps, p.out_mult};
  return head_out<T>(o, stream);
}

template <typename T, int RL4, bool HEADG>
static int scan_by_width(const MbDelta& p, int num_sms, cudaStream_t stream) {
  constexpr int max_warps = (RL4 <= 8 ? 512 : 256) / 32;
  const int head_warps = (p.vdim + 7) / 8;
  if (p.one_token && head_warps <= max_warps) return scan_launch<T, RL4, 2, HEADG>(p, head_warps, true, stream);
  // longer sequences: four columns per lane where the registers allow it (the rows are read once for all of them) and the
  // grid still has two warps per scheduler, two columns otherwise: a token is a chain of some 300 instructions for four
  // columns, and one warp alone issues one in two cycles (four prompts of 3076 tokens at most, 16 heads of 128 x 128:
  // 1151 us with four, 1065 with two). CTAs have up to four warps as long as the grid has one per SM.
  auto fit = [&](int per_warp) {
    const int hw = (p.vdim + per_warp - 1) / per_warp;
    int w = hw < 4 ? hw : 4;
    while (w > 1 && static_cast<long long>(p.B) * p.heads * ((hw + w - 1) / w) < num_sms) w >>= 1;
    return w;
  };
  if constexpr (RL4 <= 4) {
    if (p.vdim >= 16 && static_cast<long long>(p.B) * p.heads * ((p.vdim + 15) / 16) >= 8LL * num_sms)
      return scan_launch<T, RL4, 4, HEADG>(p, fit(16), false, stream);
  }
  return scan_launch<T, RL4, 2, HEADG>(p, fit(8), false, stream);
}

template <typename T, int RL4>
static int scan(const MbDelta& p, int num_sms, cudaStream_t stream) {
  return p.z ? scan_by_width<T, RL4, false>(p, num_sms, stream) : scan_by_width<T, RL4, true>(p, num_sms, stream);
}

// ---- bf16 prompts, sixteen tokens at a time
// With b_t the running product of a chunk's decays, S the state before it and L the strictly lower triangle:
//   A = L(beta_t k_t diag(b_t / b_j) k_j),  u = (1 + A)^-1 beta (v - (b k) S),  o = (b q) S + (q diag(b_t / b_j) k_j, j <= t) u
//   S <- diag(b_last) S + sum_j (b_last / b_j) k_j u_j
// b_t / b_j is formed as the product of the decays between them where a channel fades far within a chunk: nothing overflows, decays of
// zero stay zeros. delta_chunk_prep_kernel does what needs no state for all chunks at once, two warps a (chunk, head): convolution, norms and
// decays as above, the products of pairs, the inverse by substitution. delta_chunk_scan_kernel walks a sequence's chunks with S in accumulator
// fragments: a warp owns 32 rows of 16 columns of one head; the columns are the M side of every product.
// Products with S and the sums of k_j u_j run on the tensor cores. Their operands enter as three bf16 numbers, which hold all 24 bits whatever lies beside
// them, and six of the nine products of such parts are made: what is left out is below 2^-24 of the whole. Operands travel as fp32 and are taken apart in
// registers. Products with the two small matrices are FMAs, a quarter of the tokens a warp.
// 8192 tokens in four prompts of at most 3076, 16 heads of 128 x 128, prepared, walked and gated: 792 us, token by token 1381; four prompts of 1000 388
// and 544, one of 4000 681 and 1265. (Two tf32 numbers and three products an operand hold 23 bits and leave out 2^-22: 373 and 636 us, but outputs 1.3 to
// 1.5 times as far from their value as token by token. Two fp16 numbers under a power of two per row hold the row's largest entries only. The small matrices
// on the tensor cores as well: 407 and 714.) What bounds it: the walk's chain, which on the SM of the longest prompt uses 74 % of the issue slots, for
// taking operands apart (ALU 40 % on average) more than for products (tensor pipe 34 %); the preparation's instructions, half of the issue slots of the 15
// warps an SM that rows in shared memory leave.
// Error against 64 bits, root mean square, in parts of that token by token: outputs 0.83 without decay, 0.77 to 0.92 with decays near one, 0.96 with usual
// ones, 1.1 to 1.2 (1.5e-7 against 1.3e-7) where little outlasts a token, because the units cut sums off where FMAs round. States 0.64, 0.78 to 0.95, 0.94
// and 0.93 to 1.1.
constexpr int kCh = 16;
constexpr int kRec = 132;          // floats of a chunk's record: b_last [128] and a flag (something in the chunk is not finite)
constexpr int kOrder = 130;        // and in the record i of the first head the sequence that is the i-th by length
constexpr int kRowFloats = 2 * kCh;
constexpr int kChunkCols = 32;     // columns of a scan CTA

// Chunk records of a step: sequence s has chunks (q_start[s] >> 4) + s + i, which never meet another sequence's.
__device__ __forceinline__ int chunk_base(const MbDelta& p, int s) { return (p.q_start[s] >> 4) + s; }

// N values of all lanes to their sums: lane l ends with value l (N = 32) or l / 2 (N = 16)
template <int N>
__device__ __forceinline__ float lanes_reduce(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = N / 2, o = 16; n >= 1; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], o);
  }
  if (N == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float zero_times(float4 a, float acc) { return fmaf(a.x, 0.f, fmaf(a.y, 0.f, fmaf(a.z, 0.f, fmaf(a.w, 0.f, acc)))); }

// A row of the keys that enter the state: of every four channels first 0 and 2, then 1 and 3, which are the neighbours in the
// accumulator tiles of the state.
__device__ __forceinline__ float4 state_key(float4 v) { return make_float4(v.x, v.z, v.y, v.w); }

struct ChunkPrepPair {
  float4 q[kCh][32], k[kCh][32], g[kCh][32];       // rows of 128; a lane works on its four channels
  float A[kCh][kCh];                               // k_t . k_j with the decays between them
  int near, bad[2], fill;
};

__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// Pair `i` of an operand: x and y as sums of three bf16 numbers each, the next one what the rounding before left. All 24 bits.
template <int N>
__device__ __forceinline__ void split(uint32_t (&p)[3][N], int i, float x, float y) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[q][i]) : "f"(y), "f"(x));
    x -= __uint_as_float(p[q][i] << 16);
    y -= __uint_as_float(p[q][i] & 0xffff0000u);
  }
}
// the products of such parts that count, smallest first: the last one is the main part
constexpr int kProducts = 6;
__device__ constexpr int kPartA[kProducts] = {2, 0, 1, 1, 0, 0}, kPartB[kProducts] = {0, 2, 1, 0, 1, 0};

// Loops stay rolled up: a warp runs through every instruction once a chunk, and code that does not fit the instruction cache
// took 67 us for a single chunk.
template <typename T, int W>
__global__ void __launch_bounds__(256, 2) delta_chunk_prep_kernel(const __grid_constant__ MbDelta p, unsigned unit_blocks) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int pair = threadIdx.x >> 6, role = (threadIdx.x >> 5) & 1, lane = threadIdx.x & 31;
  ChunkPrepPair& sm = reinterpret_cast<ChunkPrepPair*>(smem_raw)[pair];
  auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory"); };
  const int H = p.heads, D = p.dim, V = p.vdim;
  constexpr int DP = 128, kBatch = 4;
  if (blockIdx.x >= unit_blocks) {                 // the order of the sequences, longest first
    const int i = (blockIdx.x - unit_blocks) * blockDim.x + threadIdx.x;
    if (i >= p.B) return;
    int ahead = 0;
    const int mine = p.q_len[i];
    for (int j = 0; j < p.B; ++j) ahead += p.q_len[j] > mine || (p.q_len[j] == mine && j < i);
    p.chunk[static_cast<size_t>(ahead) * H * kRec + kOrder] = __int_as_float(i);
    return;
  }
  const long long unit = static_cast<long long>(blockIdx.x) * 4 + pair;
  const int id = static_cast<int>(unit / H), h = static_cast<int>(unit % H);
  int lo = 0, hi = p.B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (chunk_base(p, mid) <= id) lo = mid; else hi = mid - 1;
  }
  const int s = lo, off = (id - chunk_base(p, s)) * kCh;
  if (off < 0 || off >= p.q_len[s]) return;
  const int m = min(kCh, p.q_len[s] - off);
  const size_t t0 = static_cast<size_t>(p.q_start[s]) + off;
  const int qkC = H * D, C = 2 * qkC + H * V, slot = p.state_idx[s];
  const float* hist = (slot >= 0 && W > 1 && p.kv_len[s] > p.q_len[s]) ? p.conv_state + static_cast<size_t>(slot) * C * (W - 1) : nullptr;
  const int c = lane * 4;
  const bool on = c < D;
  const T* x = static_cast<const T*>(p.x) + t0 * p.ldx;
  float finite = 0.f;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);

  // the rows of a chunk four at a time, the next four on their way
  auto walk = [&](int j_first, int j_end, auto&& load, auto&& use) {
    float4 nxt[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) nxt[j] = load(j_first + j);
#pragma unroll 1
    for (int j0 = j_first; j0 < j_end; j0 += kBatch) {
      float4 cur[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) { cur[j] = nxt[j]; nxt[j] = load(j0 + kBatch + j); }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) use(j0 + j, cur[j]);
    }
  };
  // decays (a half of the tokens each) and step sizes
  const float beta = lane < m ? sigmoidf(ldf(x + static_cast<size_t>(lane) * p.ldx + p.b_off + h)) : 0.f;
  {
    const float a_log = expf(p.A_log[h]);
    const float4 bias = on ? *reinterpret_cast<const float4*>(p.dt_bias + h * D + c) : zero;
    const float* z = p.z + t0 * p.ldz + h * D + c;
    auto f = [&](float v) { return expf(-a_log * softplusf(v)); };
    walk(8 * role, 8 * role + 8, [&](int j) { return on && j < m ? *reinterpret_cast<const float4*>(z + static_cast<size_t>(j) * p.ldz) : zero; },
         [&](int j, float4 v) {
           float4 g = make_float4(f(v.x + bias.x), f(v.y + bias.y), f(v.z + bias.z), f(v.w + bias.w));
           if (!on) g = zero;
           if (j >= m) g = make_float4(1.f, 1.f, 1.f, 1.f);
           sm.g[j][lane] = g;
         });
  }
  // keys, queries, values: convolution and silu; unit keys and queries
#pragma unroll 1
  for (int part = role; part < (role == 0 ? 1 : 2 + (V + 127) / 128); ++part) {       // keys; queries and values
    const int v0 = c + (part - 2) * 128;
    const bool mine = part < 2 ? on : v0 < V;
    const int col = part == 0 ? p.k_off + h * D + c : part == 1 ? p.q_off + h * D + c : p.v_off + h * V + v0;
    const int ch = part == 0 ? qkC + h * D + c : part == 1 ? h * D + c : 2 * qkC + h * V + v0;
    float4 (*rows)[32] = part == 0 ? sm.k : sm.q;
    if (mine) {
      ConvLane<W> cl;
      cl.taps(static_cast<const T*>(p.conv_w) + static_cast<size_t>(ch) * W);
      cl.start(x + col, p.ldx, off, hist ? hist + static_cast<size_t>(ch) * (W - 1) : nullptr);
      walk(0, kCh, [&](int j) { return j < m ? ld4(x + static_cast<size_t>(j) * p.ldx + col) : zero; },
           [&](int j, float4 v) {
             float4 y = cl.template step<T>(v);
             if (j >= m) y = zero;
             if (part < 2) rows[j][lane] = y;
             else if (j < m) {
               finite = zero_times(y, finite);
               *reinterpret_cast<float4*>(p.v + ((t0 + j) * H + h) * V + v0) = y;
             }
           });
    } else if (part < 2) {
#pragma unroll 4
      for (int j = 0; j < kCh; ++j) rows[j][lane] = zero;
    }
    if (part < 2) {
      float ss[kCh];
#pragma unroll
      for (int j = 0; j < kCh; ++j) {
        const float4 y = rows[j][lane];
        ss[j] = y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w;
      }
      const float f = (part == 0 ? 1.f : 1.f / sqrtf(static_cast<float>(D))) / sqrtf(lanes_reduce(ss) + 1e-6f);     // token lane / 2
#pragma unroll 4
      for (int j = 0; j < kCh; ++j) {
        const float fj = __shfl_sync(0xffffffffu, f, 2 * j);
        const float4 y = rows[j][lane];
        rows[j][lane] = make_float4(y.x * fj, y.y * fj, y.z * fj, y.w * fj);
      }
    }
  }
  // what meets the state: k_j with the decays behind it, b_t k_t, b_t q_t
  float* rec = p.chunk + (static_cast<size_t>(id) * H + h) * kRec;
  // a token's row of the inverse and of the query products
  float* rows = p.chunk_rows + (t0 * H + h) * kRowFloats;
  const size_t rstep = static_cast<size_t>(H) * kRowFloats;
  const size_t step = static_cast<size_t>(H) * DP, first = (t0 * H + h) * DP + c;
  {
    bool odd = beta * 0.f != 0.f || finite != 0.f;               // true for NaN
#pragma unroll 4
    for (int j = 0; j < kCh; ++j) {
      const float4 a = role == 0 ? sm.k[j][lane] : sm.q[j][lane];
      odd = odd || zero_times(a, 0.f) != 0.f;
      if ((j >> 3) == role) odd = odd || zero_times(sm.g[j][lane], 0.f) != 0.f;
    }
    odd = __any_sync(0xffffffffu, odd);
    if (lane == 0) sm.bad[role] = odd;
  }
  pair_sync();                     // decays are there
  const bool bad = sm.bad[0] || sm.bad[1];         // something is not finite
  // Decays relative to the chunk's start are enough as long as no channel fades below 1e-15 in it (their inverses stay far from
  // the largest number, products keep their relative error); otherwise pairs take the product of the decays between them.
  const float4 ones = make_float4(1.f, 1.f, 1.f, 1.f);
  float4 run = ones;
  if (role == 0) {
#pragma unroll 4
    for (int j = kCh - 1; j >= 0; --j) {
      if (j < m) *reinterpret_cast<float4*>(p.g + first + j * step) = state_key(mul4(run, sm.k[j][lane]));
      run = mul4(run, sm.g[j][lane]);
    }
    *reinterpret_cast<float4*>(rec + c) = run;
    const float fade = fminf(fminf(run.x, run.y), fminf(run.z, run.w));
    const bool ok = __all_sync(0xffffffffu, !on || fade >= 1e-15f);
    if (lane == 0) sm.near = ok;
    run = ones;
#pragma unroll 4
    for (int j = 0; j < kCh; ++j) {
      run = mul4(run, sm.g[j][lane]);
      if (j < m) *reinterpret_cast<float4*>(p.k + first + j * step) = mul4(run, sm.k[j][lane]);
      if (ok) sm.g[j][lane] = run;                 // from here on the running product
    }
  }
  pair_sync();                     // queries and running products are there
  const bool near = sm.near;
  if (role == 1) {
#pragma unroll 4
    for (int j = 0; j < kCh; ++j) {
      run = near ? sm.g[j][lane] : mul4(run, sm.g[j][lane]);
      if (j < m) *reinterpret_cast<float4*>(p.q + first + j * step) = mul4(run, sm.q[j][lane]);
    }
  }
  if (near) {
    // (b k) or (b q) times (k / b)^T: rows are tokens t, columns tokens j <= t
    const int g = lane >> 2, t = lane & 3;
    const float4 (*left)[32] = role == 0 ? sm.k : sm.q;
    float acc[2][4], low[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[n][e] = low[n][e] = 0.f;
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      uint32_t a[3][4], b[2][3][2];
      // channels 4 t and 4 t + 1 of the sixteen are neighbours in the products, 4 t + 2 and 4 t + 3 the other two of a lane
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float4 d = sm.g[8 * n + g][4 * i + t], k = sm.k[8 * n + g][4 * i + t], x = left[8 * n + g][4 * i + t];
        const bool in = 16 * i + 4 * t < D;
        split(b[n], 0, in ? __fdividef(k.x, d.x) : 0.f, in ? __fdividef(k.y, d.y) : 0.f);
        split(b[n], 1, in ? __fdividef(k.z, d.z) : 0.f, in ? __fdividef(k.w, d.w) : 0.f);
        split(a, n, x.x * d.x, x.y * d.y);
        split(a, 2 + n, x.z * d.z, x.w * d.w);
      }
#pragma unroll
      for (int q = 0; q < kProducts; ++q)
#pragma unroll
        for (int n = 0; n < 2; ++n) mma16(q + 1 < kProducts ? low[n] : acc[n], a[kPartA[q]], b[n][kPartB[q]]);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int tt = 8 * r + g, j = 8 * n + 2 * t;
        float2 y = make_float2(acc[n][2 * r] + low[n][2 * r], acc[n][2 * r + 1] + low[n][2 * r + 1]);
        if (role == 0) {
          *reinterpret_cast<float2*>(&sm.A[tt][j]) = y;
        } else {
          if (j > tt) y.x = 0.f;
          if (j + 1 > tt) y.y = 0.f;
          if (tt < m) *reinterpret_cast<float2*>(rows + tt * rstep + kCh + j) = y;
        }
      }
  } else {
    const float4 (*left)[32] = role == 0 ? sm.k : sm.q;
#pragma unroll 1
    for (int j = 0; j < m; ++j) {
      float4 w = sm.k[j][lane];
#pragma unroll 1
      for (int t = j; t < m; ++t) {
        if (t > j) w = mul4(w, sm.g[t][lane]);
        const float4 x = left[t][lane];
        const float y = warp_allsum(w.x * x.x + w.y * x.y + w.z * x.z + w.w * x.w);
        if (role == 0) {
          if (lane == 0) sm.A[t][j] = y;
        } else {
          if (lane == 0) {
            rows[t * rstep + kCh + j] = y;
            if (t > j) rows[j * rstep + kCh + t] = 0.f;
          }
        }
      }
      if (role == 1 && lane >= m && lane < kCh) rows[j * rstep + kCh + lane] = 0.f;
    }
  }
  __syncwarp();
  // lane l: column l of (1 + A)^-1 beta, zeros above the diagonal
  if (role == 0) {
    float xi[kCh];
#pragma unroll
    for (int i = 0; i < kCh; ++i) {
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j)
        if (j >= lane) sum = fmaf(sm.A[i][j], xi[j], sum);
      const float bi = __shfl_sync(0xffffffffu, beta, i);
      xi[i] = i == lane ? 1.f : i > lane ? -bi * sum : 0.f;
      if (lane < kCh && i < m) rows[i * rstep + lane] = i >= lane ? xi[i] * beta : 0.f;
    }
  }
  if (lane == 0 && role == 0) rec[128] = bad ? 1.f : 0.f;
}

constexpr int kScanWarps = 8;      // two groups of 16 columns, four warps each: a warp has 32 of the 128 rows of its columns
constexpr int kKeyRow = 576, kStateRow = 528, kMatRow = 40, kVRow = kChunkCols + 4, kURow = 24;   // bytes, bytes, then floats: rows that are read together lie in other banks
struct ChunkStage {
  uint8_t k[kCh * kKeyRow], q[kCh * kKeyRow], g[kCh * kStateRow];
  float mat[kCh * kMatRow], v[kCh * kVRow], rec[kRec];
};
struct ChunkScanSmem {
  ChunkStage stage[2];
  float4 part[kScanWarps][4][32];                                // what a warp's rows say about keys and queries
  float u[2][16][kURow];                                         // u of a column group, a row a column
  float2 y[2][kScanWarps][2][8];                                 // delta_chunk_plain: the same for one token
};
static_assert(sizeof(ChunkStage) % 16 == 0 && sizeof(ChunkScanSmem) <= 112 * 1024, "two CTAs an SM");

// the four warps of a column group
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

// The same chunk without matrix products, where zeros beside infinities or NaN would reach tokens before them. Operands come
// from memory again; lane (g, t) of a warp has its rows of columns g and g + 8, as in the scan.
__device__ __noinline__ void delta_chunk_plain(const MbDelta& p, ChunkScanSmem& sm, float (&S)[4][4], size_t row, const float* rec, int col0, int m) {
  constexpr int DP = 128;
  const int warp = threadIdx.x >> 5, group = warp >> 2, ks = warp & 3;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, H = p.heads, V = p.vdim;
  // rows r and u of this warp's columns take the place of its products: nobody reads those once the group has met below
  float *r = reinterpret_cast<float*>(sm.part[warp]), *u = r + kCh * 16;
  auto with_state = [&](const float* x, float (&y)[2]) {         // x . S over this warp's rows
    y[0] = y[1] = 0.f;
    for (int i = 0; i < 2; ++i) {
      const float4 a = *reinterpret_cast<const float4*>(x + 32 * ks + 16 * i + 4 * t);
#pragma unroll
      for (int e = 0; e < 2; ++e)
        y[e] = fmaf(a.x, S[2 * i][2 * e], fmaf(a.y, S[2 * i][2 * e + 1], fmaf(a.z, S[2 * i + 1][2 * e], fmaf(a.w, S[2 * i + 1][2 * e + 1], y[e]))));
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      y[e] += __shfl_xor_sync(0xffffffffu, y[e], 1);
      y[e] += __shfl_xor_sync(0xffffffffu, y[e], 2);
    }
  };
  for (int i = 0; i < m; ++i) {
    const size_t at = row + static_cast<size_t>(i) * H;
    float a[2], b[2];
    with_state(p.k + at * DP, a);
    with_state(p.q + at * DP, b);
    if (t < 2) sm.y[i & 1][warp][t][g] = t ? make_float2(b[0], b[1]) : make_float2(a[0], a[1]);
    group_sync(group);
    if (t < 2) {                   // column g + 8 t, by all four warps
      const float* mi = p.chunk_rows + at * kRowFloats;
      const int c = g + 8 * t, col = col0 + c;
      float kx = 0.f, o = 0.f;
      for (int w = 0; w < 4; ++w) {
        const float2 x = sm.y[i & 1][4 * group + w][0][g], z = sm.y[i & 1][4 * group + w][1][g];
        kx += t ? x.y : x.x;
        o += t ? z.y : z.x;
      }
      r[i * 16 + c] = (col < V ? p.v[at * V + col] : 0.f) - kx;
      float x = 0.f;
      for (int j = 0; j <= i; ++j) x = fmaf(mi[j], r[j * 16 + c], x);
      u[i * 16 + c] = x;
      for (int j = 0; j <= i; ++j) o = fmaf(mi[kCh + j], u[j * 16 + c], o);
      if (ks == 0 && col < V) p.o[at * V + col] = o;
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = 32 * ks + 16 * i + 4 * t;
    const float4 d = *reinterpret_cast<const float4*>(rec + c);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      S[2 * i][2 * e] *= d.x; S[2 * i][2 * e + 1] *= d.y; S[2 * i + 1][2 * e] *= d.z; S[2 * i + 1][2 * e + 1] *= d.w;
    }
    for (int j = 0; j < m; ++j) {
      const float4 k = state_key(*reinterpret_cast<const float4*>(p.g + (row + static_cast<size_t>(j) * H) * DP + c));
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x = u[j * 16 + g + 8 * e];
        S[2 * i][2 * e] = fmaf(k.x, x, S[2 * i][2 * e]); S[2 * i][2 * e + 1] = fmaf(k.y, x, S[2 * i][2 * e + 1]);
        S[2 * i + 1][2 * e] = fmaf(k.z, x, S[2 * i + 1][2 * e]); S[2 * i + 1][2 * e + 1] = fmaf(k.w, x, S[2 * i + 1][2 * e + 1]);
      }
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(on ? 16 : 0)
               : "memory");
}
template <typename T>
__global__ void __launch_bounds__(kScanWarps * 32, 2) delta_chunk_scan_kernel(const __grid_constant__ MbDelta p, int col_blocks, int num_sms) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  ChunkScanSmem& sm = *reinterpret_cast<ChunkScanSmem*>(smem_raw);
  constexpr int DP = 128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, group = warp >> 2, ks = warp & 3;
  const int H = p.heads, V = p.vdim;
  // The longest sequences first, and where some SMs get a second CTA, the longest to the SMs with one and the shortest beside the
  // longest of the others: a walk over 192 chunks beside another of its length takes twice its time.
  const int per_seq = H * col_blocks, all = gridDim.x, place = blockIdx.x, more = all - num_sms;
  int rank = place;
  if (more > 0 && more <= num_sms) rank = place < more ? num_sms - more + place : place < num_sms ? place - more : all - 1 - (place - num_sms);
  const int s = __float_as_int(p.chunk[static_cast<size_t>(rank / per_seq) * H * kRec + kOrder]), part = rank % per_seq;
  const int h = part / col_blocks, cbase = (part % col_blocks) * kChunkCols;
  const int t0 = p.q_start[s], n = p.q_len[s], slot = p.state_idx[s];
  const bool resume = slot >= 0 && p.kv_len[s] > n;
  if (n > 0) {
    // this thread's pieces of a chunk: rows tid / 32 and 8 more of keys and queries, and one of the values or of the small matrices
    const int fj = tid >> 5, fc = tid & 31, vj = (tid & 127) >> 3, vc = (tid & 7) * 4;
    const size_t head = static_cast<size_t>(t0) * H + h, half = static_cast<size_t>(8) * H * DP;
    size_t at = (head + static_cast<size_t>(fj) * H) * DP + fc * 4;
    const float* mat = p.chunk_rows + (head + static_cast<size_t>(vj) * H) * kRowFloats + vc;
    const float* val = p.v + (head + static_cast<size_t>(vj) * H) * V + cbase + vc;
    const float* rec = p.chunk + (static_cast<size_t>(chunk_base(p, s)) * H + h) * kRec + tid * 4;
    auto fetch = [&](int c0) {
      ChunkStage& d = sm.stage[(c0 / kCh) & 1];
      const int m = n - c0;        // rows behind the last one are zeros
      const bool on = fj < m, on8 = fj + 8 < m;
      const size_t a0 = on ? at : 0, a1 = on8 ? at + half : 0;
      cp_async16_zfill(d.k + fj * kKeyRow + fc * 16, p.k + a0, on);
      cp_async16_zfill(d.q + fj * kKeyRow + fc * 16, p.q + a0, on);
      cp_async16_zfill(d.g + fj * kStateRow + fc * 16, p.g + a0, on);
      cp_async16_zfill(d.k + (fj + 8) * kKeyRow + fc * 16, p.k + a1, on8);
      cp_async16_zfill(d.q + (fj + 8) * kKeyRow + fc * 16, p.q + a1, on8);
      cp_async16_zfill(d.g + (fj + 8) * kStateRow + fc * 16, p.g + a1, on8);
      if (tid < 128) {
        const bool von = vj < m && cbase + vc < V;
        cp_async16_zfill(d.v + vj * kVRow + vc, von ? val : p.v, von);
      } else {
        cp_async16_zfill(d.mat + vj * kMatRow + vc, vj < m ? mat : p.chunk_rows, vj < m);
      }
      if (tid < kRec / 4) cp_async16(d.rec + tid * 4, rec);
      cp_async_commit();
      at += 2 * half;
      mat += static_cast<size_t>(kCh) * H * kRowFloats;
      val += static_cast<size_t>(kCh) * H * V;
      rec += static_cast<size_t>(H) * kRec;
    };
    fetch(0);
    // S^T: fragment rows are columns col0 + g and col0 + g + 8; tiles 2 i and 2 i + 1 hold rows r0 + 16 i + 4 t + {0, 1} and {2, 3}
    const int lc = group * 16, col0 = cbase + lc, r0 = 32 * ks;
    float S[4][4];
    float* st = p.state + (static_cast<size_t>(slot >= 0 ? slot : 0) * H + h) * V * DP + r0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = col0 + g + 8 * e;
        const float4 x = resume && col < V ? *reinterpret_cast<const float4*>(st + static_cast<size_t>(col) * DP + 16 * i + 4 * t)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        S[2 * i][2 * e] = x.x; S[2 * i][2 * e + 1] = x.y; S[2 * i + 1][2 * e] = x.z; S[2 * i + 1][2 * e + 1] = x.w;
      }
    for (int c0 = 0; c0 < n; c0 += kCh) {
      const int m = min(kCh, n - c0);
      cp_async_wait<0>();
      __syncthreads();             // the chunk is here, and nobody reads the stage of the one before
      if (c0 + kCh < n) fetch(c0 + kCh);           // travels while this chunk is worked on
      const ChunkStage& in = sm.stage[(c0 / kCh) & 1];
      bool plain = in.rec[128] != 0.f;             // something is not finite
      uint32_t up[3][4];           // u of all sixteen tokens: the left side of two products
      if (!plain) {
        // what the state says about keys and queries: tiles 0, 1 keys of tokens 0-7, 8-15, tiles 2, 3 queries
        float Wm[4][4], Wl[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) Wm[i][e] = Wl[i][e] = 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          // rows 16 i + 4 t and the next one are neighbours in the products, the two behind them the other two of a lane
          uint32_t a[3][4], b[4][3][2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            split(a, 2 * u, S[2 * i + u][0], S[2 * i + u][1]);
            split(a, 2 * u + 1, S[2 * i + u][2], S[2 * i + u][3]);
          }
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const float4 x = *reinterpret_cast<const float4*>((w < 2 ? in.k : in.q) + ((w & 1) * 8 + g) * kKeyRow + (r0 + 16 * i + 4 * t) * 4);
            split(b[w], 0, x.x, x.y);
            split(b[w], 1, x.z, x.w);
          }
          // products that follow one another go to different accumulators
#pragma unroll
          for (int q = 0; q < kProducts; ++q)
#pragma unroll
            for (int w = 0; w < 4; ++w) mma16(q + 1 < kProducts ? Wl[w] : Wm[w], a[kPartA[q]], b[w][kPartB[q]]);
        }
#pragma unroll
        for (int w = 0; w < 4; ++w)
          sm.part[warp][w][lane] = make_float4(Wm[w][0] + Wl[w][0], Wm[w][1] + Wl[w][1], Wm[w][2] + Wl[w][2], Wm[w][3] + Wl[w][3]);
        group_sync(group);
        auto whole = [&](int w) {  // the four warps' parts, always in one order
          const float4 a = sm.part[4 * group][w][lane], b = sm.part[4 * group + 1][w][lane], c = sm.part[4 * group + 2][w][lane],
                       d = sm.part[4 * group + 3][w][lane];
          return make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z), (a.w + b.w) + (c.w + d.w));
        };
        // Products with the small matrices, in FMAs: warp ks makes tokens 8 (ks / 2) + 2 i + ks % 2, of which lane t ends with i = t, from sixteen
        // tokens of columns g and g + 8 spread over the lanes of a column (8 j + 2 t and the next)
        const int tok = 8 * (ks >> 1) + 2 * t + (ks & 1);
        auto small = [&](const float* mat, const float (&x)[2][4], float (&y)[2]) {
          float a[4][2], b[2][2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float* row = mat + (8 * (ks >> 1) + 2 * i + (ks & 1)) * kMatRow + 2 * t;
            const float2 lo = *reinterpret_cast<const float2*>(row), hi = *reinterpret_cast<const float2*>(row + 8);
#pragma unroll
            for (int c = 0; c < 2; ++c) a[i][c] = fmaf(hi.y, x[1][2 * c + 1], fmaf(hi.x, x[1][2 * c], fmaf(lo.y, x[0][2 * c + 1], lo.x * x[0][2 * c])));
          }
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int i = 0; i < 2; ++i) b[i][c] = ((t & 2) ? a[2 + i][c] : a[i][c]) + __shfl_xor_sync(0xffffffffu, (t & 2) ? a[i][c] : a[2 + i][c], 2);
            y[c] = ((t & 1) ? b[1][c] : b[0][c]) + __shfl_xor_sync(0xffffffffu, (t & 1) ? b[0][c] : b[1][c], 1);
          }
        };
        // u = M r, which all four warps need for their rows of the state
        float U[2][4], y[2];
        float finite = 0.f;        // 1.01: what would not be finite as a bf16 counts, too
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 w = whole(j);
          const float wj[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            U[j][e] = in.v[(8 * j + 2 * t + (e & 1)) * kVRow + lc + g + 8 * (e >> 1)] - wj[e];
            finite = fmaf(U[j][e] * 1.01f, 0.f, finite);
          }
        }
        small(in.mat, U, y);
        sm.u[group][g][tok] = y[0];
        sm.u[group][g + 8][tok] = y[1];
        group_sync(group);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const float2 u = *reinterpret_cast<const float2*>(&sm.u[group][g + 8 * c][8 * j + 2 * t]);
            finite = fmaf(u.x * 1.01f, 0.f, fmaf(u.y * 1.01f, 0.f, finite));
            U[j][2 * c] = u.x; U[j][2 * c + 1] = u.y;
            split(up, 2 * j + c, u.x, u.y);
          }
        }
        plain = __any_sync(0xffffffffu, finite != 0.f);          // the same in the four warps
        if (!plain) {
          // o = q S + Q u
          const float4 w = whole(2 + (ks >> 1));
          small(in.mat + kCh, U, y);
          float* o = p.o + (static_cast<size_t>(t0 + c0 + tok) * H + h) * V + col0 + g;
          if (tok < m && col0 + g < V) o[0] = ((ks & 1) ? w.y : w.x) + y[0];
          if (tok < m && col0 + g + 8 < V) o[8] = ((ks & 1) ? w.w : w.z) + y[1];
        }
      }
      if (!plain) {
        // S <- diag(b_last) S + sum_j k_j u_j; the sum has its own accumulators, so that S itself is rounded once a chunk
        float d[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) d[i][e] = 0.f;
        // rows of the tiles 2 i and 2 i + 1 side by side, of tokens 2 t, 2 t + 1 and 8 more
        uint32_t b[4][3][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint8_t* at = in.g + (8 * j + 2 * t) * kStateRow + (r0 + 16 * i + 2 * g) * 4;
            const float2 x = *reinterpret_cast<const float2*>(at), y = *reinterpret_cast<const float2*>(at + kStateRow);
            split(b[2 * i], j, x.x, y.x);
            split(b[2 * i + 1], j, x.y, y.y);
          }
#pragma unroll
        for (int q = 0; q < kProducts; ++q)
#pragma unroll
          for (int i = 0; i < 4; ++i) mma16(d[i], up[kPartA[q]], b[i][kPartB[q]]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 f = *reinterpret_cast<const float4*>(in.rec + r0 + 16 * i + 4 * t);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            S[2 * i][2 * e] = fmaf(S[2 * i][2 * e], f.x, d[2 * i][2 * e]);
            S[2 * i][2 * e + 1] = fmaf(S[2 * i][2 * e + 1], f.y, d[2 * i][2 * e + 1]);
            S[2 * i + 1][2 * e] = fmaf(S[2 * i + 1][2 * e], f.z, d[2 * i + 1][2 * e]);
            S[2 * i + 1][2 * e + 1] = fmaf(S[2 * i + 1][2 * e + 1], f.w, d[2 * i + 1][2 * e + 1]);
          }
        }
      } else {
        float copy[4][4];          // the state itself stays in registers
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) copy[i][e] = S[i][e];
        delta_chunk_plain(p, sm, copy, static_cast<size_t>(t0 + c0) * H + h, in.rec, col0, m);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[i][e] = copy[i][e];
      }
    }
    if (slot >= 0) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = col0 + g + 8 * e;
          if (col < V)
            *reinterpret_cast<float4*>(st + static_cast<size_t>(col) * DP + 16 * i + 4 * t) =
                make_float4(S[2 * i][2 * e], S[2 * i][2 * e + 1], S[2 * i + 1][2 * e], S[2 * i + 1][2 * e + 1]);
        }
    }
  }
  {
    const int rows = p.q_len[s], at = p.state_idx[s];   // read again: the walk has no registers to spare for them
    keep_conv_inputs<T>(p, rows, p.q_start[s], at, at >= 0 && p.kv_len[s] > rows, part, per_seq);
  }
}

template <typename T, int W>
static int chunk_launch(const MbDelta& p, int num_sms, cudaStream_t stream) {
  static PerDeviceOnce once;
  const size_t prep = 4 * sizeof(ChunkPrepPair), scan = sizeof(ChunkScanSmem);
  if (once.needed()) {
    if (cudaFuncSetAttribute(delta_chunk_prep_kernel<T, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(prep)) != cudaSuccess ||
        cudaFuncSetAttribute(delta_chunk_scan_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(scan)) != cudaSuccess)
      return MB_ERR_LAUNCH;
    once.done();
  }
  const long long units = (static_cast<long long>(p.T) / kCh + p.B + 1) * p.heads;
  const unsigned unit_blocks = static_cast<unsigned>((units + 3) / 4);
  if (launch_plain(delta_chunk_prep_kernel<T, W>, dim3(unit_blocks + (p.B + 255) / 256), dim3(256), prep, stream, p, unit_blocks) != cudaSuccess)
    return MB_ERR_LAUNCH;
  const int col_blocks = (p.vdim + kChunkCols - 1) / kChunkCols;
  if (launch_plain(delta_chunk_scan_kernel<T>, dim3(p.heads * col_blocks * p.B), dim3(kScanWarps * 32), scan, stream, p, col_blocks, num_sms) != cudaSuccess)
    return MB_ERR_LAUNCH;
  const MbHeadOut o = {p.o, p.out, p.ld_out, p.gate, p.ld_gate, p.norm_w, p.T, p.heads, p.vdim, p.vdim, p.gate_silu, p.eps, p.out_mult};
  return head_out<T>(o, stream);
}

template <typename T>
static int run(const MbDelta& p, int num_sms, cudaStream_t stream) {
  const int vC = p.heads * p.vdim;
  const int units = p.kv_heads + decay_units(p) + (vC + 127) / 128;
  // vector loads: four channels per lane, every row and block start aligned to them
  const bool fast = p.dim <= 128 && p.dim % 4 == 0 && vC % 4 == 0 && p.taps >= 2 && p.taps <= 4 && p.ldx % 8 == 0 &&
                    p.q_off % 8 == 0 && p.k_off % 8 == 0 && p.v_off % 8 == 0 && (!p.z || p.ldz % 4 == 0) &&
                    ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.z) | reinterpret_cast<uintptr_t>(p.v) |
                      reinterpret_cast<uintptr_t>(p.dt_bias)) & 15) == 0;
  if constexpr (sizeof(T) == 2) {
    if (fast && p.chunk && ((reinterpret_cast<uintptr_t>(p.chunk) | reinterpret_cast<uintptr_t>(p.chunk_rows)) & 15) == 0)
      return p.taps == 4 ? chunk_launch<T, 4>(p, num_sms, stream) : p.taps == 3 ? chunk_launch<T, 3>(p, num_sms, stream) : chunk_launch<T, 2>(p, num_sms, stream);
  }
  const int tile = p.T <= 4 * p.B ? 1 : 16;
  const dim3 grid((p.T + tile - 1) / tile, (units + 7) / 8);
  cudaError_t e;
  if (fast && p.taps == 4) e = launch_plain(delta_prep_fast_kernel<T, 4>, grid, dim3(256), 0, stream, p, tile);
  else if (fast && p.taps == 3) e = launch_plain(delta_prep_fast_kernel<T, 3>, grid, dim3(256), 0, stream, p, tile);
  else if (fast) e = launch_plain(delta_prep_fast_kernel<T, 2>, grid, dim3(256), 0, stream, p, tile);
  else e = launch_plain(delta_prep_kernel<T>, dim3(p.T, (units + 7) / 8), dim3(256), 0, stream, p);
  if (e != cudaSuccess) return MB_ERR_LAUNCH;
  switch (p.dim_pad / 32) {
    case 1: return scan<T, 1>(p, num_sms, stream);
    case 2: return scan<T, 2>(p, num_sms, stream);
    case 3: return scan<T, 3>(p, num_sms, stream);
    case 4: return scan<T, 4>(p, num_sms, stream);
    case 6: return scan<T, 6>(p, num_sms, stream);
    case 8: return scan<T, 8>(p, num_sms, stream);
    case 16: return scan<T, 16>(p, num_sms, stream);
    default: return MB_ERR_SHAPE;
  }
}

}  // namespace delta
}  // namespace mb

using namespace mb;

// Rows of the state per column: the smallest size the scan kernel is built for (0 = too large).
extern "C" int mb_delta_dim_pad(int dim) {
  const int sizes[] = {32, 64, 96, 128, 192, 256, 512};
  for (int s : sizes)
    if (dim <= s) return s;
  return 0;
}

// Floats of scratch for a step in chunks (records, then rows of pairs); 0 where steps run token by token: fp32 runs, decays per head, shared keys,
// wider heads, and steps of few tokens a sequence, where most of a chunk would be padding. While two CTAs an SM hold all walks, the longest chain is what
// a step waits for, and chunks win from 40 tokens on (16 heads of 128 x 128, us in chunks and token by token: 1 sequence of 40 tokens 48 and 56, of 1000 190 and
// 333, 4 of 40 56 and 62). Beyond, walks share the SMs, and the work counts: 16 of 1000 1327 and 1650; with a walk that took 4 % longer 64 of 40 304 and 267, of
// 100 646 and 617, 128 of 200 2295 and 2344 (heads of 100 x 64, which chunks fill up to 128: 128 of 200 1688 and 1620, 16 of 1000 1101 and 1197). One long
// prompt beside many rows of one token would gain there, too (2000 beside 40: 409 and 878), but the lengths are on the device.
extern "C" long long mb_delta_chunk_floats(int T, int B, int heads, int kv_heads, int dim, int vdim, int head_decay, int dtype) {
  if (dtype != kBf16 || head_decay || heads != kv_heads || mb_delta_dim_pad(dim) != 128 || vdim % 4 || T < 40LL * B) return 0;
  const long long walks = static_cast<long long>(heads) * ((vdim + delta::kChunkCols - 1) / delta::kChunkCols) * B;
  if (walks > 2 * 148 && T < 256LL * B) return 0;
  return (static_cast<long long>(T) / delta::kCh + B + 1) * heads * delta::kRec + static_cast<long long>(T) * heads * delta::kRowFloats;
}

extern "C" int mb_head_norm_gate(const MbHeadOut* p, int dtype, cudaStream_t stream) {
  if (p->T <= 0) return MB_OK;
  if (p->heads <= 0 || p->vdim <= 0 || p->n <= 0 || p->n > p->vdim) return MB_ERR_SHAPE;
  return dtype == kF32 ? delta::head_out<float>(*p, stream) : delta::head_out<__nv_bfloat16>(*p, stream);
}

extern "C" int mb_delta_rule(const MbDelta* p, int dtype, int num_sms, cudaStream_t stream) {
  if (p->T <= 0 || p->B <= 0) return MB_OK;
  if (p->heads <= 0 || p->kv_heads <= 0 || p->heads % p->kv_heads || p->dim <= 0 || p->vdim <= 0 || p->taps < 1 ||
      p->dim_pad != mb_delta_dim_pad(p->dim))
    return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(p->q) | reinterpret_cast<uintptr_t>(p->k) | reinterpret_cast<uintptr_t>(p->g) |
       reinterpret_cast<uintptr_t>(p->state)) & 15)
    return MB_ERR_ALIGN;
  MbDelta d = *p;
  d.chunk_rows = d.chunk ? d.chunk + (static_cast<long long>(d.T) / delta::kCh + d.B + 1) * d.heads * delta::kRec : nullptr;
  return dtype == kF32 ? delta::run<float>(d, num_sms, stream) : delta::run<__nv_bfloat16>(d, num_sms, stream);
}
