// State-space layer kernels for ragged (variable-length) batches: causal depthwise conv1d,
// the Mamba-1 selective scan and the Mamba-2 SSD recurrence, each carrying per-sequence state so the
// same entry serves prefill chunks and single-token decode, and the gated norm of a Mamba-2 block.
//
// Sequences are rows [cu_seqlens[s], cu_seqlens[s+1]) of the token-major inputs. State tensors are
// indexed by `state_idx[s]` (a slot per live request; -1 = no state: start from zero, write nothing),
// are read when `has_init[s]` is non-zero and always written back.
//
//   causal_conv1d_kernel    all tokens at once, 4 channels per thread
//   selective_scan_kernel   walks the tokens; a tile of them is staged in shared memory ahead of its use
//   ssd_scan_kernel         walks the tokens, fp32 state in registers: decode steps, short prompts, odd sizes
//   ssd_chunk_kernel        prompts, 64 tokens at a time on the tensor cores
//
// Reference counterparts: max/kernels/src/state_space/causal_conv1d.mojo (varlen fwd + update),
// selective_scan.mojo (selective_scan_fwd / _update) and the Mamba-2 SSD kernels of the same package,
// wrapped by max/python/max/nn/state_space/.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "../common/api.h"
#include "../common/launch.h"

namespace mb {
namespace ssm {

// x / (1 + e^-x): quotient by an approximate reciprocal and one Newton-Raphson correction from its residual, which leaves it as exact
// as a division (root mean square error over [-4, 4] 5.8e-8 either way, 6.4e-8 without the correction). Both sides are scaled, so that the
// reciprocal stays a normal number as long as e^-x is finite; where the residual is not, x or e^-x is infinite and the quotient stands.
__device__ __forceinline__ float silu(float x) {
  constexpr float kScale = 0.25f;
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
  const float d = fmaf(e, kScale, kScale), n = x * kScale;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r, left = fmaf(-d, q, n);
  return fabsf(left) < INFINITY ? fmaf(left, r, q) : q;
}
__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// A rate of minus infinity (a decay of zero) as the lowest finite one: rows past a sequence's end take steps of zero, and a product of the
// two would be NaN.
__device__ __forceinline__ float finite_rate(float a) { return a < -3.402823466e38f ? -3.402823466e38f : a; }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2e = 1.4426950408889634f;

template <int VEC>
__device__ __forceinline__ void load_bf16(float (&v)[VEC], const __nv_bfloat16* p) {
  if constexpr (VEC == 8) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else if constexpr (VEC == 4) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
    v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
  } else {
    v[0] = __bfloat162float(*p);
  }
}
template <int VEC>
__device__ __forceinline__ void store_bf16(__nv_bfloat16* p, const float (&v)[VEC]) {
  if constexpr (VEC >= 4) {
    uint32_t w[VEC / 2];
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    if constexpr (VEC == 8) *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    else *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
  } else {
    *p = __float2bfloat16(v[0]);
  }
}

// y[t, d] = act(bias[d] + sum_k w[d, k] * x[t - (W-1) + k, d]); tokens before the sequence start come
// from conv_state[slot, d, :] (the last W-1 inputs of the previous chunk). W <= 8.
// Bound by memory: x is read and y written once (and W - 1 rows per tile again, from L2). A thread owns VEC
// channels and the tokens of one tile, so all tiles run at once; blocks whose row is below n_seqs take the
// sequences' first W - 1 tokens instead, the only ones that need the state, and the same thread that reads
// the state writes the new one (one reader, one writer, in order).
// 4099 tokens x 4096 channels, width 4: 1104 us with one thread per channel walking a sequence, 22.6 with tiles whose rows were loaded
// four at a time, 15.3 us with all rows of a tile on their way at once and silu without a division's slow path (10 at the copy rate). A decode step is bound
// by the state, which is read and written in 16-byte pieces: 256 tokens of as many sequences x 4096 channels 11 us (19 with one
// 4-byte access per value, 12 with one thread per channel).
// WHOLE: steps that have whole tiles of one sequence (see the launch).
constexpr int kConvTile = 16;
template <int W, int VEC, bool WHOLE>
__global__ void __launch_bounds__(128) causal_conv1d_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                     const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ y,
                                     float* conv_state, const int* __restrict__ cu_seqlens,
                                     const int* __restrict__ state_idx, const int* __restrict__ has_init,
                                     int n_seqs, int D, int ldx, int ldy, int act) {
  const int d = (blockIdx.y * blockDim.x + threadIdx.x) * VEC, row = blockIdx.x;
  if (d >= D) return;
  float wk[W][VEC], b[VEC], win[W][VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) b[c] = 0.f;
  if (bias) load_bf16<VEC>(b, bias + d);
#pragma unroll
  for (int i = 0; i < W; ++i) {                    // the weights of VEC channels are one run of VEC * W values
    float v[VEC];
    load_bf16<VEC>(v, w + static_cast<size_t>(d) * W + i * VEC);
#pragma unroll
    for (int e = 0; e < VEC; ++e) wk[(i * VEC + e) % W][(i * VEC + e) / W] = v[e];
  }
  // one token: win[W - 1] holds its input, win[0 ..] those before it
  auto emit = [&](int t) {
    float acc[VEC];
#pragma unroll
    for (int c = 0; c < VEC; ++c) {
      acc[c] = b[c];
#pragma unroll
      for (int k = 0; k < W; ++k) acc[c] = fmaf(wk[k][c], win[k][c], acc[c]);
      if (act) acc[c] = silu(acc[c]);
    }
    store_bf16<VEC>(y + static_cast<size_t>(t) * ldy + d, acc);
  };
  auto shift = [&]() {
#pragma unroll
    for (int k = 0; k < W - 1; ++k)
#pragma unroll
      for (int c = 0; c < VEC; ++c) win[k][c] = win[k + 1][c];
  };
  if (row < n_seqs) {
    const int s = row, t0 = cu_seqlens[s], t1 = cu_seqlens[s + 1];
    const int slot = state_idx && conv_state ? state_idx[s] : -1;
    float* st = conv_state + static_cast<size_t>(slot >= 0 ? slot : 0) * D * (W - 1) + static_cast<size_t>(d) * (W - 1);
    const bool resume = slot >= 0 && has_init && has_init[s];
    const int head = min(t1, t0 + W - 1);
    float xs[W - 1][VEC];                          // the tokens, loaded together
#pragma unroll
    for (int k = 0; k < W - 1; ++k)
      if (t0 + k < head) load_bf16<VEC>(xs[k], x + static_cast<size_t>(t0 + k) * ldx + d);
    // the state of VEC channels is one run of VEC * (W - 1) values
    float run[VEC * (W - 1)];
    if (resume) {
      if constexpr (VEC == 4) {
#pragma unroll
        for (int q = 0; q < W - 1; ++q) {
          const float4 f = reinterpret_cast<const float4*>(st)[q];
          run[4 * q] = f.x; run[4 * q + 1] = f.y; run[4 * q + 2] = f.z; run[4 * q + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < VEC * (W - 1); ++q) run[q] = st[q];
      }
    }
#pragma unroll
    for (int k = 0; k < W - 1; ++k)
#pragma unroll
      for (int c = 0; c < VEC; ++c) win[k + 1][c] = resume ? run[c * (W - 1) + k] : 0.f;
#pragma unroll
    for (int c = 0; c < VEC; ++c) win[0][c] = 0.f;
#pragma unroll
    for (int k = 0; k < W - 1; ++k) {
      if (t0 + k >= head) break;
      shift();
#pragma unroll
      for (int c = 0; c < VEC; ++c) win[W - 1][c] = xs[k][c];
      emit(t0 + k);
    }
    if (slot < 0) return;
    if (t1 > head) {                               // the last W - 1 inputs, all of this step
#pragma unroll
      for (int k = 1; k < W; ++k) load_bf16<VEC>(win[k], x + static_cast<size_t>(t1 - W + k) * ldx + d);
    }
#pragma unroll
    for (int k = 0; k < W - 1; ++k)
#pragma unroll
      for (int c = 0; c < VEC; ++c) run[c * (W - 1) + k] = win[k + 1][c];
    if constexpr (VEC == 4) {
#pragma unroll
      for (int q = 0; q < W - 1; ++q) reinterpret_cast<float4*>(st)[q] = make_float4(run[4 * q], run[4 * q + 1], run[4 * q + 2], run[4 * q + 3]);
    } else {
#pragma unroll
      for (int q = 0; q < VEC * (W - 1); ++q) st[q] = run[q];
    }
    return;
  }
  const int lo = (row - n_seqs) * kConvTile, hi = lo + kConvTile;
  int a = 0, z = n_seqs;                           // the first sequence that ends beyond lo
  while (a < z) {
    const int m = (a + z) >> 1;
    if (cu_seqlens[m + 1] > lo) z = m; else a = m + 1;
  }
  for (int s = a; s < n_seqs; ++s) {
    const int t0 = cu_seqlens[s];
    if (t0 >= hi) break;
    const int first = max(lo, t0 + W - 1), last = min(hi, cu_seqlens[s + 1]);
    if (first >= last) continue;
    if (WHOLE && last - first == kConvTile) {     // a whole tile: all of its rows are on their way before the first is used
      uint2 raw[kConvTile + W - 1];
      const __nv_bfloat16* from = x + static_cast<size_t>(first - W + 1) * ldx + d;
#pragma unroll
      for (int k = 0; k < kConvTile + W - 1; ++k) raw[k] = *reinterpret_cast<const uint2*>(from + static_cast<size_t>(k) * ldx);
#pragma unroll
      for (int k = 0; k < kConvTile + W - 1; ++k) {
        shift();
        win[W - 1][0] = __uint_as_float(raw[k].x << 16); win[W - 1][1 % VEC] = __uint_as_float(raw[k].x & 0xffff0000u);
        win[W - 1][2 % VEC] = __uint_as_float(raw[k].y << 16); win[W - 1][3 % VEC] = __uint_as_float(raw[k].y & 0xffff0000u);
        if (k >= W - 1) emit(first + k - (W - 1));
      }
      continue;
    }
#pragma unroll
    for (int k = 1; k < W; ++k) load_bf16<VEC>(win[k], x + static_cast<size_t>(first - W + k) * ldx + d);
#pragma unroll 4
    for (int t = first; t < last; ++t) {
      shift();
      load_bf16<VEC>(win[W - 1], x + static_cast<size_t>(t) * ldx + d);
      emit(t);
    }
  }
}

// Mamba-1 selective scan. Per channel d and state n:
//   dt = softplus(delta[t, d] + dt_bias[d]);  h = exp(dt * A[d, n]) * h + dt * B[t, n] * u[t, d]
//   y[t, d] = sum_n C[t, n] * h + Dskip[d] * u[t, d];   y *= silu(z[t, d]) when z is given
// The recurrence needs one exponential per state and token (all fp32): 268 M of them for 4099 tokens x 4096
// channels x 16 states are 60 us of the special-function units, which is the floor for prompts that fill the chip.
// Eight or four lanes (LPC) share a channel, N / LPC states each in registers, so that a few long sequences still give every SM
// several warps; a CTA walks one sequence for 32 channels. Inputs arrive kScanTile tokens at a time through cp.async,
// one tile ahead; step sizes (softplus) are made once per token and channel by all threads before the walk, and
// the lanes' partial outputs of eight tokens meet in seven or six shuffles (through shared memory, for a pass of their own, they
// took 258 us where these take 218). Rows that are not 16-byte aligned are fetched with plain loads, into the same tiles.
// That prompt (three sequences): 3475 us with one thread per channel and two barriers per token, 218 us so: some 30 instructions a
// token and eight lanes, and the longest sequence alone at the end. Short sequences fetch and convert no more than their tokens
// (in eights): a decode step of 256 sequences x 4096 channels 95 us (137 with eight lanes, 167 with whole tiles of 32).
constexpr int kScanTile = 32, kScanCh = 32;
template <int NS>
__device__ __forceinline__ void load_states(float (&v)[NS], const float* p) {
  if constexpr (NS % 4 == 0) {
#pragma unroll
    for (int i = 0; i < NS; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(p + i);
      v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
    }
  } else if constexpr (NS == 2) {
    const float2 f = *reinterpret_cast<const float2*>(p);
    v[0] = f.x; v[1] = f.y;
  } else {
    v[0] = p[0];
  }
}
template <int N, int LPC>
__global__ void __launch_bounds__(kScanCh * LPC) selective_scan_kernel(const __nv_bfloat16* __restrict__ u, const __nv_bfloat16* __restrict__ delta,
                                      const float* __restrict__ A, const __nv_bfloat16* __restrict__ B,
                                      const __nv_bfloat16* __restrict__ C, const float* __restrict__ Dskip,
                                      const __nv_bfloat16* __restrict__ z, const float* __restrict__ dt_bias,
                                      __nv_bfloat16* __restrict__ y, float* __restrict__ ssm_state,
                                      const int* __restrict__ cu_seqlens, const int* __restrict__ state_idx,
                                      const int* __restrict__ has_init, int D, int ld_u, int ld_z, int ld_b, int ld_c,
                                      int dt_softplus, int vec) {
  constexpr int NS = N / LPC, TT = kScanTile, CH = kScanCh, NT = CH * LPC;
  struct Stage { __nv_bfloat16 u[TT][CH], dl[TT][CH], z[TT][CH], B[TT][N], C[TT][N]; };
  __shared__ __align__(16) Stage stages[2];
  __shared__ __align__(16) float sB[TT][N], sC[TT][N];
  __shared__ float2 sdt[TT][CH];                     // step size, step size * input
  __shared__ __align__(16) __nv_bfloat16 sy[TT][CH];
  const int s = blockIdx.y, tid = threadIdx.x, lane = tid & 31, q = lane % LPC, c = tid / LPC;
  const int d0 = blockIdx.x * CH, d = d0 + c;
  const int t0 = cu_seqlens[s], n = cu_seqlens[s + 1] - t0;
  const int slot = state_idx && ssm_state ? state_idx[s] : -1;
  const bool live = d < D, resume = live && slot >= 0 && has_init && has_init[s];
  float h[NS], a2[NS];
  float* st = ssm_state + (static_cast<size_t>(slot >= 0 ? slot : 0) * D + (live ? d : 0)) * N + q * NS;
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    a2[i] = live ? finite_rate(A[static_cast<size_t>(d) * N + q * NS + i] * kLog2e) : 0.f;
    h[i] = resume ? st[i] : 0.f;
  }
  const float dsk = (live && Dskip) ? Dskip[d] : 0.f;
  auto eights = [&](int c0) { return (min(TT, n - c0) + 7) & ~7; };      // tokens of a tile that the walk goes over
  auto fetch = [&](int c0, Stage& g) {
    const int mm = eights(c0);
    if (vec) {
      const int j = (tid >> 2) & 31, k = (tid & 3) * 8;      // 128 threads a row set; with 256 the other half fetches delta
      const bool ok = c0 + j < n && d0 + k < D;
      const size_t row = static_cast<size_t>(t0 + (c0 + j < n ? c0 + j : 0)), col = d0 + k < D ? d0 + k : 0;
      if (j < mm && tid < 128) {
        cp_async16(&g.u[j][k], u + row * ld_u + col, ok);
        if (z) cp_async16(&g.z[j][k], z + row * ld_z + col, ok);
      }
      if (j < mm && (NT == 128 || tid >= 128)) cp_async16(&g.dl[j][k], delta + row * ld_u + col, ok);
      for (int i = NT - 1 - tid; i < mm * (N / 8); i += NT) {
        const int jj = i / (N / 8), kk = (i % (N / 8)) * 8;
        const bool in = c0 + jj < n;
        const size_t r = static_cast<size_t>(t0 + (in ? c0 + jj : 0));
        cp_async16(&g.B[jj][kk], B + r * ld_b + kk, in);
        cp_async16(&g.C[jj][kk], C + r * ld_c + kk, in);
      }
    } else {
      const __nv_bfloat16 zero = __float2bfloat16(0.f);
      for (int i = tid; i < mm * CH; i += NT) {
        const int j = i / CH, k = i % CH;
        const bool ok = c0 + j < n && d0 + k < D;
        const size_t row = static_cast<size_t>(t0 + c0 + j);
        g.u[j][k] = ok ? u[row * ld_u + d0 + k] : zero;
        g.dl[j][k] = ok ? delta[row * ld_u + d0 + k] : zero;
        if (z) g.z[j][k] = ok ? z[row * ld_z + d0 + k] : zero;
      }
      for (int i = tid; i < mm * N; i += NT) {
        const int j = i / N, k = i % N;
        const bool ok = c0 + j < n;
        const size_t row = static_cast<size_t>(t0 + c0 + j);
        g.B[j][k] = ok ? B[row * ld_b + k] : zero;
        g.C[j][k] = ok ? C[row * ld_c + k] : zero;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int pc = tid & 31;                           // the channel whose step sizes this thread makes
  const float pb = (d0 + pc < D && dt_bias) ? dt_bias[d0 + pc] : 0.f;
  if (n > 0) fetch(0, stages[0]);
  for (int c0 = 0, it = 0; c0 < n; c0 += TT, ++it) {
    Stage& g = stages[it & 1];
    const int m = min(TT, n - c0), mm = eights(c0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                 // this tile is in; everyone is done with the one before
    if (c0 + TT < n) fetch(c0 + TT, stages[(it + 1) & 1]);
    auto step = [&](int j) {
      float dt = __bfloat162float(g.dl[j][pc]) + pb;
      if (dt_softplus) dt = softplus(dt);
      if (j >= m) dt = 0.f;                          // tokens beyond the sequence leave the state alone
      sdt[j][pc] = make_float2(dt, dt * __bfloat162float(g.u[j][pc]));
    };
    auto widen = [&](int i) {
      (&sB[0][0])[i] = __bfloat162float((&g.B[0][0])[i]);
      (&sC[0][0])[i] = __bfloat162float((&g.C[0][0])[i]);
    };
    if (m == TT) {
#pragma unroll
      for (int j = 0; j < TT; j += NT / 32) step(j + (tid >> 5));
#pragma unroll
      for (int i = 0; i < TT * N; i += NT) widen(i + tid);
    } else {
      for (int j = tid >> 5; j < mm; j += NT / 32) step(j);
      for (int i = tid; i < mm * N; i += NT) widen(i);
    }
    __syncthreads();
    for (int j0 = 0; j0 < m; j0 += 8) {
      float part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float2 e = sdt[j0 + r][c];
        float acc = 0.f, vb[NS], vc[NS];
        load_states<NS>(vb, &sB[j0 + r][q * NS]);
        load_states<NS>(vc, &sC[j0 + r][q * NS]);
#pragma unroll
        for (int i = 0; i < NS; ++i) {
          h[i] = fmaf(ex2(e.x * a2[i]), h[i], e.y * vb[i]);
          acc = fmaf(vc[i], h[i], acc);
        }
        part[r] = acc;
      }
      // lane q of the channel ends up with tokens j0 + q, j0 + q + LPC, ..
#pragma unroll
      for (int o = LPC / 2; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 8 / LPC * o; ++r) {
          const int lo = (r / o) * LPC + r % o;
          const float send = (q & o) ? part[lo] : part[lo + o], keep = (q & o) ? part[lo + o] : part[lo];
          part[lo] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
#pragma unroll
      for (int r = 0; r < 8 / LPC; ++r) {
        float v = part[r * LPC];
        const int j = j0 + r * LPC + q;
        v = fmaf(dsk, __bfloat162float(g.u[j][c]), v);
        if (z) v *= silu(__bfloat162float(g.z[j][c]));
        sy[j][c] = __float2bfloat16(v);
      }
    }
    __syncthreads();
    if (vec) {
      const int j = tid >> 2, k = (tid & 3) * 8;
      if (tid < 128 && j < m && d0 + k < D)
        *reinterpret_cast<uint4*>(y + static_cast<size_t>(t0 + c0 + j) * ld_u + d0 + k) = *reinterpret_cast<const uint4*>(&sy[j][k]);
    } else {
      for (int i = tid; i < m * CH; i += NT)
        if (d0 + i % CH < D) y[static_cast<size_t>(t0 + c0 + i / CH) * ld_u + d0 + i % CH] = sy[i / CH][i % CH];
    }
  }
  if (live && slot >= 0) {
#pragma unroll
    for (int i = 0; i < NS; ++i) st[i] = h[i];
  }
}

// Mamba-2 SSD recurrence. Heads H of width P, state size N, G groups of B/C (H % G == 0):
//   dt = softplus(dt_in[t, h] + dt_bias[h]);  S[p, n] = exp(dt * A[h]) * S[p, n] + dt * x[t, h, p] * B[t, g, n]
//   y[t, h, p] = sum_n S[p, n] * C[t, g, n] + D[h] * x[t, h, p]
// One CTA per (sequence, head): thread (p, j) owns the state columns n = j, j + J, ... of row p
// (J = blockDim.x / P); the row's output is reduced across its J threads with shuffles (J <= 32, power of 2).
template <int NPT>
__global__ void ssd_scan_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dt_in,
                                const float* __restrict__ A, const __nv_bfloat16* __restrict__ B,
                                const __nv_bfloat16* __restrict__ C, const float* __restrict__ Dskip,
                                const float* __restrict__ dt_bias, __nv_bfloat16* __restrict__ y,
                                float* __restrict__ ssm_state, const int* __restrict__ cu_seqlens,
                                const int* __restrict__ state_idx, const int* __restrict__ has_init,
                                int H, int P, int N, int G, int J, int ldx, int ld_dt, int ldb, int ldc, int dt_softplus) {
  extern __shared__ float sbc[];   // B_t[N] | C_t[N]
  const int s = blockIdx.y, hd = blockIdx.x;
  const int g = hd / (H / G);
  const int p = threadIdx.x / J, j = threadIdx.x % J;
  const int t0 = cu_seqlens[s], t1 = cu_seqlens[s + 1];
  const int slot = state_idx ? state_idx[s] : -1;
  float S[NPT];
  float* st = slot >= 0 ? ssm_state + ((static_cast<size_t>(slot) * H + hd) * P + p) * N : nullptr;
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const int n = j + i * J;
    S[i] = (st && has_init && has_init[s] && n < N) ? st[n] : 0.f;
  }
  const float a = A[hd];
  const float dsk = Dskip ? Dskip[hd] : 0.f;
  const float dtb = dt_bias ? dt_bias[hd] : 0.f;
  for (int t = t0; t < t1; ++t) {
    __syncthreads();
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
      sbc[n] = __bfloat162float(B[static_cast<size_t>(t) * ldb + g * N + n]);
      sbc[N + n] = __bfloat162float(C[static_cast<size_t>(t) * ldc + g * N + n]);
    }
    __syncthreads();
    float dt = __bfloat162float(dt_in[static_cast<size_t>(t) * ld_dt + hd]) + dtb;
    if (dt_softplus) dt = softplus(dt);
    const float decay = __expf(dt * a);
    const float xt = __bfloat162float(x[static_cast<size_t>(t) * ldx + hd * P + p]);
    const float dx = dt * xt;
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int n = j + i * J;
      if (n < N) {
        S[i] = decay * S[i] + dx * sbc[n];
        acc = fmaf(S[i], sbc[N + n], acc);
      }
    }
    for (int o = J >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (j == 0) y[(static_cast<size_t>(t) * H + hd) * P + p] = __float2bfloat16(acc + dsk * xt);
  }
  if (st) {
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int n = j + i * J;
      if (n < N) st[n] = S[i];
    }
  }
}

// The SSD recurrence 64 tokens at a time (the chunked form of Dao and Gu, "Transformers are SSMs", 2024). With l_i = log2 of the decay of token i of a chunk, c_i = l_0 + .. + l_i and
// the state S before the chunk:
//   y_i = 2^c_i S C_i + sum_{j <= i} 2^(c_i - c_j) dt_j (C_i . B_j) x_j + D x_i
//   S'  = 2^c_m S + sum_j 2^(l_(j+1) + .. + l_m) dt_j x_j B_j^T
// All powers are at most 1. x, B and C are 16-bit activations and enter the products as they are; what is made from them
// is fp32 and enters as a sum of bf16 numbers: two for S and the weighted products C . B (they end in a 16-bit y), three
// for the weighted inputs of the state, so that the fp32 state keeps 24 bits. The powers of the state's sum run from the
// chunk's end backwards, where the large ones are the short sums.
// S^T stays in the accumulator fragments of the warp that owns its 16 rows p, which are also the B fragments of S C.
// The chain from chunk to chunk is the bound (one CTA per sequence, head and 64 rows walks the chunks in order, about
// 7 us each), so it is kept short: two barriers a chunk, tiles and step sizes fetched one chunk ahead.
// Two sequences, 4096 tokens, 80 heads x 64 x 128: 12742 us token by token (two barriers and a load from global memory on
// every token's chain), 239 us so (in a row 224, and 231 with `rest` and the check of the products below). Up to 16 tokens a
// chunk does the work of 16: 64 sequences of 4 tokens 563 us walked, 168 as whole chunks, 111 so. Three CTAs per SM up to 32 states.
constexpr int kChunk = 64, kNV = 64, kChunkThreads = 128, kLdV = kNV + 8, kLdP = kChunk + 8;

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the bf16 pair nearest to (x, y); x and y become what is left
__device__ __forceinline__ uint32_t take_bf16(float& x, float& y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const float2 f = __bfloat1622float2(h);
  x -= f.x;
  y -= f.y;
  return *reinterpret_cast<const uint32_t*>(&h);
}

// the signs' places of two bf16 values set where one is infinite or NaN (an exponent of ones carries into them)
__device__ __forceinline__ uint32_t mark_special(uint32_t w) { return (w & 0x7f807f80u) + 0x00800080u; }

// a + b, and in `left` what its rounding left (Knuth's exact sum of two floats)
__device__ __forceinline__ float two_sum(float a, float b, float& left) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  left = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return s;
}

struct SsdChunk {
  const __nv_bfloat16 *x, *dt, *B, *C;
  const float *A, *Dskip, *dt_bias;
  __nv_bfloat16* y;
  float* state;
  const int *cu_seqlens, *state_idx, *has_init;
  int H, P, N, G, ldx, ld_dt, ldb, ldc, dt_softplus, col_blocks;
  // Long prompts in segments of `seg` tokens (0: whole sequences), each with its own CTA. parts [segments, H, P, N] holds the state that a
  // segment makes of nothing, decays [segments, H] its decay. Nobody needs that of a sequence's last segment: its entry holds a copy of the
  // kept state instead, because the CTA that walks the last segment replaces the kept one while others of its launch may not have begun.
  int seg, n_seqs;
  float *parts, *decays;
};
// Segments of a step: sequence s has numbers (cu_seqlens[s] / seg) + s + i, which never meet another sequence's.
__device__ __forceinline__ int segment_base(const SsdChunk& p, int s) { return p.cu_seqlens[s] / p.seg + s; }
// per chunk: c_i (and what its rounding left), 2^(sum beyond j) dt_j, dt_j, 2^c_i. With c_i alone a difference c_i - c_j would
// carry the rounding of sums that may be thousands of times larger than it: after a token that decays by 2^-50000 the next ones'
// weights were off by 2 in 1000.
struct alignas(8) SsdTimes { float cum[kChunk], rest[kChunk], tail[kChunk], dt[kChunk], grow[kChunk], total; };

// 16 queries (rows 16 W ..) with the keys at or before them, weighted, into sP as hi and lo parts
template <int W, int DK>
__device__ __forceinline__ void ssd_products(const __nv_bfloat16* sC, const __nv_bfloat16* sB, __nv_bfloat16* sP, const SsdTimes& tm, int lane) {
  constexpr int LDK = DK + 8;
  const int mi = lane >> 3, r8 = lane & 7, row4 = lane >> 2, col2 = 2 * (lane & 3);
  float sc[2 * (W + 1)][4];
#pragma unroll
  for (int i = 0; i < 2 * (W + 1); ++i) sc[i][0] = sc[i][1] = sc[i][2] = sc[i][3] = 0.f;
#pragma unroll
  for (int kb = 0; kb < DK / 16; ++kb) {
    uint32_t a[4];
    ldsm4(a, sC + (W * 16 + (lane & 15)) * LDK + kb * 16 + (lane >> 4) * 8);
#pragma unroll
    for (int np = 0; np <= W; ++np) {
      uint32_t b[4];
      ldsm4(b, sB + (np * 16 + (mi >> 1) * 8 + r8) * LDK + kb * 16 + (mi & 1) * 8);
      mma(sc[2 * np], a, b[0], b[1]);
      mma(sc[2 * np + 1], a, b[2], b[3]);
    }
  }
  const float ci[2] = {tm.cum[W * 16 + row4], tm.cum[W * 16 + row4 + 8]}, ri[2] = {tm.rest[W * 16 + row4], tm.rest[W * 16 + row4 + 8]};
#pragma unroll
  for (int nt = 0; nt < 2 * (W + 1); ++nt) {
    const int j = nt * 8 + col2;
    const float2 c = *reinterpret_cast<const float2*>(&tm.cum[j]), r = *reinterpret_cast<const float2*>(&tm.rest[j]),
                 d = *reinterpret_cast<const float2*>(&tm.dt[j]);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = W * 16 + row4 + 8 * e;
      float a0 = sc[nt][2 * e] * (ex2((ci[e] - c.x) + (ri[e] - r.x)) * d.x), a1 = sc[nt][2 * e + 1] * (ex2((ci[e] - c.y) + (ri[e] - r.y)) * d.y);
      if (nt >= 2 * W) {                             // the block on the diagonal
        if (i < j) a0 = 0.f;
        if (i <= j) a1 = 0.f;
      }
      *reinterpret_cast<uint32_t*>(sP + i * kLdP + j) = take_bf16(a0, a1);
      *reinterpret_cast<uint32_t*>(sP + (kChunk + i) * kLdP + j) = take_bf16(a0, a1);
    }
  }
}

// LOCAL: only the state that a segment makes of nothing, for all segments but a sequence's last one, and the copy of the kept state.
template <int DK, bool LOCAL>
__global__ void __launch_bounds__(kChunkThreads, DK == 32 ? 3 : 2) ssd_chunk_kernel(const SsdChunk p) {
  typedef __nv_bfloat16 bf16;
  constexpr int LDK = DK + 8, KB = DK / 16, kStage = kChunk * (2 * LDK + kLdV);
  extern __shared__ __align__(16) uint8_t smem_raw[];
  bf16* stages = reinterpret_cast<bf16*>(smem_raw);
  bf16* sP = stages + 2 * kStage;                    // [hi | lo][chunk][kLdP]
  __shared__ SsdTimes times[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mi = lane >> 3, r8 = lane & 7, row4 = lane >> 2, col2 = 2 * (lane & 3);
  const int h = blockIdx.x / p.col_blocks, v0 = (blockIdx.x % p.col_blocks) * kNV, P = p.P, N = p.N;
  int s = blockIdx.y, part = 0;
  if (p.seg > 0) {
    int lo = 0, hi = p.n_seqs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (segment_base(p, mid) <= static_cast<int>(blockIdx.y)) lo = mid; else hi = mid - 1;
    }
    s = lo;
    part = blockIdx.y - segment_base(p, s);
  }
  const int slot = p.state_idx && p.state ? p.state_idx[s] : -1;
  const bool resume = slot >= 0 && p.has_init && p.has_init[s];
  float* st = p.state + (static_cast<size_t>(slot >= 0 ? slot : 0) * p.H + h) * P * N;
  const float* kept = st;
  int t0 = p.cu_seqlens[s], n = p.cu_seqlens[s + 1] - t0;
  bool last = true;
  if (p.seg > 0) {
    const int from = part * p.seg;
    if (part < 0 || (part > 0 && from >= n)) return;     // before the first sequence, or behind the end of this one
    last = from + p.seg >= n;
    if (part > 0 || !last) {
      float* copy = p.parts + (static_cast<size_t>(blockIdx.y - part + (n - 1) / p.seg) * p.H + h) * P * N;
      kept = copy;
      if (LOCAL && last && resume)
        for (int i = v0 * N + 2 * tid; i < min(v0 + kNV, P) * N; i += 2 * kChunkThreads)
          *reinterpret_cast<float2*>(copy + i) = *reinterpret_cast<const float2*>(st + i);
    }
    if (LOCAL && last) return;
    t0 += from;
    n = min(n - from, p.seg);
  }
  const int group = h / (p.H / p.G);
  const bf16 *xh = p.x + static_cast<size_t>(t0) * p.ldx + h * P, *Bh = p.B + static_cast<size_t>(t0) * p.ldb + group * N,
             *Ch = p.C + static_cast<size_t>(t0) * p.ldc + group * N, *dth = p.dt + static_cast<size_t>(t0) * p.ld_dt + h;
  auto fetch = [&](int c0, bf16* dst) {              // rows beyond the sequence and columns beyond the head become zero
    constexpr int CH = DK / 8;
    for (int i = tid; i < kChunk * CH; i += kChunkThreads) {
      const int j = i / CH, c = (i % CH) * 8;
      const bool ok = c0 + j < n && c < N;
      const size_t row = ok ? c0 + j : 0;
      cp_async16(dst + j * LDK + c, Ch + row * p.ldc + (ok ? c : 0), ok);
      cp_async16(dst + (kChunk + j) * LDK + c, Bh + row * p.ldb + (ok ? c : 0), ok);
    }
    bf16* dv = dst + 2 * kChunk * LDK;
    for (int i = tid; i < kChunk * (kNV / 8); i += kChunkThreads) {
      const int j = i / (kNV / 8), c = (i % (kNV / 8)) * 8;
      const bool ok = c0 + j < n && v0 + c < P;
      cp_async16(dv + j * kLdV + c, xh + (ok ? static_cast<size_t>(c0 + j) * p.ldx + v0 + c : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // warp 0 makes the step sizes and their sums, two tokens per lane; the raw values are read one chunk earlier
  const float a2 = finite_rate(p.A[h] * kLog2e), dtb = p.dt_bias ? p.dt_bias[h] : 0.f;
  float raw[2];
  auto read_dt = [&](int c0) {
#pragma unroll
    for (int e = 0; e < 2; ++e) raw[e] = c0 + 2 * lane + e < n ? __bfloat162float(dth[static_cast<size_t>(c0 + 2 * lane + e) * p.ld_dt]) : 0.f;
  };
  auto make_times = [&](int c0, SsdTimes& tm) {
    float dt[2], l[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      dt[e] = raw[e] + dtb;
      if (p.dt_softplus) dt[e] = softplus(dt[e]);
      if (c0 + 2 * lane + e >= n) dt[e] = 0.f;
      l[e] = dt[e] * a2;
      if (l[e] < -1e6f) l[e] = -1e6f;                // zero either way, and the sums stay finite
    }
    // sums up to this pair as a float and what its rounding left, and from it (the large powers are the short sums)
    float rest, hi = two_sum(l[0], l[1], rest), down = hi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_up_sync(0xffffffffu, hi, o), v = __shfl_up_sync(0xffffffffu, rest, o), w = __shfl_down_sync(0xffffffffu, down, o);
      if (lane >= o) {
        float left;
        hi = two_sum(hi, u, left);
        rest += v + left;
      }
      if (lane + o < 32) down += w;
    }
    float before = __shfl_up_sync(0xffffffffu, hi, 1), before_rest = __shfl_up_sync(0xffffffffu, rest, 1);
    float after = __shfl_down_sync(0xffffffffu, down, 1), left;
    if (lane == 0) before = before_rest = 0.f;
    if (lane == 31) after = 0.f;
    const float c0_ = two_sum(before, l[0], left), c1_ = hi;
    tm.cum[2 * lane] = c0_; tm.cum[2 * lane + 1] = c1_;
    tm.rest[2 * lane] = before_rest + left; tm.rest[2 * lane + 1] = rest;
    tm.grow[2 * lane] = ex2(c0_); tm.grow[2 * lane + 1] = ex2(c1_);
    tm.tail[2 * lane] = ex2(after + l[1]) * dt[0]; tm.tail[2 * lane + 1] = ex2(after) * dt[1];
    tm.dt[2 * lane] = dt[0]; tm.dt[2 * lane + 1] = dt[1];
    if (lane == 31) tm.total = ex2(c1_);
  };
  if (n > 0) {
    fetch(0, stages);
    if (warp == 0) {
      read_dt(0);
      make_times(0, times[0]);
      read_dt(kChunk);
    }
  }
  const float dsk = p.Dskip ? p.Dskip[h] : 0.f;
  // S^T: 16 rows p of this warp as accumulator tiles of 8 columns n: [0], [1] row row4, [2], [3] row row4 + 8
  float S[2 * KB][4];
  const int vr = v0 + warp * 16 + row4;
#pragma unroll
  for (int t = 0; t < 2 * KB; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float2 f = make_float2(0.f, 0.f);
      if (!LOCAL && resume && vr + 8 * e < P && 8 * t < N) f = *reinterpret_cast<const float2*>(kept + static_cast<size_t>(vr + 8 * e) * N + 8 * t + col2);
      S[t][2 * e] = f.x; S[t][2 * e + 1] = f.y;
    }
  bool have_state = !LOCAL && resume;
  float decay = 1.f;
  if (!LOCAL && part > 0) {                          // through the segments before
    for (int i = 0; i < part; ++i) {
      const size_t at = static_cast<size_t>(blockIdx.y - part + i) * p.H + h;
      const float f = p.decays[at];
      const float* from = p.parts + at * P * N;
#pragma unroll
      for (int t = 0; t < 2 * KB; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (vr + 8 * e >= P || 8 * t >= N) continue;
          const float2 x = *reinterpret_cast<const float2*>(from + static_cast<size_t>(vr + 8 * e) * N + 8 * t + col2);
          S[t][2 * e] = have_state ? fmaf(S[t][2 * e], f, x.x) : x.x;
          S[t][2 * e + 1] = have_state ? fmaf(S[t][2 * e + 1], f, x.y) : x.y;
        }
      have_state = true;
    }
  }
  for (int c0 = 0, it = 0; c0 < n; c0 += kChunk, ++it) {
    const int m = min(kChunk, n - c0);
    const bf16 *sC = stages + (it & 1) * kStage, *sB = sC + kChunk * LDK, *sV = sB + kChunk * LDK;
    const SsdTimes& tm = times[it & 1];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                 // this chunk is in; everyone is done with the last one's stage, times and sP
    if (c0 + kChunk < n) fetch(c0 + kChunk, stages + ((it + 1) & 1) * kStage);
    // NB: blocks of 16 tokens that have any
    auto chunk = [&](auto blocks) {
      constexpr int NB = decltype(blocks)::value;
      if constexpr (LOCAL) {
        if (warp == 0 && c0 + kChunk < n) {
          make_times(c0 + kChunk, times[(it + 1) & 1]);
          read_dt(c0 + 2 * kChunk);
        }
        decay *= tm.total;
      } else {
      switch (warp) {
        case 0:                                        // the fewest products: this warp also prepares the next chunk's times
          ssd_products<0, DK>(sC, sB, sP, tm, lane);
          if (c0 + kChunk < n) {
            make_times(c0 + kChunk, times[(it + 1) & 1]);
            read_dt(c0 + 2 * kChunk);
          }
          break;
        case 1: if constexpr (NB > 1) ssd_products<1, DK>(sC, sB, sP, tm, lane); break;
        case 2: if constexpr (NB > 2) ssd_products<2, DK>(sC, sB, sP, tm, lane); break;
        default: if constexpr (NB > 3) ssd_products<3, DK>(sC, sB, sP, tm, lane); break;
      }
      // what the state before the chunk contributes, for all tokens and this warp's 16 rows
      float o[NB][2][4];
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) o[i][j][0] = o[i][j][1] = o[i][j][2] = o[i][j][3] = 0.f;
      if (have_state) {
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
          uint32_t hi[2][2], lo[2][2];
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float u = S[2 * kb + e][2 * j], w = S[2 * kb + e][2 * j + 1];
              hi[j][e] = take_bf16(u, w);
              lo[j][e] = take_bf16(u, w);
            }
          uint32_t a[NB][4];
#pragma unroll
          for (int i = 0; i < NB; ++i) ldsm4(a[i], sC + (i * 16 + (lane & 15)) * LDK + kb * 16 + (lane >> 4) * 8);
#pragma unroll
          for (int i = 0; i < NB; ++i) { mma(o[i][0], a[i], hi[0][0], hi[0][1]); mma(o[i][1], a[i], hi[1][0], hi[1][1]); }
#pragma unroll
          for (int i = 0; i < NB; ++i) { mma(o[i][0], a[i], lo[0][0], lo[0][1]); mma(o[i][1], a[i], lo[1][0], lo[1][1]); }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          const float f0 = tm.grow[i * 16 + row4], f1 = tm.grow[i * 16 + row4 + 8];
#pragma unroll
          for (int j = 0; j < 2; ++j) { o[i][j][0] *= f0; o[i][j][1] *= f0; o[i][j][2] *= f1; o[i][j][3] *= f1; }
        }
      }
      __syncthreads();                               // the products of every warp are in sP
      // The products with later tokens are zeros, and zero times an infinite or NaN input is NaN: a warp that finds such an input
      // takes its products one token at a time, over the tokens at or before each row.
      uint32_t bv[NB][4], marks = 0;
#pragma unroll
      for (int kb = 0; kb < NB; ++kb) {
        ldsm4_t(bv[kb], sV + (kb * 16 + (mi & 1) * 8 + r8) * kLdV + warp * 16 + (mi >> 1) * 8);
#pragma unroll
        for (int q = 0; q < 4; ++q) marks |= mark_special(bv[kb][q]);
      }
      if (!__any_sync(0xffffffffu, marks & 0x80008000u)) {
#pragma unroll
        for (int kb = 0; kb < NB; ++kb)
#pragma unroll
          for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int i = kb; i < NB; ++i) {
              uint32_t a[4];
              ldsm4(a, sP + (half * kChunk + i * 16 + (lane & 15)) * kLdP + kb * 16 + (lane >> 4) * 8);
              mma(o[i][0], a, bv[kb][0], bv[kb][1]);
              mma(o[i][1], a, bv[kb][2], bv[kb][3]);
            }
      } else {
        for (int t = 0; t < m; ++t) {
          float v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = __bfloat162float(sV[t * kLdV + warp * 16 + (j >> 1) * 8 + col2 + (j & 1)]);
#pragma unroll
          for (int i = 0; i < 2 * NB; ++i) {           // rows i / 2, its lower or upper half
            const int r = (i >> 1) * 16 + row4 + 8 * (i & 1);
            if (r < t) continue;
            const float w = __bfloat162float(sP[r * kLdP + t]) + __bfloat162float(sP[(kChunk + r) * kLdP + t]);
#pragma unroll
            for (int j = 0; j < 4; ++j) o[i >> 1][j >> 1][2 * (i & 1) + (j & 1)] = fmaf(w, v[j], o[i >> 1][j >> 1][2 * (i & 1) + (j & 1)]);
          }
        }
      }
      bf16* out = p.y + (static_cast<size_t>(t0 + c0) * p.H + h) * P;
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = i * 16 + row4 + 8 * e;
          if (r >= m) continue;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int cl = warp * 16 + j * 8 + col2, c = v0 + cl;
            if (c >= P) continue;
            const float2 xv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sV + r * kLdV + cl));
            *reinterpret_cast<__nv_bfloat162*>(out + static_cast<size_t>(r) * p.H * P + c) =
                __floats2bfloat162_rn(fmaf(dsk, xv.x, o[i][j][2 * e]), fmaf(dsk, xv.y, o[i][j][2 * e + 1]));
          }
        }
      }
      // the state after the chunk
      if (have_state) {
        const float f = tm.total;
#pragma unroll
        for (int t = 0; t < 2 * KB; ++t) { S[t][0] *= f; S[t][1] *= f; S[t][2] *= f; S[t][3] *= f; }
      }
      have_state = true;
#pragma unroll
      for (int kb = 0; kb < NB; ++kb) {
        uint32_t a[4], w3[3][4];                       // rows p: transposed fragments of x, weighted, in three parts
        ldsm4_t(a, sV + (kb * 16 + (mi >> 1) * 8 + r8) * kLdV + warp * 16 + (mi & 1) * 8);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = kb * 16 + (q >> 1) * 8 + col2;
          const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a[q]));
          float u = f.x * tm.tail[j], w = f.y * tm.tail[j + 1];
#pragma unroll
          for (int part = 0; part < 3; ++part) w3[part][q] = take_bf16(u, w);
        }
#pragma unroll
        for (int t = 0; t < KB; t += 2) {
          uint32_t b[4], c[4];
          ldsm4_t(b, sB + (kb * 16 + (mi & 1) * 8 + r8) * LDK + t * 16 + (mi >> 1) * 8);
          ldsm4_t(c, sB + (kb * 16 + (mi & 1) * 8 + r8) * LDK + t * 16 + 16 + (mi >> 1) * 8);
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            mma(S[2 * t], w3[part], b[0], b[1]);
            mma(S[2 * t + 1], w3[part], b[2], b[3]);
            mma(S[2 * t + 2], w3[part], c[0], c[1]);
            mma(S[2 * t + 3], w3[part], c[2], c[3]);
          }
        }
      }
    };
    if (m > 16) chunk(std::integral_constant<int, 4>());
    else chunk(std::integral_constant<int, 1>());      // a short prompt, or a prompt's end
  }
  if (LOCAL) {
    const size_t at = static_cast<size_t>(blockIdx.y) * p.H + h;
    st = p.parts + at * P * N;
    if (tid == 0 && v0 == 0) p.decays[at] = decay;
  }
  if (LOCAL || (slot >= 0 && last)) {
#pragma unroll
    for (int t = 0; t < 2 * KB; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (vr + 8 * e < P && 8 * t < N)
          *reinterpret_cast<float2*>(st + static_cast<size_t>(vr + 8 * e) * N + 8 * t + col2) = make_float2(S[t][2 * e], S[t][2 * e + 1]);
  }
}

template <int DK>
static int launch_ssd_chunk(const SsdChunk& p, int n_seqs, int tokens, cudaStream_t stream) {
  constexpr int smem = (2 * kChunk * (2 * (DK + 8) + kLdV) + 2 * kChunk * kLdP) * 2;
  static PerDeviceOnce configured;
  if (configured.needed()) {
    if (cudaFuncSetAttribute(ssd_chunk_kernel<DK, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaFuncSetAttribute(ssd_chunk_kernel<DK, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return MB_ERR_LAUNCH;
    configured.done();
  }
  const dim3 grid(p.H * p.col_blocks, p.seg > 0 ? tokens / p.seg + n_seqs : n_seqs);
  if (p.seg > 0) ssd_chunk_kernel<DK, true><<<grid, kChunkThreads, smem, stream>>>(p);
  ssd_chunk_kernel<DK, false><<<grid, kChunkThreads, smem, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// out = rmsnorm(y * silu(z)) * w, rows of up to 256 x 8 x NV values held in registers by one CTA (one pass over memory,
// bound by it; the same steps as separate operators read and wrote seven fp32 copies of the row).
template <int NV>
__global__ void __launch_bounds__(256) gated_rms_norm_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ z,
                                                             const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                             int D, int ldz, float eps) {
  __shared__ float part[8];
  const size_t t = blockIdx.x;
  const int tid = threadIdx.x;
  float g[NV][8], sum = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * 256 + tid) * 8;
    if (c >= D) break;
    float gate[8];
    load_bf16<8>(g[i], y + t * D + c);
    load_bf16<8>(gate, z + t * ldz + c);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      g[i][e] *= silu(gate[e]);
      sum = fmaf(g[i][e], g[i][e], sum);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((tid & 31) == 0) part[tid >> 5] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) sum += part[i];
  const float r = rsqrtf(sum / D + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * 256 + tid) * 8;
    if (c >= D) break;
    float wv[8];
    load_bf16<8>(wv, w + c);
#pragma unroll
    for (int e = 0; e < 8; ++e) wv[e] *= g[i][e] * r;
    store_bf16<8>(out + t * D + c, wv);
  }
}

}  // namespace ssm
}  // namespace mb

using namespace mb::ssm;

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// `tokens`: rows of x, an upper bound of cu_seqlens[n_seqs]
extern "C" int mb_causal_conv1d_varlen(const void* x, const void* w, const void* bias, void* y, float* conv_state,
                                       const int* cu_seqlens, const int* state_idx, const int* has_init,
                                       int n_seqs, int tokens, int D, int width, int ldx, int ldy, int act,
                                       cudaStream_t stream) {
  if (n_seqs <= 0 || D <= 0) return MB_OK;
  // 8-byte accesses where every row starts on such a boundary (of 16-byte ones a thread's eight channels take 120 registers)
  const bool vec = D % 8 == 0 && ldx % 8 == 0 && ldy % 8 == 0 && aligned16(x) && aligned16(y) && aligned16(w) &&
                   (bias == nullptr || aligned16(bias)) && aligned16(conv_state);
  const int per = 128 * (vec ? 4 : 1);
  dim3 grid(n_seqs + (tokens + kConvTile - 1) / kConvTile, (D + per - 1) / per);
  // Steps whose sequences are no longer than a tile on average go without the code for whole tiles, which others wait for: one token of
  // 64 sequences x 2048 channels 4.1 us (4.4 with it), of 16 3.5 (3.8); 33 tokens of 64 x 4096 25 us with it (31).
  const bool whole = vec && tokens > kConvTile * static_cast<long long>(n_seqs);
#define MB_CONV(Wv, Vv, Whole)                                                                                   \
  causal_conv1d_kernel<Wv, Vv, Whole><<<grid, 128, 0, stream>>>(                                                 \
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w),                                \
      static_cast<const __nv_bfloat16*>(bias), static_cast<__nv_bfloat16*>(y), conv_state, cu_seqlens, state_idx, \
      has_init, n_seqs, D, ldx, ldy, act)
#define MB_CONV2(Wv) do { if (whole) MB_CONV(Wv, 4, true); else if (vec) MB_CONV(Wv, 4, false); else MB_CONV(Wv, 1, false); } while (0)
  switch (width) {
    case 2: MB_CONV2(2); break;
    case 3: MB_CONV2(3); break;
    case 4: MB_CONV2(4); break;
    case 8: MB_CONV2(8); break;
    default: return MB_ERR_SHAPE;
  }
#undef MB_CONV2
#undef MB_CONV
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_selective_scan_varlen(const void* u, const void* delta, const float* A, const void* B,
                                        const void* C, const float* Dskip, const void* z, const float* dt_bias,
                                        void* y, float* ssm_state, const int* cu_seqlens, const int* state_idx,
                                        const int* has_init, int n_seqs, int tokens, int D, int N, int ld_u, int ld_z,
                                        int ld_b, int ld_c, int dt_softplus, cudaStream_t stream) {
  if (n_seqs <= 0 || D <= 0) return MB_OK;
  const int vec = D % 8 == 0 && ld_u % 8 == 0 && ld_b % 8 == 0 && ld_c % 8 == 0 && aligned16(u) && aligned16(delta) &&
                  aligned16(B) && aligned16(C) && aligned16(y) && (z == nullptr || (ld_z % 8 == 0 && aligned16(z)));
  dim3 grid((D + kScanCh - 1) / kScanCh, n_seqs);
  // Four lanes a channel take 40 % fewer instructions per token than eight (wider reads of B and C, one exchange less) but give
  // half the warps; from 2048 warps on they win: 4096 channels, 4099 tokens in 3, 4 and 8 sequences 239, 187 and 145 us against 218,
  // 203 and 184; 2000 tokens in 32 72 against 86, one token of 256 each 95 against 125, 200 in two 14.1 against 13.3.
  // With 32 states a lane then has eight, whose chain is longer than the work it saves until sequences have some 32 tokens: one token of 64
  // each 50.6 against 46.8, 16 of each level, 60 of 16 each 61 against 68 (eight lanes second).
  const bool many = static_cast<long long>(D) * n_seqs >= 16384 && (N < 32 || tokens >= 32LL * n_seqs);
#define MB_SCAN(Nv)                                                                                             \
  if (many) MB_SCAN_L(Nv, 4); else MB_SCAN_L(Nv, 8)
#define MB_SCAN_L(Nv, Lv)                                                                                                \
  selective_scan_kernel<Nv, Lv><<<grid, kScanCh * Lv, 0, stream>>>(                                                      \
      static_cast<const __nv_bfloat16*>(u), static_cast<const __nv_bfloat16*>(delta), A,                        \
      static_cast<const __nv_bfloat16*>(B), static_cast<const __nv_bfloat16*>(C), Dskip,                        \
      static_cast<const __nv_bfloat16*>(z), dt_bias, static_cast<__nv_bfloat16*>(y), ssm_state, cu_seqlens,     \
      state_idx, has_init, D, ld_u, ld_z, ld_b, ld_c, dt_softplus, vec)
  switch (N) {
    case 8: MB_SCAN(8); break;
    case 16: MB_SCAN(16); break;
    case 32: MB_SCAN(32); break;
    default: return MB_ERR_SHAPE;
  }
#undef MB_SCAN_L
#undef MB_SCAN
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// Long prompts whose chains do not fill the chip are walked in segments of 512 tokens, or a sixteenth of the step if that is more (the states
// of all segments lie in scratch): one launch makes every segment's state out of
// nothing, another walks all segments at once from the states before them. Half of the products are done twice, so it pays where whole walks leave
// SMs idle and sequences are long: up to two walks for three SMs, with states of up to 32 columns, whose products weigh less, up to five for four. us
// whole and in segments, rows of 64: state 128, one sequence of 4096, 80 walks 369 and 265, 100 379 and 316, 111 381 and 334, 128 393 and 397, 160 472
// and 474 (10000 tokens 1133 and 1232); 1536 tokens, 100 walks 147 and 146, in two sequences 110 145 and 150, four of 2048, 108 walks 180 and 194; state 64, two
// of 2048, 100 walks 154 and 128, 160 177 and 183; state 32, two of 2048, 160 walks 148 and 134, 184 152 and 142, four of 1536, 184 114 and 115.
extern "C" int mb_ssd_segment(int tokens, int n_seqs, int H, int P, int N) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  }
  const long long chains = static_cast<long long>(n_seqs) * H * ((P + kNV - 1) / kNV);
  if (N <= 32 ? chains * 4 > sms * 5LL : chains * 3 > sms * 2LL) return 0;
  if (tokens < 1536LL * n_seqs) return 0;
  const int sixteenth = (tokens / 16 + kChunk - 1) / kChunk * kChunk;
  return sixteenth > 512 ? sixteenth : 512;
}

extern "C" int mb_ssd_scan_varlen(const void* x, const void* dt, const float* A, const void* B, const void* C,
                                  const float* Dskip, const float* dt_bias, void* y, float* ssm_state,
                                  const int* cu_seqlens, const int* state_idx, const int* has_init, int n_seqs,
                                  int tokens, int H, int P, int N, int G, int ldx, int ld_dt, int ldb, int ldc,
                                  int dt_softplus, float* scratch, long long scratch_floats, cudaStream_t stream) {
  if (n_seqs <= 0 || H <= 0) return MB_OK;
  if (P <= 0 || P > 256 || (P & (P - 1)) || G <= 0 || H % G || N <= 0 || N > 256) return MB_ERR_SHAPE;
  // From four tokens per sequence on, the chunks win (64 sequences of 4 tokens: 80 heads x 64 x 128 563 against 111 us, 24 heads x 64 x
  // 16 17 against 16.5), and earlier where one sequence is much longer than the others. They take 16-byte copies of whole 8-value
  // groups, so sizes and addresses that do not fit stay with the walk.
  if (tokens >= 4LL * n_seqs && N <= 128 && N % 8 == 0 && P % 8 == 0 && ldx % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0 &&
      aligned16(x) && aligned16(B) && aligned16(C) && (reinterpret_cast<uintptr_t>(ssm_state) & 7) == 0) {
    SsdChunk p{static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dt), static_cast<const __nv_bfloat16*>(B),
               static_cast<const __nv_bfloat16*>(C), A, Dskip, dt_bias, static_cast<__nv_bfloat16*>(y), ssm_state, cu_seqlens,
               state_idx, has_init, H, P, N, G, ldx, ld_dt, ldb, ldc, dt_softplus, (P + kNV - 1) / kNV, 0, n_seqs, nullptr, nullptr};
    const int seg = mb_ssd_segment(tokens, n_seqs, H, P, N);
    const long long segments = seg > 0 ? static_cast<long long>(tokens) / seg + n_seqs : 0;
    if (seg > 0 && scratch != nullptr && scratch_floats >= segments * H * (static_cast<long long>(P) * N + 1) && segments <= 65535) {
      p.seg = seg;
      p.parts = scratch;
      p.decays = scratch + segments * H * P * N;
    }
    if (N <= 32) return launch_ssd_chunk<32>(p, n_seqs, tokens, stream);
    if (N <= 64) return launch_ssd_chunk<64>(p, n_seqs, tokens, stream);
    return launch_ssd_chunk<128>(p, n_seqs, tokens, stream);
  }
  int J = 256 / P;            // threads per state row
  if (J > 32) J = 32;
  if (J < 1) J = 1;
  const int npt = (N + J - 1) / J;
  dim3 grid(H, n_seqs);
  const int threads = P * J;
  const size_t smem = 2 * static_cast<size_t>(N) * sizeof(float);
#define MB_SSD(NPTv)                                                                                            \
  ssd_scan_kernel<NPTv><<<grid, threads, smem, stream>>>(                                                       \
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dt), A,                           \
      static_cast<const __nv_bfloat16*>(B), static_cast<const __nv_bfloat16*>(C), Dskip, dt_bias,               \
      static_cast<__nv_bfloat16*>(y), ssm_state, cu_seqlens, state_idx, has_init, H, P, N, G, J, ldx, ld_dt,    \
      ldb, ldc, dt_softplus)
  if (npt <= 4) MB_SSD(4);
  else if (npt <= 8) MB_SSD(8);
  else if (npt <= 16) MB_SSD(16);
  else if (npt <= 32) MB_SSD(32);
  else if (npt <= 64) MB_SSD(64);
  else return MB_ERR_SHAPE;
#undef MB_SSD
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_gated_rms_norm(const void* y, const void* z, const void* w, void* out, int T, int D, int ldz, float eps,
                                 cudaStream_t stream) {
  if (T <= 0) return MB_OK;
  if (D <= 0 || D % 8 || D > 16384 || ldz % 8 || !aligned16(y) || !aligned16(z) || !aligned16(w) || !aligned16(out))
    return MB_ERR_SHAPE;
#define MB_NORM(NV)                                                                                                      \
  gated_rms_norm_kernel<NV><<<T, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(z), \
                                                   static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(out), D, ldz, eps)
  if (D <= 2048) MB_NORM(1);
  else if (D <= 4096) MB_NORM(2);
  else if (D <= 6144) MB_NORM(3);
  else if (D <= 8192) MB_NORM(4);
  else MB_NORM(8);
#undef MB_NORM
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}
