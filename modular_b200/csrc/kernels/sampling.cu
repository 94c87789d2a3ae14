// Token sampling on the device: greedy argmax, temperature / top-k / top-p / min-p
// sampling with per-request seeds, and frequency / presence / repetition penalties.
//
// sample_kernel: one CTA of 1024 threads owns one batch row. Top-k and top-p cut-offs are found by
// bisection on the order-preserving integer image of the fp32 logits, so no sort and
// no scratch memory is needed; pure temperature sampling takes the one-pass Gumbel-max
// route. sample_cluster_kernel spreads a row over a thread-block cluster and runs for all but large batches without a filter;
// sample_kernel is for those and for devices that cannot place such clusters. Behavioural counterparts in the reference: max/kernels/src/nn/topk.mojo
// (fused token sampling :2037, Gumbel argmax :2369), nn/sampling/topk_fi.mojo,
// nn/sampling/sampling.mojo:31 (penalties).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "../common/api.h"
#include "../common/launch.h"
#include "../common/ptx.cuh"

namespace mb {

constexpr int kSampThreads = 1024;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform01(uint64_t seed, uint64_t step, uint64_t idx) {
  const uint64_t h = mix64(mix64(seed ^ (step * 0xD1342543DE82EF95ull)) + idx);
  return (static_cast<float>(h >> 40) + 0.5f) * (1.0f / 16777216.0f);  // (0,1)
}
// Monotone map fp32 -> uint32 (larger float <=> larger key).
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax amax2(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ ArgMax block_argmax(ArgMax a, ArgMax* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = amax2(a, b);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[warp] = a;
  __syncthreads();
  ArgMax r = lane < (blockDim.x >> 5) ? sh[lane] : ArgMax{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b;
    b.v = __shfl_xor_sync(0xffffffffu, r.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, r.i, o);
    r = amax2(r, b);
  }
  __syncthreads();
  return r;
}
__device__ __forceinline__ float block_sum_f(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float r = lane < (blockDim.x >> 5) ? sh[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  __syncthreads();
  return r;
}

// Visit every element of a row as f(value, index). Rows that start on a 16-byte boundary are read as float4 with
// four loads in flight per thread: with one scalar load per iteration a pass over 128 k logits is bound by
// the latency of its 125 dependent round trips (about 60 us per pass on B200), not by bandwidth.
template <typename F>
__device__ __forceinline__ void for_each_logit(const float* __restrict__ row, int vocab, F&& f) {
  if ((reinterpret_cast<uintptr_t>(row) & 15) != 0) {
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) f(row[i], i);
    return;
  }
  const int n4 = vocab >> 2;
  const float4* __restrict__ r4 = reinterpret_cast<const float4*>(row);
  const int step = blockDim.x;
  int i = threadIdx.x;
  for (; i + 3 * step < n4; i += 4 * step) {
    const float4 a = r4[i];
    const float4 b = r4[i + step];
    const float4 c = r4[i + 2 * step];
    const float4 d = r4[i + 3 * step];
    const int ia = i << 2, ib = (i + step) << 2, ic = (i + 2 * step) << 2, id = (i + 3 * step) << 2;
    f(a.x, ia); f(a.y, ia + 1); f(a.z, ia + 2); f(a.w, ia + 3);
    f(b.x, ib); f(b.y, ib + 1); f(b.z, ib + 2); f(b.w, ib + 3);
    f(c.x, ic); f(c.y, ic + 1); f(c.z, ic + 2); f(c.w, ic + 3);
    f(d.x, id); f(d.y, id + 1); f(d.z, id + 2); f(d.w, id + 3);
  }
  for (; i < n4; i += step) {
    const float4 a = r4[i];
    const int ia = i << 2;
    f(a.x, ia); f(a.y, ia + 1); f(a.z, ia + 2); f(a.w, ia + 3);
  }
  for (int t = (n4 << 2) + threadIdx.x; t < vocab; t += blockDim.x) f(row[t], t);
}

__global__ void __launch_bounds__(kSampThreads)
argmax_kernel(const float* __restrict__ logits, int64_t* __restrict__ out, int vocab, int ld) {
  __shared__ ArgMax sh[32];
  const float* row = logits + static_cast<size_t>(blockIdx.x) * ld;
  ArgMax a{-FLT_MAX, 0x7fffffff};
  for_each_logit(row, vocab, [&](float v, int i) { a = amax2(a, ArgMax{v, i}); });
  a = block_argmax(a, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = a.i;
}

// ---- threshold search for the top-k / top-p filters
// Wanted: the largest key t with measure{ i : fkey(x_i) >= t } >= target, where the measure is a count
// (MASS = false) or the softmax mass exp(x_i - mx) (MASS = true). The search keeps an interval [lo, hi]
// that holds t and `above` = measure{ key > hi }. One sixteen-way pass evaluates fifteen thresholds at
// once (per-thread bucket accumulators, one block reduction) and shrinks the interval sixteen-fold. A pass
// over the whole row costs about 70 instructions per element, so before every such pass the elements that
// still lie inside [lo, hi] are collected into shared memory; as soon as they fit (they do after one or
// two passes for any peaked distribution) the rest of the search runs on that list alone.
constexpr int kListPerWarp = 256;

struct SearchSmem {
  float list[(kSampThreads / 32) * kListPerWarp];   // per warp, in index order: x_i / T of the candidates
  float acc[(kSampThreads / 32) * 16];
  float tot[16];
  int wcnt[kSampThreads / 32];
  int over;
};

// Per warp (warp w scans its own contiguous share of the row): x / T of the elements with key in [lo, hi].
// Returns false if some warp found more than it can hold.
__device__ bool compact_range(const float* __restrict__ row, int vocab, float invT, uint32_t lo, uint32_t hi,
                              SearchSmem* sm) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) sm->over = 0;
  __syncthreads();
  // each warp owns a contiguous share of the row (a multiple of 128 elements, so float4 loads stay aligned);
  // candidates are appended in a fixed order (element slot of the float4, then lane), which keeps the list -
  // and with it every later floating-point sum - the same from run to run
  const int seg = (((vocab + 31) / 32) + 127) & ~127;
  const int beg = warp * seg;
  const int end = beg + seg < vocab ? beg + seg : vocab;
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  int cnt = 0;   // warp-uniform
  for (int i0 = beg; i0 < end && cnt <= kListPerWarp; i0 += 128) {
    const int i = i0 + 4 * lane;
    float xv[4] = {0.f, 0.f, 0.f, 0.f};
    if (vec && i + 3 < end) {
      const float4 q = *reinterpret_cast<const float4*>(row + i);
      xv[0] = q.x; xv[1] = q.y; xv[2] = q.z; xv[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) xv[e] = i + e < end ? row[i + e] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = xv[e] * invT;
      const uint32_t key = fkey(x);
      const bool in = i + e < end && key >= lo && key <= hi;
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int pos = cnt + __popc(m & ((1u << lane) - 1u));
        if (pos < kListPerWarp) sm->list[warp * kListPerWarp + pos] = x;
      }
      cnt += __popc(m);
    }
  }
  if (lane == 0) {
    sm->wcnt[warp] = cnt < kListPerWarp ? cnt : kListPerWarp;
    if (cnt > kListPerWarp) sm->over = 1;
  }
  __syncthreads();
  return sm->over == 0;
}

// One sixteen-way pass over the row (LIST = false) or over the collected candidates (LIST = true).
template <bool MASS, bool LIST>
__device__ void multiway_pass(const float* __restrict__ row, int vocab, float invT, float mx, SearchSmem* sm,
                              uint32_t& lo, uint32_t& hi, float target, float& above) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // bucket j = [lo + (j << sh), lo + ((j + 1) << sh)): a power-of-two width makes the bucket index a shift
  // (a division per element costs as much as the sixteen accumulations); sixteen buckets cover [lo, hi]
  const uint32_t span16 = (hi - lo) >> 4;
  const int sh = span16 == 0 ? 0 : 32 - __clz(span16);
  const uint32_t width = 1u << sh;
  float acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = 0.f;
  auto visit = [&](float x) {
    const uint32_t key = fkey(x);
    if (key < lo || key > hi) return;
    const int b = static_cast<int>((key - lo) >> sh);
    const float w = MASS ? __expf(x - mx) : 1.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j] += (b == j) ? w : 0.f;
  };
  bool empty = false;   // warp-uniform: a warp without candidates has nothing to add up
  if (LIST) {
    const int n = sm->wcnt[warp];
    empty = n == 0;
    for (int q = lane; q < n; q += 32) visit(sm->list[warp * kListPerWarp + q]);
  } else {
    for_each_logit(row, vocab, [&](float v, int) { visit(v * invT); });
  }
  if (empty) {
    if (lane < 16) sm->acc[warp * 16 + lane] = 0.f;
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
      if (lane == 0) sm->acc[warp * 16 + j] = acc[j];
    }
  }
  __syncthreads();
  // warp j adds bucket j over the 32 warps (lane q holds warp q's share); a loop over all of them in every
  // thread would cost 480 shared-memory reads per thread and pass, several microseconds
  if (warp < 16) {
    float t = sm->acc[lane * 16 + warp];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) sm->tot[warp] = t;
  }
  __syncthreads();
  // every thread derives the same decision: the highest bucket whose suffix measure reaches the target
  float run = above, above_new = 0.f;
  int best = 0;
  bool found = false;
  for (int j = 15; j >= 1; --j) {
    const float t = sm->tot[j];
    if (!found && run + t >= target) { best = j; found = true; above_new = run; }
    run += t;
  }
  if (!found) above_new = run;   // bucket 0 (its lower end is lo itself, which qualifies by the invariant)
  __syncthreads();
  // a qualifying bucket holds a key, so lo + best * width cannot wrap; the bucket's upper end can
  lo += static_cast<uint32_t>(best) * width;
  const uint64_t new_hi = static_cast<uint64_t>(lo) + width - 1;
  hi = new_hi < hi ? static_cast<uint32_t>(new_hi) : hi;
  above = above_new;
}

// Count (or softmax mass) of the collected candidates; every thread gets the same value.
template <bool MASS>
__device__ float list_measure(SearchSmem* sm, float mx) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float v = 0.f;
  if (MASS) {
    const int n = sm->wcnt[warp];
    for (int q = lane; q < n; q += 32) v += __expf(sm->list[warp * kListPerWarp + q] - mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  } else {
    v = static_cast<float>(sm->wcnt[warp]);
  }
  __syncthreads();
  if (lane == 0) sm->acc[warp] = v;
  __syncthreads();
  float tot = 0.f;
  for (int q = 0; q < kSampThreads / 32; ++q) tot += sm->acc[q];
  __syncthreads();
  return tot;
}

// Requires measure{ key >= lo } >= target and measure{ key > hi } == 0 on entry (hi = key of the maximum).
template <bool MASS>
__device__ uint32_t find_threshold(const float* __restrict__ row, int vocab, float invT, float mx, uint32_t lo,
                                   uint32_t hi, float target, SearchSmem* sm) {
  float above = 0.f;
  // Shortcut for the usual case that the wanted set sits within a few units below the maximum: collect the
  // elements of a window under the maximum in one cheap pass; if they fit and already reach the target, the
  // whole search runs on that list. Windows that hold too much (flat distributions) or too little fall
  // through to the general search.
  for (int wi = 0; wi < 3 && lo < hi; ++wi) {
    const float window = wi == 0 ? 2.f : (wi == 1 ? 6.f : 12.f);
    const uint32_t wlo = fkey(mx - window);
    if (wlo <= lo) break;                                   // the window is the whole remaining range
    if (!compact_range(row, vocab, invT, wlo, hi, sm)) break;   // too many candidates
    if (list_measure<MASS>(sm, mx) >= target) {
      lo = wlo;
      while (lo < hi) multiway_pass<MASS, true>(row, vocab, invT, mx, sm, lo, hi, target, above);
      return lo;
    }
  }
  while (lo < hi) {
    if (compact_range(row, vocab, invT, lo, hi, sm)) {
      while (lo < hi) multiway_pass<MASS, true>(row, vocab, invT, mx, sm, lo, hi, target, above);
      return lo;
    }
    multiway_pass<MASS, false>(row, vocab, invT, mx, sm, lo, hi, target, above);
  }
  return lo;
}

__global__ void __launch_bounds__(kSampThreads, 1)
sample_kernel(const float* __restrict__ logits, int64_t* __restrict__ out, int vocab, int ld,
              const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ min_p,
              const uint64_t* __restrict__ seeds, uint64_t step) {
  __shared__ ArgMax sh_am[32];
  __shared__ float sh_f[32];
  __shared__ float sh_scan[kSampThreads / 32];
  __shared__ SearchSmem sh_search;
  __shared__ int sh_pick;
  pdl_wait();
  pdl_trigger();
  const int rowi = blockIdx.x;
  const float* row = logits + static_cast<size_t>(rowi) * ld;
  const float T = temperature ? temperature[rowi] : 1.f;
  const int k = top_k ? top_k[rowi] : 0;
  const float tp = top_p ? top_p[rowi] : 1.f;
  const float mp = min_p ? min_p[rowi] : 0.f;
  const uint64_t seed = seeds ? seeds[rowi] : 0x1234ull + rowi;

  // greedy
  if (T <= 0.f || k == 1) {
    ArgMax a{-FLT_MAX, 0x7fffffff};
    for_each_logit(row, vocab, [&](float v, int i) { a = amax2(a, ArgMax{v, i}); });
    a = block_argmax(a, sh_am);
    if (threadIdx.x == 0) out[rowi] = a.i;
    return;
  }
  const float invT = 1.f / T;
  const bool use_k = k > 0 && k < vocab, use_p = tp < 1.f, use_m = mp > 0.f;
  if (!use_k && !use_p && !use_m) {
    // Gumbel-max: argmax(x/T + g), g = -log(-log u)
    ArgMax a{-FLT_MAX, 0x7fffffff};
    for_each_logit(row, vocab, [&](float v, int i) {
      const float u = uniform01(seed, step, i);
      a = amax2(a, ArgMax{v * invT - __logf(-__logf(u)), i});
    });
    a = block_argmax(a, sh_am);
    if (threadIdx.x == 0) out[rowi] = a.i;
    return;
  }
  // max of scaled logits
  ArgMax a{-FLT_MAX, 0x7fffffff};
  for_each_logit(row, vocab, [&](float v, int i) { a = amax2(a, ArgMax{v * invT, i}); });
  a = block_argmax(a, sh_am);
  const float mx = a.v;
  uint32_t thr_key = 0;  // keep x with fkey(x*invT) >= thr_key
  if (use_k) {
    // largest key t with count(key >= t) >= k
    const uint32_t lo = find_threshold<false>(row, vocab, invT, mx, 0u, fkey(mx), static_cast<float>(k), &sh_search);
    thr_key = lo;
  }
  if (use_m) {
    const uint32_t km = fkey(mx + __logf(mp));
    thr_key = max(thr_key, km);
  }
  float Z = 0.f;
  for_each_logit(row, vocab, [&](float v, int) {
    const float x = v * invT;
    Z += fkey(x) >= thr_key ? __expf(x - mx) : 0.f;
  });
  Z = block_sum_f(Z, sh_f);
  if (use_p) {
    // largest key t (>= thr_key) with mass(key >= t) >= tp * Z
    const float target = tp * Z;
    const uint32_t lo = find_threshold<true>(row, vocab, invT, mx, thr_key, fkey(mx), target, &sh_search);
    thr_key = lo;
    Z = 0.f;
    for_each_logit(row, vocab, [&](float v, int) {
      const float x = v * invT;
      Z += fkey(x) >= thr_key ? __expf(x - mx) : 0.f;
    });
    Z = block_sum_f(Z, sh_f);
  }
  // inverse-CDF draw over the kept set, in index order
  const float target = uniform01(seed, step, 0xffffffffull) * Z;
  if (threadIdx.x == 0) sh_pick = -1;
  __syncthreads();
  float base = 0.f;
  int last_kept = -1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  for (int c0 = 0; c0 < vocab; c0 += 4 * kSampThreads) {
    // four consecutive elements per thread and iteration
    const int i = c0 + 4 * threadIdx.x;
    float xv[4] = {0.f, 0.f, 0.f, 0.f};
    if (vec && i + 3 < vocab) {
      const float4 q = *reinterpret_cast<const float4*>(row + i);
      xv[0] = q.x; xv[1] = q.y; xv[2] = q.z; xv[3] = q.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) xv[e] = i + e < vocab ? row[i + e] : 0.f;
    }
    float w[4];
    float mine = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = xv[e] * invT;
      w[e] = (i + e < vocab && fkey(x) >= thr_key) ? __expf(x - mx) : 0.f;
      mine += w[e];
    }
    float incl = mine;  // warp inclusive scan of the per-thread sums
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) sh_scan[warp] = incl;
    __syncthreads();
    float woff = 0.f, total = 0.f;
    for (int q = 0; q < kSampThreads / 32; ++q) {
      const float t = sh_scan[q];
      if (q < warp) woff += t;
      total += t;
    }
    float cum = base + woff + incl - mine;   // mass before this thread's first element
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (w[e] > 0.f) {
        if (cum + w[e] >= target && cum < target) atomicMax(&sh_pick, i + e);
        last_kept = i + e;
      }
      cum += w[e];
    }
    base += total;
    __syncthreads();
    if (sh_pick >= 0) break;
  }
  if (sh_pick < 0) {
    // rounding left the target just above the total mass: take the last kept index
    ArgMax b{static_cast<float>(last_kept), last_kept < 0 ? 0x7fffffff : -last_kept};
    b = block_argmax(b, sh_am);
    if (threadIdx.x == 0) out[rowi] = b.v >= 0.f ? static_cast<int64_t>(b.v) : a.i;
  } else if (threadIdx.x == 0) {
    out[rowi] = sh_pick;
  }
}

// ---- a row spread over a cluster of CTAs
// The 16 c warps of a cluster each own a contiguous share of the row and read it two or three times (L2 hits after the
// first). Greedy and plain-temperature rows are one pass. Top-k and min-p rows take the maximum and then go straight to the
// elements of the bins of mx - x / T (1/32 wide) that can hold the kept set; those (at most kList) go to the first CTA, which
// ranks them by counting and reads both cut-offs off the sorted values. A nucleus over the whole row takes the maximum, then a
// histogram of the bins' softmax mass in shared memory (bins that narrow spread the bulk of the row over hundreds of counters,
// so the atomics hardly meet), then the weight above the bin in which it ends and that bin's elements, among which the first
// CTA finds the cut-off by their keys. What does not fit (more candidates than the lists hold, cut-offs in the open last bin, a
// nucleus within a long top-k) is found exactly by refining the bin it lies in, 1024 buckets of keys at a time (a few more
// passes), and the draw is a prefix sum over the warps' shares.
// Masses are integers, so sums do not depend on their order: 42 fractional bits where few weights meet in registers, and
// per bin the weights relative to the bin's upper edge as 26-bit numbers in two halves, because 32-bit atomics on shared
// memory are native and 64-bit ones are not.
// What bounds it: the chain of a nucleus row. Of its 51 thousand cycles (64 rows, two CTAs an SM) the histogram takes 20, nine
// cycles an atomic and SM; the passes over the row 6 (from memory) and 9; the rest are barriers of the cluster and round trips
// between its CTAs, each about one.
// 64 rows of 128256 logits with top-k, top-p and min-p mixed: 31 us (64 when every row was counted, elements in the order of a
// long list were ranked one by one, and a bin refined over the cluster), 20 rows 25 us (54), one row 19 us (28); 64 greedy
// rows 11 us.
constexpr int kClu = 8;          // largest cluster; the launcher picks 8, 4, 2 or 1 CTAs per row from the batch size
constexpr int kCluThreads = 512, kCluWarps = kCluThreads / 32;
constexpr int kBins = 1024, kOwn = kBins / kCluThreads;   // 32 units: what lies below weighs nothing
static_assert(kOwn == 2, "a thread reads its bins as one vector");
constexpr int kList = kCluThreads;
constexpr int kBinList = 2048;   // halves of 2^11 weights below 2^42 add up below 2^32
constexpr float kBinsPerUnit = 32.f;
constexpr int kMaxShare = 1 << 18;   // elements per CTA: the halves of 2^18 weights of one bin still add up below 2^32
typedef unsigned long long u64;

struct ClusterSmem {
  uint32_t cnt[kBins], hi[kBins], lo[kBins];
  float lx[kList];              // x / T of the candidates and their indices, as they arrive (first CTA only)
  int li[kList];
  float sx[kList];              // by rank
  u64 sp[kList];                // by rank: inclusive prefix of the masses
  float ox[kList];              // by index
  int oi[kList];
  float bx[kBinList];           // elements of the bin in which a nucleus ends and their indices (first CTA only)
  int bi[kBinList];
  uint32_t kept_hi[kClu * kCluWarps], kept_lo[kClu * kCluWarps];   // their weights by owning warp, in two halves
  ArgMax cmax;                  // maximum of this CTA's share
  u64 wsum[kCluWarps];          // kept mass of every warp's share
  u64 all[kClu * kCluWarps];
  u64 red[kCluWarps];
  u64 above;
  int bin, n, cut;
  uint32_t fill;
};

__device__ __forceinline__ void load4(const float* __restrict__ row, int i, int end, bool vec, float (&xv)[4]) {
  if (vec && i + 3 < end) {
    const float4 q = *reinterpret_cast<const float4*>(row + i);
    xv[0] = q.x; xv[1] = q.y; xv[2] = q.z; xv[3] = q.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) xv[e] = i + e < end ? row[i + e] : -FLT_MAX;
  }
}
// 2^-42 is the smallest weight: a token about 29 units below the maximum is not drawn (uniform01 has 24 bits, so that no draw
// could tell it from one of weight 1e-38). NaN (an infinite maximum minus itself, a NaN logit) weighs nothing.
__device__ __forceinline__ u64 weight_of(float below) { return __float2ull_rn(fmaxf(__expf(-below) * 4398046511104.f, 0.f)); }
// The bin of an element `below` >= 0 under the maximum; NaN goes to the last bin. Rounding down while adding 2^23 leaves the
// integer in the low bits: conversions run on the unit of the exponentials, 16 lanes a cycle, and four of those per element
// were what a counting pass took its time for (31 cycles per 32 elements and scheduler).
__device__ __forceinline__ int bin_of(float below) {
  return __float_as_int(__fadd_rd(fminf(below * kBinsPerUnit, static_cast<float>(kBins - 1)), 8388608.f)) - 0x4b000000;
}
// the lowest bin that min-p reaches (negative: none but the maximum's)
__device__ __forceinline__ int min_p_bin(float mp) {
  const float b = (0.01f - __logf(mp)) * kBinsPerUnit;
  return b < static_cast<float>(kBins - 1) ? static_cast<int>(b) : kBins - 1;
}
// e^-y as a 26-bit fraction. Elements of one bin have y below 1/32, where four terms of the series are within 2^-25 and the
// sum's own bits are the fraction.
__device__ __forceinline__ uint32_t fraction26(float y) {
  if (y < 0.0625f) {
    const float e = fmaf(-y, fmaf(-y, fmaf(-y, fmaf(-y, 1.f / 24.f, 1.f / 6.f), 0.5f), 1.f), 1.f);
    return e < 1.f ? ((__float_as_uint(e) & 0x7fffffu) | 0x800000u) << 2 : 1u << 26;
  }
  return __float2uint_rn(__expf(-y) * 67108864.f);
}
__device__ __forceinline__ uint2 ld_cluster_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster_u64(uint32_t addr, u64 v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ u64 ld_cluster_u64(uint32_t addr) {
  u64 v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
// sum of `mine` over the threads before this one, and over all of them
__device__ __forceinline__ u64 block_before(u64 mine, u64* red, u64& total) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  u64 incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u64 t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  u64 before = 0;
  total = 0;
#pragma unroll
  for (int q = 0; q < kCluWarps; ++q) {
    const u64 t = red[q];
    if (q < warp) before += t;
    total += t;
  }
  __syncthreads();
  return before + incl - mine;
}

__global__ void __launch_bounds__(kCluThreads, 2)
sample_cluster_kernel(const float* __restrict__ logits, int64_t* __restrict__ out, int vocab, int ld,
                      const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
                      const float* __restrict__ top_p, const float* __restrict__ min_p,
                      const uint64_t* __restrict__ seeds, uint64_t step) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  ClusterSmem* sm = reinterpret_cast<ClusterSmem*>(sm_raw);
  __shared__ ArgMax sh_am[32];
  pdl_wait();
  pdl_trigger();
  const int rowi = blockIdx.y, tid = threadIdx.x;
  const uint32_t rank = cluster_ctarank(), nclu = cluster_nctarank();
  const int warp = tid >> 5, lane = tid & 31;
  const float* row = logits + static_cast<size_t>(rowi) * ld;
  const float T = temperature ? temperature[rowi] : 1.f;
  const int k = top_k ? top_k[rowi] : 0;
  const float tp = top_p ? top_p[rowi] : 1.f;
  const float mp = min_p ? min_p[rowi] : 0.f;
  const uint64_t seed = seeds ? seeds[rowi] : 0x1234ull + rowi;
  const bool greedy = T <= 0.f || k == 1;
  const bool use_k = k > 0 && k < vocab, use_p = tp < 1.f, use_m = mp > 0.f;
  const bool plain = !greedy && !(use_k || use_p || use_m);
  const float invT = greedy ? 1.f : 1.f / T;
  const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  // warp g of the cluster owns [g * seg, (g + 1) * seg): a multiple of 128 elements (aligned float4 loads)
  const int nwarps = static_cast<int>(nclu) * kCluWarps;
  const int seg = (((vocab + nwarps - 1) / nwarps) + 127) & ~127;
  const int gw = static_cast<int>(rank) * kCluWarps + warp;
  const int beg = static_cast<long long>(gw) * seg < vocab ? gw * seg : vocab;
  const int end = vocab - beg < seg ? vocab : beg + seg;
  // f(x / T, index) for every element of this warp's share, sixteen loads in flight per lane (-0 as 0: equal values are
  // one tie, whatever their sign bit)
  auto visit = [&](auto&& f) {
    int i0 = beg;
    for (; vec && i0 + 512 <= end; i0 += 512) {
      float4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = *reinterpret_cast<const float4*>(row + i0 + u * 128 + 4 * lane);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * 128 + 4 * lane;
        f(__fadd_rn(__fmul_rn(q[u].x, invT), 0.f), i);
        f(__fadd_rn(__fmul_rn(q[u].y, invT), 0.f), i + 1);
        f(__fadd_rn(__fmul_rn(q[u].z, invT), 0.f), i + 2);
        f(__fadd_rn(__fmul_rn(q[u].w, invT), 0.f), i + 3);
      }
    }
    for (; i0 < end; i0 += 512) {
      float xv[4][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) load4(row, i0 + u * 128 + 4 * lane, end, vec, xv[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + u * 128 + 4 * lane + e;
          if (i < end) f(__fadd_rn(__fmul_rn(xv[u][e], invT), 0.f), i);
        }
    }
  };

  auto clear_bins = [&](int want) {
    for (int i = 4 * tid; i < kBins; i += 4 * kCluThreads) {
      const uint4 z = make_uint4(0u, 0u, 0u, 0u);
      if (want & 1) *reinterpret_cast<uint4*>(&sm->cnt[i]) = z;
      if (want & 2) { *reinterpret_cast<uint4*>(&sm->hi[i]) = z; *reinterpret_cast<uint4*>(&sm->lo[i]) = z; }
    }
  };
  if (!greedy && !plain) clear_bins(3);

  // 1. maximum of x / T (greedy: of x; no filter: of x / T + Gumbel noise, which is the draw)
  ArgMax a{-FLT_MAX, 0x7fffffff};
  if (plain) {
    visit([&](float x, int i) { a = amax2(a, ArgMax{x - __logf(-__logf(uniform01(seed, step, i))), i}); });
  } else {
    visit([&](float x, int i) { a = amax2(a, ArgMax{x, i}); });
  }
  const float lane_max = a.v;
  a = block_argmax(a, sh_am);
  if (tid == 0) { sm->cmax = a; sm->fill = 0; }
  cluster_sync_all();
  {
    // lane r asks CTA r: one round trip, where a loop over the CTAs would take one each
    ArgMax g{-FLT_MAX, 0x7fffffff};
    if (lane < static_cast<int>(nclu)) {
      g.v = __uint_as_float(ld_cluster_u32(mapa_shared(&sm->cmax.v, lane)));
      g.i = static_cast<int>(ld_cluster_u32(mapa_shared(&sm->cmax.i, lane)));
    }
#pragma unroll
    for (int o = 1; o < kClu; o <<= 1) {
      ArgMax b;
      b.v = __shfl_xor_sync(0xffffffffu, g.v, o);
      b.i = __shfl_xor_sync(0xffffffffu, g.i, o);
      g = amax2(g, b);
    }
    g.v = __shfl_sync(0xffffffffu, g.v, 0);
    g.i = __shfl_sync(0xffffffffu, g.i, 0);
    a = g;
  }
  if (greedy || plain) {           // the same decision in all CTAs of the cluster
    if (rank == 0 && tid == 0) out[rowi] = a.i;
    cluster_sync_all();            // nobody leaves while a peer may still read its maximum
    return;
  }
  const float mx = a.v;
  const uint32_t hi_key = fkey(mx);
  const uint32_t km = use_m ? fkey(mx + __logf(mp)) : 0u;

  // Weights relative to the edge of unit bin b (or of bin `all_in`, where every element placed lies), 26 bits, in units of
  // 2^-42 under the maximum: 2^16 e^(-b / 32). One exponential per thread covers its bins.
  constexpr double kStep[kOwn] = {1.0, 0.9692332344763441};                  // e^(-j / 32)
  auto edge = [](int b) { return 65536.0 * exp(-b / static_cast<double>(kBinsPerUnit)); };
  auto count_in = [&](int want, int b, int rel, float below) {
    if (want & 1) atomicAdd(&sm->cnt[b], 1u);
    if (want & 2) {
      const uint32_t q = fraction26(below - rel / kBinsPerUnit);
      atomicAdd(&sm->hi[b], q >> 13);
      atomicAdd(&sm->lo[b], q & 0x1fffu);
    }
  };
  // This thread's kOwn bins, added up over CTAs [r0, r1), as counts (want & 1) and masses (want & 2).
  auto add_bins = [&](int want, bool scaled, double unit, uint32_t r0, uint32_t r1, u64 (&c)[kOwn], u64 (&m)[kOwn]) {
#pragma unroll
    for (int j = 0; j < kOwn; ++j) c[j] = m[j] = 0;
#pragma unroll 4
    for (uint32_t r = r0; r < r1; ++r) {
      if (want & 1) {
        const uint2 v = ld_cluster_v2(mapa_shared(&sm->cnt[tid * kOwn], r));
        c[0] += v.x; c[1] += v.y;
      }
      if (want & 2) {
        const uint2 h = ld_cluster_v2(mapa_shared(&sm->hi[tid * kOwn], r)), l = ld_cluster_v2(mapa_shared(&sm->lo[tid * kOwn], r));
        m[0] += (static_cast<u64>(h.x) << 13) + l.x; m[1] += (static_cast<u64>(h.y) << 13) + l.y;
      }
    }
    if (want & 2) {
#pragma unroll
      for (int j = 0; j < kOwn; ++j)
        if (m[j]) m[j] = static_cast<u64>(static_cast<double>(m[j]) * (scaled ? unit * kStep[j] : unit));
    }
  };
  // Histogram over the cluster: place(x, below, key) gives an element's bin or -1; `all_in` is the unit bin that holds every
  // element placed, or -1 when the bins are the unit bins themselves. `fresh`: the bins are still those cleared at the start.
  auto histogram = [&](int want, int all_in, double unit, bool fresh, auto&& place, u64 (&c)[kOwn], u64 (&m)[kOwn]) {
    if (!fresh) {
      cluster_sync_all();          // peers are done reading the bins of the pass before
      clear_bins(want);
      __syncthreads();
    }
    visit([&](float x, int) {
      const float below = __fsub_rn(mx, x);
      const int b = place(below, fkey(x));
      if (b >= 0) count_in(want, b, all_in < 0 ? b : all_in, below);
    });
    cluster_sync_all();
    add_bins(want, all_in < 0, unit, 0, nclu, c, m);
  };
  // the first bin where the running sum of v reaches `target` (-1: none) and the sum before it
  // (`full` scales what one element of this thread's first bin weighs at most: sm->n then tells how many the bin has at least)
  auto cross = [&](const u64 (&v)[kOwn], u64 target, int& bin, u64& above, float full = 0.f) {
    if (tid == 0) sm->bin = -1;
    u64 sum = 0, total;
#pragma unroll
    for (int j = 0; j < kOwn; ++j) sum += v[j];
    u64 run = block_before(sum, sm->red, total);
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      if (run < target && run + v[j] >= target) {
        sm->bin = tid * kOwn + j;
        sm->above = run;
        if (full > 0.f) sm->n = static_cast<int>(fminf(__ull2float_rz(v[j]) / (full * static_cast<float>(kStep[j])), 1e9f));
      }
      run += v[j];
    }
    __syncthreads();
    bin = sm->bin;
    above = sm->above;
    __syncthreads();
  };
  // the part of `whole` that a fraction in (0, 1) covers, at least 1
  auto portion = [](float f, u64 whole) {
    const double t = ceil(static_cast<double>(f) * static_cast<double>(whole));
    const u64 r = t < 1.0 ? 1 : static_cast<u64>(t);
    return r > whole ? whole : r;
  };

  // 2. The bins that hold the kept set. A top-k set lies in the bins that reach k when every lane of the cluster counts only its
  // maximum, and what min-p keeps is known from the maximum, so such rows go straight to the elements of those bins (2a): a
  // pass less than counting the row first, and no atomics for what cannot be kept (20 of 60 thousand cycles). Up to half a list:
  // the bins that the lanes' maxima reach hold more than k elements, and a list that runs over costs its pass. Where they are
  // too many, and for a nucleus over the whole row, the row is counted (2b).
  u64 c[kOwn], m[kOwn], z_all = 0;
  const bool nucleus = use_p && !use_k && !use_m;
  int last = -1, kbin = -1, n = 0x7fffffff;
  u64 kabove = 0, pabove = 0, ptarget = 0;
  bool listed = false;
  // a bound under every element of bins 0 .. b (none for the last bin, which is open): most elements need no look at their bin
  auto under = [&](int b) { return b >= kBins - 1 ? -INFINITY : mx - (b + 1) / kBinsPerUnit - fmaxf(fabsf(mx), 64.f) * 2e-6f; };
  // an element of the list in the first CTA
  auto push = [&](float* xs, int* is, uint32_t pos, float x, int i) {
    st_cluster_u32(mapa_shared(xs, 0) + 4u * pos, __float_as_uint(x == x ? x : -INFINITY));      // ranks need an order: NaN is the lowest
    st_cluster_u32(mapa_shared(is, 0) + 4u * pos, static_cast<uint32_t>(i));
  };
  if (!nucleus && k <= kList / 2) {
    if (use_k) {
      atomicAdd(&sm->cnt[bin_of(__fsub_rn(mx, lane_max))], 1u);
      cluster_sync_all();
      add_bins(1, false, 0.0, 0, nclu, c, m);
      cross(c, static_cast<u64>(k), last, kabove);
    }
    if (use_m && (last >= 0 || !use_k)) last = max(last, min_p_bin(mp));
    if (last >= 0) {
      const float least = under(last);
      // What min-p reaches may be much more than a list. Lanes that have something to list tell (n elements spread over L lanes leave e^(-n / L)
      // of them without): from a quarter more than a list on, the pass is not begun, if lanes have eight elements or more. The sum below then
      // says so to the whole cluster. (min_p 1e-4 on 128256 logits: 64 rows 53 us, 49 without the pass.)
      if (use_m && seg > 128 && __syncthreads_count(lane_max >= least) > static_cast<int>(kCluThreads * (1.f - __expf(-1.25f / nclu)))) {
        if (tid == 0) sm->fill = kList + 1;
      } else {
        visit([&](float x, int i) {
          if (x < least || bin_of(__fsub_rn(mx, x)) > last) return;
          const uint32_t pos = atomicAdd(&sm->fill, 1u);
          if (pos < kList) { sm->sx[pos] = x; sm->oi[pos] = i; }
        });
      }
      cluster_sync_all();
      const uint32_t there = lane < static_cast<int>(nclu) ? ld_cluster_u32(mapa_shared(&sm->fill, lane)) : 0u;
      const uint32_t first = __reduce_add_sync(0xffffffffu, lane < static_cast<int>(rank) ? there : 0u);
      const uint32_t all = __reduce_add_sync(0xffffffffu, there);
      if (all <= kList && static_cast<int>(all) >= (use_k ? k : 1)) {
        listed = true;
        n = static_cast<int>(all);
        if (tid < static_cast<int>(sm->fill)) push(sm->lx, sm->li, first + tid, sm->sx[tid], sm->oi[tid]);
        cluster_sync_all();
        if (rank != 0) return;
      }
    }
  }
  if (!listed) {
    // 2b. bins under the maximum
    const double unit = nucleus ? edge(tid * kOwn) : 0.0;
    const bool fresh = nucleus || k > kList / 2;
    bool fits = false;
    // (the last bin's elements have no weight)
    if (nucleus) histogram(2, -1, unit, fresh, [](float below, uint32_t) { const int b = bin_of(below); return b < kBins - 1 ? b : -1; }, c, m);
    else histogram(1, -1, unit, fresh, [](float below, uint32_t) { return bin_of(below); }, c, m);
    last = -1;
    if (nucleus) {
      block_before(m[0] + m[1], sm->red, z_all);
      ptarget = portion(tp, z_all);
      // The bin's mass says how many elements it has at least, up to 1/32 too few: more than the list holds would cost a pass for
      // nothing (flat rows of 128256, T = 5: 74 us for one and 500 for 300, 64 and 408 without that pass).
      cross(m, ptarget, last, pabove, static_cast<float>(unit) * 67108864.f);
      fits = last >= 0 && last < kBins - 1 && sm->n < kBinList;
    } else {
      if (use_k) { cross(c, static_cast<u64>(k), kbin, kabove); last = kbin; }
      if (use_m) last = max(last, min_p_bin(mp));
      u64 total, run = block_before(c[0] + c[1], sm->red, total);
#pragma unroll
      for (int j = 0; j < kOwn; ++j) {
        run += c[j];
        if (tid * kOwn + j == last) sm->n = run > 0x7fffffffu ? 0x7fffffff : static_cast<int>(run);
      }
      __syncthreads();
      if (last >= 0) n = sm->n;
    }
    uint32_t all = 0x7fffffffu;
    if (fits) {
      // One more pass takes the weight of the bins above the last one, warp by warp, and the last bin's elements, which go to
      // the first CTA: it finds the cut-off among them and draws.
      const float least = under(last);
      u64 mass = 0;
      // a lane marks its elements that can be kept, then takes them one by one: a few of sixteen, in other places in every lane
      auto take = [&](float x, int i) {
        const float below = __fsub_rn(mx, x);
        const int b = bin_of(below);
        if (b > last) return;
        if (b < last) { mass += weight_of(below); return; }
        const uint32_t pos = atomicAdd(&sm->fill, 1u);
        if (pos < kBinList) { sm->bx[pos] = x; sm->bi[pos] = i; }
      };
      for (int i0 = beg; i0 < end; i0 += 512) {
        float xv[4][4];
        uint32_t mark = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) load4(row, i0 + u * 128 + 4 * lane, end, vec, xv[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (__fmul_rn(xv[u][e], invT) >= least) mark |= 1u << (4 * u + e);
        while (mark) {
          const int j = __ffs(mark) - 1, i = i0 + (j >> 2) * 128 + 4 * lane + (j & 3);
          mark &= mark - 1;
          if (i < end) take(__fadd_rn(__fmul_rn(row[i], invT), 0.f), i);
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
      if (lane == 0) st_cluster_u64(mapa_shared(&sm->all[gw], 0), mass);
      cluster_sync_all();
      const uint32_t there = lane < static_cast<int>(nclu) ? ld_cluster_u32(mapa_shared(&sm->fill, lane)) : 0u;
      const uint32_t first = __reduce_add_sync(0xffffffffu, lane < static_cast<int>(rank) ? there : 0u);
      all = __reduce_add_sync(0xffffffffu, there);
      if (all < kBinList && rank != 0)                 // the first CTA's own elements lie at the front already
        for (uint32_t j = tid; j < sm->fill; j += kCluThreads) push(sm->bx, sm->bi, first + j, sm->bx[j], sm->bi[j]);
    }
    if (all < kBinList) {
      cluster_sync_all();
      if (rank != 0) return;
      const int in_last = static_cast<int>(all);
      const float slack = fmaxf(fabsf(mx), 64.f) * 2e-6f;    // rounding of mx - x
      uint32_t khi = min(hi_key, fkey(mx - last / kBinsPerUnit + slack));
      uint32_t klo = min(fkey(mx - (last + 1) / kBinsPerUnit - slack), khi);
      uint32_t from = 0u, to = 0xffffffffu, thr = klo;
      const double at = edge(last);
      if (tid < kClu * kCluWarps) { sm->kept_hi[tid] = 0; sm->kept_lo[tid] = 0; }
      for (;;) {
        const uint32_t range = khi - klo;
        const int sh = range < static_cast<uint32_t>(kBins) ? 0 : 22 - __clz(range);
        clear_bins(2);
        __syncthreads();
        for (int j = tid; j < in_last; j += kCluThreads) {
          const float x = sm->bx[j];
          const uint32_t key = fkey(x);
          if (key >= from && key <= to) count_in(2, static_cast<int>((khi - min(max(key, klo), khi)) >> sh), last, __fsub_rn(mx, x));
        }
        __syncthreads();
        add_bins(2, false, at, 0, 1, c, m);
        int b;
        u64 before;
        cross(m, ptarget - pabove, b, before);
        thr = klo;
        if (b < 0) break;
        pabove += before;
        const uint32_t top = khi - (static_cast<uint32_t>(b) << sh);
        thr = top;
        if (sh == 0) break;
        const uint32_t width = (1u << sh) - 1;
        klo = top - klo < width ? klo : top - width;
        khi = top;
        from = klo;
        to = khi;
      }
      // inverse-CDF draw in index order: the shares' masses, then the share that holds the target
      for (int j = tid; j < in_last; j += kCluThreads) {
        if (fkey(sm->bx[j]) < thr) continue;
        const u64 w = weight_of(__fsub_rn(mx, sm->bx[j]));
        atomicAdd(&sm->kept_hi[sm->bi[j] / seg], static_cast<uint32_t>(w >> 21));
        atomicAdd(&sm->kept_lo[sm->bi[j] / seg], static_cast<uint32_t>(w) & 0x1fffffu);
      }
      __syncthreads();
      u64 Z;
      const u64 mine = tid < nwarps ? sm->all[tid] + (static_cast<u64>(sm->kept_hi[tid]) << 21) + sm->kept_lo[tid] : 0;
      const u64 base = block_before(mine, sm->red, Z);
      if (Z == 0) {
        if (tid == 0) out[rowi] = a.i;
        return;
      }
      const u64 target = portion(uniform01(seed, step, 0xffffffffull), Z);
      if (base < target && base + mine >= target) { sm->bin = tid; sm->above = base; }
      __syncthreads();
      const int s0 = sm->bin * seg, s1 = vocab - s0 < seg ? vocab : s0 + seg;
      u64 run = sm->above;
      for (int i0 = s0; i0 < s1 && run < target; i0 += 4 * kCluThreads) {
        float xv[4];
        load4(row, i0 + 4 * tid, s1, vec, xv);
        u64 w[4], four = 0, total;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = __fadd_rn(__fmul_rn(xv[e], invT), 0.f);
          w[e] = (i0 + 4 * tid + e < s1 && fkey(x) >= thr) ? weight_of(__fsub_rn(mx, x)) : 0;
          four += w[e];
        }
        u64 cum = run + block_before(four, sm->red, total);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (w[e] > 0 && cum < target && cum + w[e] >= target) out[rowi] = i0 + 4 * tid + e;
          cum += w[e];
        }
        run += total;
      }
      return;
    } else if (n <= kList) {
      // elements of the bins up to the last into a list of the first CTA, in any order within a CTA's part of it. The positions
      // come from a local counter: one shared by the cluster is a queue of remote atomics (512 of them took 25 us).
      u64 part = 0, here;
#pragma unroll
      for (int j = 0; j < kOwn; ++j)
        if (tid * kOwn + j <= last) part += sm->cnt[tid * kOwn + j];
      block_before(part, sm->red, here);
      if (tid == 0) { sm->wsum[0] = here; sm->fill = 0; }
      cluster_sync_all();
      const uint32_t first = __reduce_add_sync(0xffffffffu, lane < static_cast<int>(rank) ? static_cast<uint32_t>(ld_cluster_u64(mapa_shared(&sm->wsum[0], lane))) : 0u);
      const float least = under(last);
      visit([&](float x, int i) {
        if (x < least || bin_of(__fsub_rn(mx, x)) > last) return;
        const uint32_t pos = first + atomicAdd(&sm->fill, 1u);
        if (pos < kList) push(sm->lx, sm->li, pos, x, i);      // always: the same elements were counted
      });
      cluster_sync_all();
      if (rank != 0) return;
      listed = true;
    }
  }

  if (listed) {
    // 3a. the first CTA alone
    // one candidate per thread: its rank by value and by index, counted directly
    const int n4 = (n + 3) & ~3;
    if (tid >= n && tid < n4) { sm->lx[tid] = -INFINITY; sm->li[tid] = 0x7fffffff; }   // behind every candidate, masked ones too
    if (tid == 0) sm->cut = -1;
    __syncthreads();
    float x = 0.f;
    int rk = 0;
    if (tid < n) {
      x = sm->lx[tid];
      const int id = sm->li[tid];
      int ri = 0;
      for (int j = 0; j < n4; j += 4) {
        const float4 q = *reinterpret_cast<const float4*>(&sm->lx[j]);
        const int4 o = *reinterpret_cast<const int4*>(&sm->li[j]);
        rk += (q.x > x || (q.x == x && o.x < id)) + (q.y > x || (q.y == x && o.y < id)) + (q.z > x || (q.z == x && o.z < id)) +
              (q.w > x || (q.w == x && o.w < id));
        ri += (o.x < id) + (o.y < id) + (o.z < id) + (o.w < id);
      }
      sm->sx[rk] = x;
      sm->ox[ri] = x;
      sm->oi[ri] = id;
    }
    __syncthreads();
    u64 total;
    const u64 mine = tid < n ? weight_of(__fsub_rn(mx, sm->sx[tid])) : 0;
    const u64 incl = block_before(mine, sm->red, total) + mine;
    sm->sp[tid] = incl;
    __syncthreads();
    const float mx_rank = tid < n ? sm->sx[tid] : 0.f;
    const uint32_t mykey = fkey(mx_rank);
    uint32_t thr = 0;
    if (use_k) thr = fkey(sm->sx[k - 1]);                  // k <= n by the choice of the bins
    if (use_m) thr = max(thr, km);
    if (thr > hi_key) thr = hi_key;                        // a min_p above one keeps the maximum alone
    const int kept = __syncthreads_count(tid < n && mykey >= thr);
    if (use_p && kept > 0) {
      const u64 target = portion(tp, sm->sp[kept - 1]);
      if (tid < kept && incl >= target && incl - mine < target) sm->cut = tid;
      __syncthreads();
      const int r = sm->cut >= 0 ? sm->cut : kept - 1;
      thr = max(thr, fkey(sm->sx[r]));
    }
    // inverse-CDF draw over the kept entries in index order
    const float xo = tid < n ? sm->ox[tid] : 0.f;
    const u64 w = (tid < n && fkey(xo) >= thr) ? weight_of(__fsub_rn(mx, xo)) : 0;
    const u64 cum = block_before(w, sm->red, total);
    const u64 target = portion(uniform01(seed, step, 0xffffffffull), total);
    if (w > 0 && cum < target && cum + w >= target) out[rowi] = sm->oi[tid];
    if (total == 0 && tid == 0) out[rowi] = a.i;           // nothing has a weight (infinite or NaN logits)
    return;
  }

  // 3b. exact cut-offs by refining the bin they lie in
  auto refine = [&](int want, uint32_t least, int bin, u64 above, u64 target) -> uint32_t {
    const float slack = fmaxf(fabsf(mx), 64.f) * 2e-6f;    // rounding of mx - x
    uint32_t khi = min(hi_key, fkey(mx - bin / kBinsPerUnit + slack));
    uint32_t klo = bin == kBins - 1 ? 0u : fkey(mx - (bin + 1) / kBinsPerUnit - slack);
    klo = min(max(klo, least), khi);
    uint32_t from = 0u, to = 0xffffffffu;
    const double at = want & 2 ? edge(bin) : 0.0;
    for (;;) {
      const uint32_t range = khi - klo;
      const int sh = range < static_cast<uint32_t>(kBins) ? 0 : 22 - __clz(range);
      histogram(want, bin, at, false, [&](float below, uint32_t key) {
        if (key < from || key > to || key < least || bin_of(below) != bin) return -1;
        return static_cast<int>((khi - min(max(key, klo), khi)) >> sh);
      }, c, m);
      int b;
      u64 before;
      cross(want & 1 ? c : m, target - above, b, before);
      if (b < 0) return klo;
      above += before;
      const uint32_t top = khi - (static_cast<uint32_t>(b) << sh);
      if (sh == 0) return top;
      const uint32_t width = (1u << sh) - 1;
      klo = top - klo < width ? klo : top - width;
      khi = top;
      from = klo;
      to = khi;
    }
  };
  uint32_t thr = 0;
  if (use_k) thr = kbin >= 0 ? refine(1, 0u, kbin, kabove, static_cast<u64>(k)) : 0u;
  if (use_m) thr = max(thr, km);
  if (thr > hi_key) thr = hi_key;
  if (use_p) {
    int bin = last;
    if (!nucleus) {                                        // the mass of what the other filters keep
      const uint32_t least = thr;
      histogram(2, -1, edge(tid * kOwn), false, [&](float below, uint32_t key) { return key >= least ? bin_of(below) : -1; }, c, m);
      block_before(m[0] + m[1], sm->red, z_all);
      ptarget = portion(tp, z_all);
      cross(m, ptarget, bin, pabove);
    }
    if (bin >= 0) thr = max(thr, refine(2, thr, bin, pabove, ptarget));
  }
  // inverse-CDF draw in index order: the shares' masses, then the share that holds the target
  u64 mass = 0;
  visit([&](float x, int) { if (fkey(x) >= thr) mass += weight_of(__fsub_rn(mx, x)); });
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
  if (lane == 0) sm->wsum[warp] = mass;
  cluster_sync_all();
  if (tid < nwarps) sm->all[tid] = ld_cluster_u64(mapa_shared(&sm->wsum[tid % kCluWarps], tid / kCluWarps));
  __syncthreads();
  u64 Z = 0, base = 0;
  for (int q = 0; q < nwarps; ++q) {
    if (q == gw) base = Z;
    Z += sm->all[q];
  }
  if (Z == 0) {
    if (rank == 0 && tid == 0) out[rowi] = a.i;
  } else {
    const u64 target = portion(uniform01(seed, step, 0xffffffffull), Z);
    if (base < target && base + mass >= target) {
      for (int i0 = beg; i0 < end && base < target; i0 += 128) {
        float xv[4];
        load4(row, i0 + 4 * lane, end, vec, xv);
        u64 w[4], mine = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = __fadd_rn(__fmul_rn(xv[e], invT), 0.f);
          w[e] = (i0 + 4 * lane + e < end && fkey(x) >= thr) ? weight_of(__fsub_rn(mx, x)) : 0;
          mine += w[e];
        }
        u64 incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const u64 t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        u64 cum = base + incl - mine;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (w[e] > 0 && cum < target && cum + w[e] >= target) out[rowi] = i0 + 4 * lane + e;
          cum += w[e];
        }
        base += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
  }
  cluster_sync_all();              // nobody leaves while a peer may still read its sums
}

// One thread per (row, distinct history token). counts > 0 are output-token counts for
// frequency/presence; repetition applies to every listed token.
__global__ void penalties_kernel(float* __restrict__ logits, int rows, int vocab, int ld,
                                 const int32_t* __restrict__ tok, const int32_t* __restrict__ cnt,
                                 const int32_t* __restrict__ offsets, const float* __restrict__ freq,
                                 const float* __restrict__ pres, const float* __restrict__ rep) {
  const int row = blockIdx.y;
  const int beg = offsets[row], end = offsets[row + 1];
  for (int j = beg + blockIdx.x * blockDim.x + threadIdx.x; j < end; j += gridDim.x * blockDim.x) {
    const int t = tok[j];
    if (t < 0 || t >= vocab) continue;
    float x = logits[static_cast<size_t>(row) * ld + t];
    const float r = rep ? rep[row] : 1.f;
    if (r != 1.f) x = x > 0.f ? x / r : x * r;
    const int c = cnt[j];
    if (c > 0) x -= (freq ? freq[row] : 0.f) * c + (pres ? pres[row] : 0.f);
    logits[static_cast<size_t>(row) * ld + t] = x;
  }
}

}  // namespace mb

using namespace mb;

static bool g_sample_cluster = true;

extern "C" int mb_argmax(const float* logits, int64_t* out, int rows, int vocab, int ld,
                         cudaStream_t stream) {
  if (rows <= 0) return MB_OK;
  argmax_kernel<<<rows, kSampThreads, 0, stream>>>(logits, out, vocab, ld);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_sample_topk_topp(const float* logits, int64_t* out, int rows, int vocab, int ld,
                                   const float* temperature, const int32_t* top_k,
                                   const float* top_p, const float* min_p, const uint64_t* seeds,
                                   uint64_t step, cudaStream_t stream) {
  if (rows <= 0) return MB_OK;
  // Without any filter a row is one pass, and a batch that fills the SMs is faster with a large CTA a row: 128256 logits, 128 rows greedy 10
  // us, 18 on clusters, sampled 29 and 40; 64 rows 9 and 11, 29 and 23; 1 row 9 and 9, 29 and 10.
  const bool one_pass = top_k == nullptr && top_p == nullptr && min_p == nullptr && rows >= 128;
  if (g_sample_cluster && !one_pass && rows <= 65535 && vocab <= kClu * kMaxShare) {
    static PerDeviceOnce once;
    if (once.needed()) {
      if (cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(sizeof(ClusterSmem))) != cudaSuccess)
        return MB_ERR_LAUNCH;
      once.done();
    }
    // as many CTAs per row as still lets the whole batch run at once (two CTAs of this size per SM)
    static int sms = 0;
    if (sms == 0) {
      int dev = 0;
      cudaGetDevice(&dev);
      if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    int c = kClu;
    while (c > 1 && rows * c > 2 * sms && vocab <= (kMaxShare / 2) * c) c >>= 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c, rows);
    cfg.blockDim = dim3(kCluThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    if (cudaLaunchKernelEx(&cfg, sample_cluster_kernel, logits, out, vocab, ld, temperature, top_k, top_p, min_p,
                           seeds, step) == cudaSuccess)
      return MB_OK;
    // a device (or partition) that cannot place such clusters: every row goes to the one-CTA kernel from now on
    cudaGetLastError();
    g_sample_cluster = false;
  }
  return launch_k(sample_kernel, dim3(rows), dim3(kSampThreads), 0, stream, logits, out, vocab, ld, temperature,
                  top_k, top_p, min_p, seeds, step) == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// 0: every row is sampled by the one-CTA kernel (the cluster kernel is not launched)
extern "C" void mb_set_sample_cluster(int on) { g_sample_cluster = on != 0; }

// logits[r, v] = -inf where bit (v % 32) of bitmask[r, v / 32] is clear (grammar-constrained decoding)
__global__ void token_bitmask_kernel(float* __restrict__ logits, const int32_t* __restrict__ bitmask, int vocab,
                                     int ld, int words) {
  const int r = blockIdx.y;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < vocab; v += gridDim.x * blockDim.x)
    if (!((static_cast<uint32_t>(bitmask[static_cast<size_t>(r) * words + (v >> 5)]) >> (v & 31)) & 1u))
      logits[static_cast<size_t>(r) * ld + v] = -INFINITY;
}

extern "C" int mb_apply_token_bitmask(float* logits, const int32_t* bitmask, int rows, int vocab, int ld,
                                      cudaStream_t stream) {
  if (rows <= 0) return MB_OK;
  token_bitmask_kernel<<<dim3(16, rows), 256, 0, stream>>>(logits, bitmask, vocab, ld, (vocab + 31) / 32);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_apply_penalties(float* logits, int rows, int vocab, int ld, const int32_t* tok,
                                  const int32_t* cnt, const int32_t* offsets, const float* freq,
                                  const float* pres, const float* rep, cudaStream_t stream) {
  if (rows <= 0) return MB_OK;
  penalties_kernel<<<dim3(8, rows), 256, 0, stream>>>(logits, rows, vocab, ld, tok, cnt, offsets,
                                                      freq, pres, rep);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}
