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
// first). Greedy and plain-temperature rows are one pass. Rows with a filter take the maximum, then a histogram of
// mx - x / T in shared memory (bins of 1/32, counts and, for a nucleus over the whole row, softmax mass; bins that
// narrow spread the bulk of the row over hundreds of counters, so the atomics hardly meet). If the bins that provably
// hold the kept set have at most kList elements, those go to the first CTA, which ranks them by counting and reads both
// cut-offs off the sorted values. Otherwise the cut-off is found exactly by refining the bin it lies in, 2048 buckets
// of keys at a time (a few more passes), and the draw is a prefix sum over the warps' shares.
// Masses are integers, so sums do not depend on their order: 42 fractional bits where few weights meet in registers, and
// per bin the weights relative to the bin's upper edge as 26-bit numbers in two halves, because 32-bit atomics on shared
// memory are native and 64-bit ones are not (with those 64 nucleus rows took 122 us, with these 101).
// (One or four rows with a nucleus over the whole row and nothing else, of a spread of 3.75: 45 us when unit bins were counted in registers,
// 49 so; counts alone here and masses only where a long nucleus is cut: 55, and 78 for the mixed 64 rows below.)
// 64 rows of 128256 logits, a quarter of the rows with a nucleus of thousands of tokens: 364 us when such rows (and
// confident ones, whose k-th token lies far below the first) were left to sample_kernel, which walks a row with one
// CTA, 58 to 66 us so (127 us before where all kept sets were short); one row 28 us, 64 greedy rows 11 us.
constexpr int kClu = 8;          // largest cluster; the launcher picks 8, 4, 2 or 1 CTAs per row from the batch size
constexpr int kCluThreads = 512, kCluWarps = kCluThreads / 32;
constexpr int kBins = 2048, kOwn = kBins / kCluThreads;
static_assert(kOwn == 4, "a thread reads its bins as one vector");
constexpr int kList = kCluThreads;
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
__device__ __forceinline__ int bin_of(float below) {       // NaN goes to the last bin
  const float b = below * kBinsPerUnit;
  return b < static_cast<float>(kBins - 1) ? static_cast<int>(b) : kBins - 1;
}
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
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
    for (int i0 = beg; i0 < end; i0 += 512) {
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

  // 1. maximum of x / T (greedy: of x; no filter: of x / T + Gumbel noise, which is the draw)
  ArgMax a{-FLT_MAX, 0x7fffffff};
  if (plain) {
    visit([&](float x, int i) { a = amax2(a, ArgMax{x - __logf(-__logf(uniform01(seed, step, i))), i}); });
  } else {
    visit([&](float x, int i) { a = amax2(a, ArgMax{x, i}); });
  }
  a = block_argmax(a, sh_am);
  if (tid == 0) sm->cmax = a;
  cluster_sync_all();
  {
    ArgMax g{-FLT_MAX, 0x7fffffff};
    for (uint32_t r = 0; r < nclu; ++r) {
      ArgMax b;
      b.v = __uint_as_float(ld_cluster_u32(mapa_shared(&sm->cmax.v, r)));
      b.i = static_cast<int>(ld_cluster_u32(mapa_shared(&sm->cmax.i, r)));
      g = amax2(g, b);
    }
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

  // Histogram over the cluster: place(x, below, key) gives an element's bin or -1. This thread's kOwn bins come back as
  // counts (want & 1) and masses (want & 2).
  // `all_in`: the unit bin that holds every element placed, or -1 when the bins are the unit bins themselves.
  auto histogram = [&](int want, int all_in, auto&& place, u64 (&c)[kOwn], u64 (&m)[kOwn]) {
    cluster_sync_all();            // peers are done reading the bins of the pass before
    for (int i = tid; i < kBins; i += kCluThreads) { sm->cnt[i] = 0; sm->hi[i] = 0; sm->lo[i] = 0; }
    __syncthreads();
    visit([&](float x, int) {
      const float below = __fsub_rn(mx, x);
      const int b = place(below, fkey(x));
      if (b < 0) return;
      if (want & 1) atomicAdd(&sm->cnt[b], 1u);
      if (want & 2) {
        const uint32_t q = __float2uint_rn(__expf((all_in < 0 ? b : all_in) / kBinsPerUnit - below) * 67108864.f);
        atomicAdd(&sm->hi[b], q >> 13);
        atomicAdd(&sm->lo[b], q & 0x1fffu);
      }
    });
    cluster_sync_all();
#pragma unroll
    for (int j = 0; j < kOwn; ++j) c[j] = m[j] = 0;
    for (uint32_t r = 0; r < nclu; ++r) {
      if (want & 1) {
        const uint4 v = ld_cluster_v4(mapa_shared(&sm->cnt[tid * kOwn], r));
        c[0] += v.x; c[1] += v.y; c[2] += v.z; c[3] += v.w;
      }
      if (want & 2) {
        const uint4 h = ld_cluster_v4(mapa_shared(&sm->hi[tid * kOwn], r)), l = ld_cluster_v4(mapa_shared(&sm->lo[tid * kOwn], r));
        m[0] += (static_cast<u64>(h.x) << 13) + l.x; m[1] += (static_cast<u64>(h.y) << 13) + l.y;
        m[2] += (static_cast<u64>(h.z) << 13) + l.z; m[3] += (static_cast<u64>(h.w) << 13) + l.w;
      }
    }
    if (want & 2) {                // from 26 bits under the bin's edge to 42 under the maximum
#pragma unroll
      for (int j = 0; j < kOwn; ++j)
        if (m[j]) m[j] = static_cast<u64>(static_cast<double>(m[j]) * (65536.0 * exp(-(all_in < 0 ? tid * kOwn + j : all_in) / static_cast<double>(kBinsPerUnit))));
    }
  };
  // the first bin where the running sum of v reaches `target` (-1: none) and the sum before it
  auto cross = [&](const u64 (&v)[kOwn], u64 target, int& bin, u64& above) {
    if (tid == 0) sm->bin = -1;
    u64 sum = 0, total;
#pragma unroll
    for (int j = 0; j < kOwn; ++j) sum += v[j];
    u64 run = block_before(sum, sm->red, total);
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      if (run < target && run + v[j] >= target) { sm->bin = tid * kOwn + j; sm->above = run; }
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

  // 2. bins under the maximum
  u64 c[kOwn], m[kOwn], z_all = 0;
  const bool nucleus = use_p && !use_k && !use_m;
  histogram(nucleus ? 3 : 1, -1, [](float below, uint32_t) { return bin_of(below); }, c, m);
  int last = -1, kbin = -1;
  u64 kabove = 0, pabove = 0, ptarget = 0;
  if (use_k) { cross(c, static_cast<u64>(k), kbin, kabove); last = kbin; }
  if (use_m) last = max(last, bin_of(-__logf(mp) + 0.01f));
  if (nucleus) {
    block_before(m[0] + m[1] + m[2] + m[3], sm->red, z_all);
    ptarget = portion(tp, z_all);
    cross(m, ptarget, last, pabove);
  }
  int n = 0x7fffffff;
  {
    u64 sum = c[0] + c[1] + c[2] + c[3], total, run = block_before(sum, sm->red, total);
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      run += c[j];
      if (tid * kOwn + j == last) sm->n = run > 0x7fffffffu ? 0x7fffffff : static_cast<int>(run);
    }
    __syncthreads();
    if (last >= 0) n = sm->n;
  }

  if (n <= kList) {
    // 3a. candidates into the first CTA's list, in any order within a CTA's part of it. The positions come from a local
    // counter: one shared by the cluster is a queue of remote atomics (512 of them took 25 us).
    u64 part = 0, here;
#pragma unroll
    for (int j = 0; j < kOwn; ++j)
      if (tid * kOwn + j <= last) part += sm->cnt[tid * kOwn + j];
    block_before(part, sm->red, here);
    if (tid == 0) { sm->wsum[0] = here; sm->fill = 0; }
    cluster_sync_all();
    uint32_t first = 0;
    for (uint32_t r = 0; r < rank; ++r) first += static_cast<uint32_t>(ld_cluster_u64(mapa_shared(&sm->wsum[0], r)));
    const uint32_t lx = mapa_shared(&sm->lx[0], 0), li = mapa_shared(&sm->li[0], 0);
    visit([&](float x, int i) {
      if (bin_of(__fsub_rn(mx, x)) > last) return;
      const uint32_t pos = first + atomicAdd(&sm->fill, 1u);
      if (pos >= kList) return;    // cannot happen: the same elements were counted
      st_cluster_u32(lx + 4u * pos, __float_as_uint(x == x ? x : -INFINITY));      // ranks need an order: NaN is the lowest
      st_cluster_u32(li + 4u * pos, static_cast<uint32_t>(i));
    });
    cluster_sync_all();
    if (rank != 0) return;
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
      const u64 target = nucleus ? ptarget : portion(tp, sm->sp[kept - 1]);
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
    for (;;) {
      const uint32_t range = khi - klo;
      const int sh = range < static_cast<uint32_t>(kBins) ? 0 : 21 - __clz(range);
      histogram(want, bin, [&](float below, uint32_t key) {
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
      histogram(2, -1, [&](float below, uint32_t key) { return key >= least ? bin_of(below) : -1; }, c, m);
      block_before(m[0] + m[1] + m[2] + m[3], sm->red, z_all);
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
