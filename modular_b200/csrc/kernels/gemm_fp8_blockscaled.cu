// Block-scaled fp8 (e4m3) GEMM for sm_100a and the matching activation quantiser.
//
//   Y[M, N] = (Xq ⊙ sx)[M, K] · (Wq ⊙ sw)[N, K]^T
//
//   Wq  e4m3 [N, K], sw fp32 [ceil(N/128), ceil(K/128)]   one scale per 128x128 weight block
//   Xq  e4m3 [M, K], sx fp32 [ceil(K/128), M]             one scale per token per 128-wide K group
//                                                          (stored K-group-major so that a tile's
//                                                          tokens are contiguous)
//
// tcgen05.mma kind::f8f6f4 accumulates 128 K (four K=32 instructions) into one of four TMEM
// buffers; two epilogue warpgroups then "promote" that partial: read it back with tcgen05.ld,
// multiply by sw * sx and add it into fp32 register accumulators while the tensor core already
// works on the next K groups in the other buffers. The combined scales of a K group are fetched
// one group ahead and staged per warp in shared memory, so no global load sits between the
// accumulator barrier and the promotion. Token counts that give fewer CTAs than SMs split K
// over grid.z: every split writes fp32 partials that a small kernel sums (and adds the residual). For decode-sized token counts the promotion
// hides completely under the weight stream; for large token counts it bounds the kernel at
// roughly the bf16 rate, which is the price of arbitrary (non power-of-two) fp32 scales.
//
// Warp roles (320 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 promote token
// columns [0, BN/2), warps 6-9 columns [BN/2, BN). Weights sit on the UMMA M side (128 rows),
// tokens on the N side (BN = 32..128, multiple of 32).
//
// Reference counterparts: max/kernels/src/linalg/matmul/gpu/sm100/
// warp_specialized_blockwise_fp8.mojo:898 (promote_accumulators :520) and
// linalg/fp8_quantization.mojo:369 (per-token-group dynamic quantisation).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/api.h"
#include "../common/launch.h"
#include "../common/ptx.cuh"
#include "gemm_common.h"

namespace mb {
namespace f8 {

constexpr int kBM = 128;
constexpr int kBKBytes = 128;     // one swizzle row = 128 fp8 elements
constexpr int kThreads = 320;
constexpr int kATile = kBM * kBKBytes;
constexpr int kStgWarp = 16 * 32 * 2;

struct Params {
  __nv_bfloat16* Y;
  const __nv_bfloat16* R;
  const float* sw;
  const float* sx;
  int* err;
  int M, N, K, ldy, ldr, sw_ld, BN, stages;
  int splits, kb_per_split;
  float* partial;   // [splits, M, N] fp32 when splits > 1
  // grouped (mixture-of-experts) mode: blockIdx.x walks the token tiles of all experts in expert order
  // (expert e owns rows [offsets[e], offsets[e+1]) and ceil(rows / BN) tiles); weights / weight scales of
  // expert e start at row e * w_rows / e * sw_rows
  const int* expert_offsets;
  int w_rows, sw_rows, n_experts;
};

constexpr int kAccBufs = 4;

struct Tail {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[kAccBufs];
  uint64_t acc_empty[kAccBufs];
  uint32_t tmem_base;
  int abort_word;
  alignas(16) float scales[8][2][64];   // per promotion warp, double-buffered: sw * sx of its token columns
};

template <bool RESID>
__global__ void __launch_bounds__(kThreads, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int stage_bytes = kATile + p.BN * kBKBytes;
  uint8_t* stg_base = smem + p.stages * stage_bytes;
  Tail* tail = reinterpret_cast<Tail*>(stg_base + 8 * kStgWarp);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.y * kBM;
  int t0 = blockIdx.x * p.BN;
  int Mlim = p.M, w_row0 = 0, sw_row0 = 0, zsplit = blockIdx.z;
  if (p.expert_offsets != nullptr) {
    // every warp finds the expert of this CTA's tile: a prefix sum of the experts' tile counts, 32 experts
    // per round. The grid is sized for the worst case, so CTAs past the last tile leave here, before any
    // barrier or TMEM allocation.
    const int tile = blockIdx.x;
    int e = -1, row_end = 0, base = 0;
    for (int c = 0; c < p.n_experts; c += 32) {
      const int j = c + lane;
      const int b = j < p.n_experts ? p.expert_offsets[j] : 0;
      const int en = j < p.n_experts ? p.expert_offsets[j + 1] : 0;
      const int nt = (en - b + p.BN - 1) / p.BN;
      int incl = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const int before = base + incl - nt;
      const unsigned hit = __ballot_sync(0xffffffffu, tile >= before && tile < before + nt);
      if (hit != 0) {
        const int src = __ffs(hit) - 1;
        e = c + src;
        row_end = __shfl_sync(0xffffffffu, en, src);
        t0 = __shfl_sync(0xffffffffu, b, src) + (tile - __shfl_sync(0xffffffffu, before, src)) * p.BN;
        break;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (e < 0) return;
    Mlim = row_end;
    w_row0 = e * p.w_rows;
    sw_row0 = e * p.sw_rows;
    zsplit = 0;
  }
  const int kb_all = (p.K + 127) / 128;
  const int kb_begin = zsplit * p.kb_per_split;
  const int kb_end = kb_begin + p.kb_per_split < kb_all ? kb_begin + p.kb_per_split : kb_all;
  const int kb_total = kb_end - kb_begin;          // K groups of this split
  const uint32_t want_cols = p.BN * kAccBufs;
  const uint32_t tmem_cols = want_cols <= 128 ? 128 : (want_cols <= 256 ? 256 : 512);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int b = 0; b < kAccBufs; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], 8);
    }
    tail->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(&tail->tmem_base, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tail->tmem_base;
  volatile int* abort_word = &tail->abort_word;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;       // stage and phase are carried: no division on the pipeline's latency path
      uint32_t ph = 0;
      for (int kb = 0; kb < kb_total; ++kb, s = (s + 1 == p.stages ? 0 : s + 1), ph ^= (s == 0)) {
        if (!mbar_wait(&tail->empty[s], ph ^ 1, abort_word, p.err, 501)) break;
        uint8_t* sa = smem + s * stage_bytes;
        mbar_arrive_expect_tx(&tail->full[s], stage_bytes);
        tma_load_2d(sa, &tmW, &tail->full[s], (kb_begin + kb) * 128, w_row0 + n0);
        tma_load_2d(sa + kATile, &tmX, &tail->full[s], (kb_begin + kb) * 128, t0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc(kBM, p.BN, 0, 0);  // e4m3 x e4m3 -> fp32
      int s = 0;
      uint32_t ph = 0;
      for (int kb = 0; kb < kb_total; ++kb, s = (s + 1 == p.stages ? 0 : s + 1), ph ^= (s == 0)) {
        const int buf = kb % kAccBufs;
        const uint32_t bph = (kb / kAccBufs) & 1;
        if (!mbar_wait(&tail->acc_empty[buf], bph ^ 1, abort_word, p.err, 502)) break;
        if (!mbar_wait(&tail->full[s], ph, abort_word, p.err, 503)) break;
        tc_fence_after();
        uint8_t* sa = smem + s * stage_bytes;
        const uint64_t da = umma_desc_sw128(sa);
        const uint64_t db = umma_desc_sw128(sa + kATile);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t koff = static_cast<uint64_t>(k * 32 >> 4);  // 32 bytes per K=32 step
          umma_fp8(tmem_base + buf * p.BN, da + koff, db + koff, idesc, k > 0 ? 1u : 0u);
        }
        tc_commit(&tail->empty[s]);
        tc_commit(&tail->acc_full[buf]);
      }
    }
  } else {
    // ---------------------------------------------------------------- promotion + epilogue
    const int ew = warp - 2;            // 0..7
    const int quad = warp & 3;          // TMEM lane quadrant
    const int half = ew >> 2;           // which half of the token columns
    const int cols = p.BN >> 1;         // columns handled by this warpgroup (multiple of 16)
    const int c_base = half * cols;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    const float* sw_row = p.sw + static_cast<size_t>(sw_row0 + blockIdx.y) * p.sw_ld + kb_begin;
    const float* sx_base = p.sx + static_cast<size_t>(kb_begin) * p.M + t0 + c_base;
    float* sc = &tail->scales[ew][0][0];
    // lane l owns the scales of token columns l and l + 32 of this warpgroup's half
    const bool in0 = lane < cols && t0 + c_base + lane < Mlim;
    const bool in1 = lane + 32 < cols && t0 + c_base + lane + 32 < Mlim;
    float s0 = 0.f, s1 = 0.f;
    if (kb_total > 0) {
      const float w = sw_row[0];
      s0 = in0 ? sx_base[lane] * w : 0.f;
      s1 = in1 ? sx_base[lane + 32] * w : 0.f;
    }
    sc[lane] = s0;
    sc[lane + 32] = s1;
    __syncwarp();
    bool ok = true;
    for (int kb = 0; kb < kb_total && ok; ++kb) {
      const int buf = kb % kAccBufs;
      const uint32_t bph = (kb / kAccBufs) & 1;
      // next group's scales: in flight while this group's accumulator is awaited and promoted
      if (kb + 1 < kb_total) {
        const float w = sw_row[kb + 1];
        const float* sx_row = sx_base + static_cast<size_t>(kb + 1) * p.M;
        s0 = in0 ? sx_row[lane] * w : 0.f;
        s1 = in1 ? sx_row[lane + 32] * w : 0.f;
      }
      ok = mbar_wait(&tail->acc_full[buf], bph, abort_word, p.err, 504);
      if (!ok) break;
      tc_fence_after();
      const float* scur = sc + (kb & 1) * 64;
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        if (c < cols) {
          uint32_t v[16];
          tmem_ld_32x16(lane_addr + buf * p.BN + c_base + c, v);
          float4 sv[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) sv[q] = *reinterpret_cast<const float4*>(scur + c + q * 4);
          tc_wait_ld();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[c + q * 4 + 0] = fmaf(__uint_as_float(v[q * 4 + 0]), sv[q].x, acc[c + q * 4 + 0]);
            acc[c + q * 4 + 1] = fmaf(__uint_as_float(v[q * 4 + 1]), sv[q].y, acc[c + q * 4 + 1]);
            acc[c + q * 4 + 2] = fmaf(__uint_as_float(v[q * 4 + 2]), sv[q].z, acc[c + q * 4 + 2]);
            acc[c + q * 4 + 3] = fmaf(__uint_as_float(v[q * 4 + 3]), sv[q].w, acc[c + q * 4 + 3]);
          }
        }
      }
      tc_fence_before();
      float* snext = sc + ((kb + 1) & 1) * 64;
      snext[lane] = s0;
      snext[lane + 32] = s1;
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->acc_empty[buf]);
    }
    if (ok && p.splits > 1) {
      // fp32 partials of this split: lane = weight row, so each token's 32 floats are contiguous
      const int n = n0 + quad * 32 + lane;
      float* dst = p.partial + static_cast<size_t>(zsplit) * p.M * p.N;
#pragma unroll
      for (int c = 0; c < 64; ++c) {
        const int t = t0 + c_base + c;
        if (c < cols && t < Mlim && n < p.N) dst[static_cast<size_t>(t) * p.N + n] = acc[c];
      }
      ok = false;   // nothing left for the bf16 epilogue
    }
    if (ok) {
      __nv_bfloat16* stg = reinterpret_cast<__nv_bfloat16*>(stg_base + ew * kStgWarp);
      const int n_base = n0 + quad * 32;
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        if (c < cols && t0 + c_base + c < Mlim) {
#pragma unroll
          for (int j = 0; j < 16; ++j) stg[j * 32 + lane] = __float2bfloat16(acc[c + j]);
          __syncwarp();
#pragma unroll
          for (int pass = 0; pass < 2; ++pass) {
            const int j = pass * 8 + (lane >> 2);
            const int seg = lane & 3;
            const int t = t0 + c_base + c + j;
            const int n = n_base + seg * 8;
            if (t < Mlim && n < p.N) {
              uint4 val = *reinterpret_cast<const uint4*>(stg + j * 32 + seg * 8);
              if (RESID) {
                const uint4 rv = *reinterpret_cast<const uint4*>(p.R + static_cast<size_t>(t) * p.ldr + n);
                __nv_bfloat162* a = reinterpret_cast<__nv_bfloat162*>(&val);
                const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const float2 fa = __bfloat1622float2(a[q]);
                  const float2 fb = __bfloat1622float2(b[q]);
                  a[q] = __floats2bfloat162_rn(fa.x + fb.x, fa.y + fb.y);
                }
              }
              *reinterpret_cast<uint4*>(p.Y + static_cast<size_t>(t) * p.ldy + n) = val;
            }
          }
          __syncwarp();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}

// ---------------------------------------------------------------- tokens on the M side
// The same product for larger token counts, operands the other way round: 128 token rows per CTA on the MMA's M side, 256
// weight rows (two scale blocks) on its N side, so a promotion thread owns one token and 128 features and one K group
// has one factor per thread, in a register. With weights on M every column has a factor of its own, and reading those
// from shared memory (512 wavefronts a K group, beside 512 for the operands) is what bounds that form: L1 pipe 80 % busy,
// tensor pipe 20 %. Accumulators are 128 fp32 registers per thread, added two at a time; the K group after next is
// multiplied into the other of two 256-column TMEM buffers meanwhile. The sums run over K in the same order as above.
// CTAs are persistent, so one tile's stores run under the next one's first loads.
//   PAIR    dense: two CTAs share the tile (256 tokens x 256 weight rows, each loads half of either operand), which halves
//           the bytes per operation that come from L2: 2050 x 57344 x 8192 in 1080 us (2094 with weights on M). A K group
//           takes a promotion warp about 1100 cycles at two of them a scheduler (wait, four TMEM reads of 150 cycles, 64 packed FMAs,
//           release), while its MMAs take 512: that chain is the bound, not a unit.
//   !PAIR   experts: the tiles of one expert's tokens after another; weights are read from memory once and are the bound:
//           16800 rows, 256 experts of 4096 x 7168: 1400 us (2998 with weights on M).
constexpr int kRowStages = 6, kRowTileN = 256, kMaxRowTiles = 1024;
// warp 0 TMA, warp 1 MMA, warp 2 the experts' tiles, warps 4-11 promotion (setmaxnreg works on groups of four warps)
constexpr int kRowThreads = 384;
constexpr int kAhead = 4;             // K groups whose factors are on their way
constexpr int kRowsFrom = 128, kRowsAlways = 1024;

struct RowTail {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_word;
  int n_tiles;                        // grouped: token tiles
  int2 tile[kMaxRowTiles];            // grouped: expert, first row
  float factor[8][kAhead][64];        // grouped: per promotion warp and K group: sx of its 32 rows, then sw 32 times
};

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ uint64_t fma2(uint32_t lo, uint32_t hi, uint64_t s, uint64_t acc) {
  uint64_t v, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(v), "l"(s), "l"(acc));
  return r;
}

template <bool PAIR, bool RESID>
__global__ void __launch_bounds__(kRowThreads, 1)
gemm_fp8_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int kB = PAIR ? kATile : 2 * kATile, kStage = kATile + kB;
  RowTail* tail = reinterpret_cast<RowTail*>(smem + p.stages * kStage);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const int worker = PAIR ? blockIdx.x >> 1 : blockIdx.x, workers = PAIR ? gridDim.x >> 1 : gridDim.x;
  const int kb_total = (p.K + 127) / 128;
  const int n_blocks = (p.N + kRowTileN - 1) / kRowTileN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], PAIR ? 16 : 8);
    }
    tail->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(&tail->tmem_base, 512); tmem_relinquish_pair(); }
    else { tmem_alloc(&tail->tmem_base, 512); tmem_relinquish(); }
  }
  if (!PAIR && warp == 2) {
    // the token tiles of all experts, in expert order
    int base = 0;
    for (int c = 0; c < p.n_experts; c += 32) {
      const int j = c + lane;
      const int b = j < p.n_experts ? p.expert_offsets[j] : 0;
      const int en = j < p.n_experts ? p.expert_offsets[j + 1] : 0;
      const int nt = (en - b + kBM - 1) / kBM;
      int incl = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      for (int i = 0; i < nt && base + incl - nt + i < kMaxRowTiles; ++i) tail->tile[base + incl - nt + i] = make_int2(j, b + i * kBM);
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) tail->n_tiles = min(base, kMaxRowTiles);
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();         // the peer's barriers exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = tail->tmem_base;
  volatile int* abort_word = &tail->abort_word;
  const int m_tiles = PAIR ? (p.M + 2 * kBM - 1) / (2 * kBM) : tail->n_tiles;
  const int total = m_tiles * n_blocks;
  // tile t: first token row of this CTA, end of its rows, first weight row, first rows of the expert
  auto place = [&](int t, int& row0, int& row_end, int& n0, int& expert) {
    if (PAIR) {
      row0 = (t % m_tiles) * (2 * kBM) + static_cast<int>(rank) * kBM;
      row_end = p.M;
      n0 = (t / m_tiles) * kRowTileN;
      expert = 0;
    } else {
      const int2 at = tail->tile[t / n_blocks];
      row0 = at.y;
      row_end = p.expert_offsets[at.x + 1];
      n0 = (t % n_blocks) * kRowTileN;
      expert = at.x;
    }
  };

  // 384 x 168 registers at launch: four warps give theirs up, eight take them (128 x 56 + 256 x 224 is the same sum)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0 && lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = worker; t < total && ok; t += workers) {
        int row0, row_end, n0, expert;
        place(t, row0, row_end, n0, expert);
        const int w0 = expert * p.w_rows + n0;
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait(&tail->empty[s], ph ^ 1, abort_word, p.err, 511)) { ok = false; break; }
          uint8_t* sa = smem + s * kStage;
          if (PAIR) {
            if (rank == 0) mbar_arrive_expect_tx(&tail->full[s], 2 * kStage);
            const uint32_t full_leader = mapa_shared(&tail->full[s], 0);
            tma_load_2d_pair(sa, &tmX, full_leader, kb * 128, row0);
            tma_load_2d_pair(sa + kATile, &tmW, full_leader, kb * 128, w0 + static_cast<int>(rank) * kBM);
          } else {
            mbar_arrive_expect_tx(&tail->full[s], kStage);
            tma_load_2d(sa, &tmX, &tail->full[s], kb * 128, row0);
            tma_load_2d(sa + kATile, &tmW, &tail->full[s], kb * 128, w0);
            tma_load_2d(sa + 2 * kATile, &tmW, &tail->full[s], kb * 128, w0 + kBM);
          }
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1 && lane == 0 && rank == 0) {
      const uint32_t idesc = umma_idesc(PAIR ? 2 * kBM : kBM, kRowTileN, 0, 0);
      const uint32_t empty0 = mapa_shared(&tail->empty[0], 0), empty1 = PAIR ? mapa_shared(&tail->empty[0], 1) : 0u;
      const uint32_t afull0 = mapa_shared(&tail->acc_full[0], 0), afull1 = PAIR ? mapa_shared(&tail->acc_full[0], 1) : 0u;
      int s = 0;
      uint32_t ph = 0, g = 0;            // g: K groups so far, over all tiles
      bool ok = true;
      for (int t = worker; t < total && ok; t += workers) {
        for (int kb = 0; kb < kb_total; ++kb, ++g) {
          const uint32_t buf = g & 1;
          ok = mbar_wait(&tail->acc_empty[buf], ((g >> 1) & 1) ^ 1, abort_word, p.err, 512) &&
               mbar_wait(&tail->full[s], ph, abort_word, p.err, 513);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = umma_desc_sw128(smem + s * kStage), db = umma_desc_sw128(smem + s * kStage + kATile);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t koff = static_cast<uint64_t>(k * 32 >> 4);
            if (PAIR) umma_fp8_pair(tmem_base + buf * kRowTileN, da + koff, db + koff, idesc, k > 0 ? 1u : 0u);
            else umma_fp8(tmem_base + buf * kRowTileN, da + koff, db + koff, idesc, k > 0 ? 1u : 0u);
          }
          if (PAIR) {
            tc_commit_pair(empty0 + 8u * s);
            tc_commit_pair(empty1 + 8u * s);
            tc_commit_pair(afull0 + 8u * buf);
            tc_commit_pair(afull1 + 8u * buf);
          } else {
            tc_commit(&tail->empty[s]);
            tc_commit(&tail->acc_full[buf]);
          }
          if (++s == p.stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    const int quad = warp & 3, half = (warp - 4) >> 2;
    const uint32_t addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + half * 128;
    const uint32_t aempty = mapa_shared(&tail->acc_empty[0], 0);
    uint32_t g = 0;
    bool ok = true;
    for (int t = worker; t < total && ok; t += workers) {
      int row0, row_end, n0, expert;
      place(t, row0, row_end, n0, expert);
      const int row = row0 + quad * 32 + lane, col0 = n0 + half * 128;
      const bool live = row < row_end;
      const float* sx = p.sx + (live ? row : 0);
      const float* sw = p.sw + static_cast<size_t>(expert * p.sw_rows + (col0 < p.N ? col0 : 0) / 128) * p.sw_ld;
      uint64_t acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0;
      // A lane reads its own factors kAhead K groups ahead: into registers (through shared memory the two copies and their wait were 150
      // of a group's thousand cycles; 2050 x 57344 x 8192 1147 -> 1082 us), experts through shared memory (one commit per K group, empty
      // beyond the last one), because they have no registers left: with the factors in them the kernel spills and takes 2 % longer.
      float px[kAhead], pw[kAhead];
      float* mine = &tail->factor[warp - 4][0][lane];
      auto fetch = [&](int kb) {
        if (kb < kb_total) {
          cp_async4(mine + (kb % kAhead) * 64, sx + static_cast<size_t>(kb) * p.M);
          cp_async4(mine + (kb % kAhead) * 64 + 32, sw + kb);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if constexpr (PAIR) {
          px[j] = live && j < kb_total ? sx[static_cast<size_t>(j) * p.M] : 0.f;
          pw[j] = j < kb_total ? sw[j] : 0.f;
        } else {
          fetch(j);
        }
      }
      for (int kb = 0; kb < kb_total; ++kb) {
        float f;
        if constexpr (PAIR) {
          f = px[0] * pw[0];
#pragma unroll
          for (int j = 0; j < kAhead - 1; ++j) { px[j] = px[j + 1]; pw[j] = pw[j + 1]; }
          const int next = kb + kAhead;
          if (next < kb_total) {
            px[kAhead - 1] = live ? sx[static_cast<size_t>(next) * p.M] : 0.f;
            pw[kAhead - 1] = sw[next];
          }
        } else {
          asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
          const float* at = mine + (kb % kAhead) * 64;
          f = live ? at[0] * at[32] : 0.f;
          fetch(kb + kAhead);
        }
        uint64_t f2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(f2) : "r"(__float_as_uint(f)));
        const uint32_t buf = g & 1;
        // One lane asks: 32 of them are served one after the other. The others learn of it by a shuffle, which orders no memory: the
        // barrier of the warp makes what lane 0 saw complete hold for them as well.
        ok = (PAIR && lane != 0) || mbar_wait(&tail->acc_full[buf], (g >> 1) & 1, abort_word, p.err, 514);
        if (PAIR) {
          __syncwarp();
          ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        if (!ok) break;
        ++g;
        tc_fence_after();
        // a load of the next columns is in flight while these are added
        constexpr int W = 32;
        uint32_t v[2][W];
        tmem_ld_32x32(addr + buf * kRowTileN, v[0]);
#pragma unroll
        for (int c = 0; c < 128 / W; ++c) {
          tc_wait_ld();
          if (c < 128 / W - 1) {
            tmem_ld_32x32(addr + buf * kRowTileN + (c + 1) * W, v[(c + 1) & 1]);
          } else {                     // everything is read: the buffer may be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(aempty + 8u * buf);
          }
#pragma unroll
          for (int i = 0; i < W / 2; ++i) acc[c * (W / 2) + i] = fma2(v[c & 1][2 * i], v[c & 1][2 * i + 1], f2, acc[c * (W / 2) + i]);
        }
      }
      if (!PAIR) asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (!ok) break;
      // 64 features (one 128-byte line) at a time; a residual line is read before the line before it is written
      __nv_bfloat16* y = p.Y + static_cast<size_t>(live ? row : 0) * p.ldy + col0;
      const __nv_bfloat16* r = RESID ? p.R + static_cast<size_t>(live ? row : 0) * p.ldr + col0 : nullptr;
      uint4 res[2][8];
      auto read_line = [&](int l, uint4 (&to)[8]) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          to[q] = live && col0 + l * 64 + q * 8 + 8 <= p.N ? *reinterpret_cast<const uint4*>(r + l * 64 + q * 8) : make_uint4(0, 0, 0, 0);
      };
      if (RESID) read_line(0, res[0]);
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        if (RESID && l == 0) read_line(1, res[1]);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint4 o;
          uint32_t* w = &o.x;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t a = acc[l * 32 + q * 4 + i];
            __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(static_cast<uint32_t>(a)), __uint_as_float(static_cast<uint32_t>(a >> 32)));
            if (RESID) {                 // the product is rounded before the residual is added, as with weights on M
              const float2 fa = __bfloat1622float2(h);
              const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&(&res[l][q].x)[i]));
              h = __floats2bfloat162_rn(fa.x + fb.x, fa.y + fb.y);
            }
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
          if (live && col0 + l * 64 + q * 8 + 8 <= p.N) *reinterpret_cast<uint4*>(y + l * 64 + q * 8) = o;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();         // neither CTA leaves while the other may still use its memory or barriers
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

template <bool PAIR, bool RESID>
static int launch_rows(const Params& q, int num_sms, int tiles, const CUtensorMap& tw, const CUtensorMap& tx, cudaStream_t stream) {
  Params p = q;
  p.stages = PAIR ? kRowStages : 4;
  const size_t smem = static_cast<size_t>(p.stages) * (PAIR ? 2 : 3) * kATile + sizeof(RowTail) + 1024;
  auto kern = gemm_fp8_rows_kernel<PAIR, RESID>;
  static PerDeviceOnce configured;
  if (configured.needed()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return MB_ERR_LAUNCH;
    configured.done();
  }
  cudaLaunchConfig_t cfg = {};
  const int workers = PAIR ? num_sms / 2 : num_sms;
  cfg.gridDim = dim3(static_cast<unsigned>((tiles < workers ? tiles : workers) * (PAIR ? 2 : 1)));
  cfg.blockDim = dim3(kRowThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2 : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, tw, tx, p) == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// Sum of the split-K partials [splits, M, N] (+ residual) -> bf16 Y; N % 4 == 0.
__global__ void fp8_splitk_reduce_kernel(const float* __restrict__ part, const __nv_bfloat16* __restrict__ R,
                                         __nv_bfloat16* __restrict__ Y, int M, int N, int splits) {
  const size_t idx = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
  const size_t total = static_cast<size_t>(M) * N;
  if (idx >= total) return;
  float4 a = *reinterpret_cast<const float4*>(part + idx);
  for (int s = 1; s < splits; ++s) {
    const float4 b = *reinterpret_cast<const float4*>(part + s * total + idx);
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
  }
  if (R != nullptr) {
    const uint2 rv = *reinterpret_cast<const uint2*>(R + idx);
    const __nv_bfloat162* rb = reinterpret_cast<const __nv_bfloat162*>(&rv);
    const float2 r0 = __bfloat1622float2(rb[0]), r1 = __bfloat1622float2(rb[1]);
    a.x += r0.x; a.y += r0.y; a.z += r1.x; a.w += r1.y;
  }
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
  uint2 out;
  out.x = *reinterpret_cast<const uint32_t*>(&lo);
  out.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(Y + idx) = out;
}

// Sixteen lanes per (token, 128-wide K group), eight values a lane: amax -> scale = amax / 448, q = x / scale. Bound by memory;
// with a whole warp and eight bytes a lane, 64-bit divisions for the place included, 2050 x 28672 took 74 us; 2050 x 8192 take 12.4 so.
__device__ __forceinline__ void unpack8(float (&v)[8], const uint4 raw) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
// this lane's eight values of a group as e4m3 (the scale is the same in all sixteen lanes)
__device__ __forceinline__ uint2 quant8(const float (&v)[8], float& scale) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  scale = fmaxf(amax, 1e-12f) / 448.0f;
  const float inv = 1.0f / scale;
  const __nv_fp8x4_e4m3 lo(make_float4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv)), hi(make_float4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv));
  return make_uint2(lo.__x, hi.__x);
}
// With `order`, row t is row order[t] / top_k of x (the tokens in expert order) and rows from *n_rows_dev on are left alone: 2100
// tokens of 7168 to 8 experts each in 61 us, 75 + 84 us when the bf16 rows are copied into expert order first.
// U groups of a row per half warp, their loads in flight together.
template <int U>
__global__ void __launch_bounds__(256) quant_fp8_group128_vec_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                                                     float* __restrict__ scales, int M, int K, int ldx, int k_major,
                                                                     const int32_t* __restrict__ order, const int32_t* __restrict__ n_rows_dev,
                                                                     int top_k) {
  const unsigned groups = (K + 127) / 128, per_row = (groups + U - 1) / U, unit = (blockIdx.x * 256u + threadIdx.x) >> 4, sub = threadIdx.x & 15;
  const unsigned t = unit / per_row, g0 = unit % per_row * U;
  const bool live = t < static_cast<unsigned>(n_rows_dev != nullptr ? min(M, *n_rows_dev) : M);
  const int k0 = g0 * 128 + sub * 8;
  uint4 raw[U];
#pragma unroll
  for (int i = 0; i < U; ++i) raw[i] = make_uint4(0, 0, 0, 0);
  if (live) {
    const __nv_bfloat16* row = x + static_cast<size_t>(order != nullptr ? order[t] / top_k : t) * ldx + k0;
#pragma unroll
    for (int i = 0; i < U; ++i)
      if (k0 + i * 128 < K) raw[i] = *reinterpret_cast<const uint4*>(row + i * 128);
  }
#pragma unroll
  for (int i = 0; i < U; ++i) {
    float v[8], scale;
    unpack8(v, raw[i]);
    const uint2 packed = quant8(v, scale);
    if (live && k0 + i * 128 < K) *reinterpret_cast<uint2*>(q + static_cast<size_t>(t) * K + k0 + i * 128) = packed;
    if (live && sub == 0 && g0 + i < groups) scales[k_major ? static_cast<size_t>(g0 + i) * M + t : static_cast<size_t>(t) * groups + g0 + i] = scale;
  }
}
// Rows that fill the chip several times over take four groups a half warp (16800 x 7168 into expert order: 61 us, 92 with one), fewer take one.
static int launch_quant_vec(const void* x, void* q, float* scales, int M, int K, int ldx, int k_major, const int32_t* order,
                            const int32_t* n_rows_dev, int top_k, cudaStream_t stream) {
  const long long groups = (K + 127) / 128;
  const bool many = M * groups >= 148LL * 16 * 16;
  const long long units = M * (many ? (groups + 3) / 4 : groups);
  auto kern = many ? quant_fp8_group128_vec_kernel<4> : quant_fp8_group128_vec_kernel<1>;
  kern<<<static_cast<unsigned>((units + 15) / 16), 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), scales, M, K,
                                                                     ldx, k_major, order, n_rows_dev, top_k);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// The same for rows without 16-byte alignment, one warp per group.
__global__ void quant_fp8_group128_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q,
                                          float* __restrict__ scales, int M, int K, int ldx,
                                          int k_major) {
  const int groups = (K + 127) / 128;
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= static_cast<long long>(M) * groups) return;
  const int t = static_cast<int>(wid / groups), g = static_cast<int>(wid % groups);
  const int k0 = g * 128 + lane * 4;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (k0 < K) {
    const uint2 raw = *reinterpret_cast<const uint2*>(x + static_cast<size_t>(t) * ldx + k0);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
    const float2 a = __bfloat1622float2(b[0]), c = __bfloat1622float2(b[1]);
    v[0] = a.x; v[1] = a.y; v[2] = c.x; v[3] = c.y;
  }
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = fmaxf(amax, 1e-12f) / 448.0f;
  const float inv = 1.0f / scale;
  if (k0 < K) {
    const __nv_fp8x4_e4m3 packed(make_float4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv));
    *reinterpret_cast<uint32_t*>(q + static_cast<size_t>(t) * K + k0) = packed.__x;
  }
  if (lane == 0) scales[k_major ? static_cast<size_t>(g) * M + t : static_cast<size_t>(t) * groups + g] = scale;
}

// SwiGLU and the 1x128 quantisation of its result in one pass: gu [M, 2I] bf16 (gate | up) -> q [M, I] e4m3
// and scales [I/128, ld_s] (group-major). The product is rounded to bf16 first, so the result equals the
// two-pass form bit for bit. Rows at or past *n_rows_dev (when given) are skipped: grouped GEMMs whose row
// count is only known on the device pay for the rows that exist. Sixteen lanes per (row, group), grid-stride.
// 2050 x 28672: 83 us (silu_mul and the quantiser apart: 69 + 74 us).
__global__ void __launch_bounds__(256) silu_mul_quant_fp8_kernel(const __nv_bfloat16* __restrict__ gu, uint8_t* __restrict__ q,
                                          float* __restrict__ scales, int M, int I, int ld_s,
                                          const int32_t* __restrict__ n_rows_dev) {
  const int rows = n_rows_dev != nullptr ? min(M, *n_rows_dev) : M;
  const unsigned groups = I >> 7, sub = threadIdx.x & 15;
  const long long total = static_cast<long long>(rows) * groups, stride = static_cast<long long>(gridDim.x) * 16;
  for (long long unit0 = static_cast<long long>(blockIdx.x) * 16 + (threadIdx.x >> 5) * 2; unit0 < total; unit0 += stride) {   // per warp
    const long long unit = unit0 + ((threadIdx.x >> 4) & 1);
    const bool live = unit < total;
    const unsigned t = static_cast<unsigned>(live ? unit : 0) / groups, g = static_cast<unsigned>(live ? unit : 0) % groups;
    const int k0 = g * 128 + sub * 8;
    const __nv_bfloat16* row = gu + static_cast<size_t>(t) * 2 * I + k0;
    float a[8], u[8];
    unpack8(a, *reinterpret_cast<const uint4*>(row));
    unpack8(u, *reinterpret_cast<const uint4*>(row + I));
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = __bfloat162float(__float2bfloat16_rn(a[j] / (1.f + __expf(-a[j])) * u[j]));
    float scale;
    const uint2 packed = quant8(a, scale);
    if (live) {
      *reinterpret_cast<uint2*>(q + static_cast<size_t>(t) * I + k0) = packed;
      if (sub == 0) scales[static_cast<size_t>(g) * ld_s + t] = scale;
    }
  }
}

// The inverse of the 1x128 quantisation: q [M, K] e4m3 with group-major scales [K/128, ld_s] -> bf16 [M, K].
// Rows at or past *n_rows_dev (when given) are skipped.
__global__ void dequant_fp8_group128_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scales,
                                            __nv_bfloat16* __restrict__ out, int M, int K, int ld_s,
                                            const int32_t* __restrict__ n_rows_dev) {
  const int rows = n_rows_dev != nullptr ? min(M, *n_rows_dev) : M;
  const int per_row = K >> 2;
  const long long total = static_cast<long long>(rows) * per_row;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int r = static_cast<int>(i / per_row), c = static_cast<int>(i % per_row) * 4;
    const float scale = scales[static_cast<size_t>(c >> 7) * ld_s + r];
    __nv_fp8x4_e4m3 v;
    v.__x = *reinterpret_cast<const uint32_t*>(q + static_cast<size_t>(r) * K + c);
    const float4 f = static_cast<float4>(v);
    const __nv_bfloat162 lo = __floats2bfloat162_rn(f.x * scale, f.y * scale);
    const __nv_bfloat162 hi = __floats2bfloat162_rn(f.z * scale, f.w * scale);
    uint2 o;
    o.x = *reinterpret_cast<const uint32_t*>(&lo);
    o.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(out + static_cast<size_t>(r) * K + c) = o;
  }
}

}  // namespace f8
}  // namespace mb

using namespace mb;

extern "C" int mb_dequant_fp8_group128(const void* q_fp8, const float* scales, void* out_bf16, int M, int K, int ld_s,
                                       const int32_t* n_rows_dev, cudaStream_t stream) {
  if (M <= 0) return MB_OK;
  if (K % 128 || ld_s < M) return MB_ERR_SHAPE;
  long long blocks = (static_cast<long long>(M) * (K / 4) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  f8::dequant_fp8_group128_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      static_cast<const uint8_t*>(q_fp8), scales, static_cast<__nv_bfloat16*>(out_bf16), M, K, ld_s, n_rows_dev);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_silu_mul_quant_fp8(const void* gate_up, void* q_fp8, float* scales, int M, int inter, int ld_s,
                                     const int32_t* n_rows_dev, cudaStream_t stream) {
  if (M <= 0) return MB_OK;
  if (inter % 128 || ld_s < M) return MB_ERR_SHAPE;
  const long long units = static_cast<long long>(M) * (inter / 128);
  if (units >= (1ll << 31)) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(gate_up) & 15) | (reinterpret_cast<uintptr_t>(q_fp8) & 7)) return MB_ERR_ALIGN;
  long long blocks = (units + 15) / 16;
  if (blocks > 148 * 32) blocks = 148 * 32;
  f8::silu_mul_quant_fp8_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(gate_up), static_cast<uint8_t*>(q_fp8), scales, M, inter, ld_s, n_rows_dev);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_quant_fp8_group128(const void* x_bf16, void* q_fp8, float* scales, int M, int K,
                                     int ldx, int scale_ld, int scales_k_major, cudaStream_t stream) {
  (void)scale_ld;
  if (M <= 0) return MB_OK;
  if (K % 4 || ldx % 4) return MB_ERR_SHAPE;
  const long long warps = static_cast<long long>(M) * ((K + 127) / 128);
  if (K % 8 == 0 && ldx % 8 == 0 && ((reinterpret_cast<uintptr_t>(x_bf16) & 15) | (reinterpret_cast<uintptr_t>(q_fp8) & 7)) == 0 &&
      warps < (1ll << 28)) {
    return f8::launch_quant_vec(x_bf16, q_fp8, scales, M, K, ldx, scales_k_major, nullptr, nullptr, 1, stream);
  }
  const int threads = 256;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  f8::quant_fp8_group128_kernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x_bf16), static_cast<uint8_t*>(q_fp8), scales, M, K, ldx,
      scales_k_major);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// src [tokens, K] bf16 rows -> q [max_rows, K] e4m3 and scales [ceil(K / 128), max_rows] of the rows order[r] / top_k
extern "C" int mb_moe_permute_quant_fp8(const void* src, const int32_t* order, const int32_t* n_rows_dev, void* q_fp8, float* scales,
                                        int max_rows, int K, int top_k, cudaStream_t stream) {
  if (max_rows <= 0) return MB_OK;
  const long long units = static_cast<long long>(max_rows) * ((K + 127) / 128);
  if (K <= 0 || K % 8 || top_k <= 0 || units >= (1ll << 28)) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(src) & 15) | (reinterpret_cast<uintptr_t>(q_fp8) & 7)) return MB_ERR_ALIGN;
  return f8::launch_quant_vec(src, q_fp8, scales, max_rows, K, K, 1, order, n_rows_dev, top_k, stream);
}

namespace mb {
namespace f8 {
// Number of K splits for a grid of `ctas` output tiles: the split count (<= 8, at least four K groups
// each) that fills whole waves of SMs best, with a small bias towards fewer splits.
static int fp8_pick_splits(int ctas, int kb_total, int num_sms) {
  if (ctas >= num_sms || num_sms <= 0) return 1;
  int best = 1;
  float best_score = -1.f;
  for (int s = 1; s <= 8 && kb_total / s >= 4; ++s) {
    const int total = ctas * s;
    const int waves = (total + num_sms - 1) / num_sms;
    const float score = static_cast<float>(total) / (waves * num_sms) - 0.02f * s;
    if (score > best_score) { best_score = score; best = s; }
  }
  return best;
}

// Token tile and K splits of the form with weights on M.
static void fp8_split_plan(int M, int N, int K, size_t workspace_bytes, int num_sms, int* bn, int* splits) {
  const int kb = K > 0 ? (K + 127) / 128 : 1;
  if (*bn <= 0) {
    const int mt = (M + 127) / 128;
    *bn = ((M + mt - 1) / mt + 31) / 32 * 32;
  }
  int s = *splits;
  if (s <= 0) s = fp8_pick_splits(((M + *bn - 1) / *bn) * ((N + kBM - 1) / kBM), kb, num_sms);
  if (s > kb) s = kb;
  if (N % 4 || static_cast<size_t>(s) * M * N * sizeof(float) > workspace_bytes) s = 1;
  const int per = (kb + s - 1) / s;
  *splits = (kb + per - 1) / per;
}
}  // namespace f8
}  // namespace mb

// Whether a dense product takes the form with tokens on M (1) or with weights on M (0, with its token tile and K splits): the one whose
// time is less. Tokens on M give a pair of SMs one 256 x 256 tile for the whole of K, so that a narrow output leaves SMs idle; the
// other form splits K until they are busy. In us, from 240 shapes (129 to 2048 tokens, 576 to 16384 features, K 2048 to 14336) on 148
// SMs:  tokens on M  10.5 + 0.55 a K group and round of tiles;  weights on M  4 + 1.5 a wave + 0.64 a K group and wave (0.42 with token
// tiles of 32), and with splits 3 + 1.7 for every million partial sums. 200 tokens, 1280 x 7168: 41 against 17 us; 512 tokens, 4096 x
// 14336: 72 against 75; 2048 tokens, 8192 x 14336: 279 against 490. Splits change the order of a sum, so they have to gain 2.8 us, and
// from 1024 tokens on no sum depends on them: only outputs of fewer than some 700 features would still gain (1024 tokens, 576 x 7168:
// 42 against 27 us; 1536 tokens 42 against 38). No shape below 1024 tokens takes more than 1.14 of its faster form's time.
// Up to 128 tokens weights on M stream faster at any width (one token, 57344 x 8192: 113 against 178 us).
extern "C" int mb_gemm_fp8_plan(int M, int N, int K, size_t workspace_bytes, int num_sms, int* bn, int* splits) {
  *bn = *splits = 0;
  mb::f8::fp8_split_plan(M, N, K, workspace_bytes, num_sms, bn, splits);
  using namespace mb::f8;
  if (M <= kRowsFrom || N < kRowTileN || num_sms < 2) return 0;
  if (M >= kRowsAlways) return 1;
  const int groups = (K + 127) / 128, per = (groups + *splits - 1) / *splits;
  const long long pairs = num_sms / 2, tiles = static_cast<long long>((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kRowTileN - 1) / kRowTileN);
  const long long ctas = static_cast<long long>((M + *bn - 1) / *bn) * ((N + kBM - 1) / kBM) * *splits;
  const double rounds = static_cast<double>((tiles + pairs - 1) / pairs), waves = static_cast<double>((ctas + num_sms - 1) / num_sms);
  const double rows_us = 10.5 + 0.55 * rounds * groups;
  double split_us = 4. + waves * (1.5 + (0.34 + 0.3 * *bn / 128.) * per);
  if (*splits > 1) split_us += 3. + 1.7e-6 * *splits * M * N;
  return rows_us <= split_us + 2.8;
}

// flags: bit1 residual add. Xs is K-group-major [ceil(K/128), M]; Ws is [ceil(N/128), ceil(K/128)].
// bn, splits <= 0: chosen here (no splits without a workspace of splits*M*N floats) from the sizes and num_sms. A caller that names
// any of bn, stages or splits gets the form with weights on M, which has them.
extern "C" int mb_gemm_fp8_blockscaled(const void* Xq, const float* Xs, const void* Wq, const float* Ws,
                                       void* Y, const void* R, int M, int N, int K, int flags, int bn,
                                       int stages, int splits, void* workspace, size_t workspace_bytes,
                                       int num_sms, int* err, cudaStream_t stream) {
  using namespace mb::f8;
  if (M <= 0 || N <= 0) return MB_OK;
  if (K % 16 || N % 8) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(Xq) | reinterpret_cast<uintptr_t>(Wq) | reinterpret_cast<uintptr_t>(Y) |
       reinterpret_cast<uintptr_t>(R)) & 15)
    return MB_ERR_ALIGN;
  if (workspace == nullptr) workspace_bytes = 0;
  bool rows_form = false;
  if (bn <= 0 && splits <= 0 && stages <= 0) rows_form = mb_gemm_fp8_plan(M, N, K, workspace_bytes, num_sms, &bn, &splits) != 0;
  else fp8_split_plan(M, N, K, workspace_bytes, num_sms, &bn, &splits);
  if (bn % 32 || bn < 32 || bn > 128) return MB_ERR_SHAPE;
  Params p = {};
  p.Y = static_cast<__nv_bfloat16*>(Y);
  p.R = static_cast<const __nv_bfloat16*>(R);
  p.sw = Ws; p.sx = Xs; p.err = err;
  p.M = M; p.N = N; p.K = K; p.ldy = N; p.ldr = N; p.sw_ld = (K + 127) / 128; p.BN = bn;
  if (rows_form) {
    CUtensorMap tw, tx;
    int rc = cached_tmap(&tw, Wq, N, K, K, kBM, 1);
    if (rc != MB_OK) return rc;
    rc = cached_tmap(&tx, Xq, M, K, K, kBM, 1);
    if (rc != MB_OK) return rc;
    const int tiles = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + kRowTileN - 1) / kRowTileN);
    return (flags & 2) ? launch_rows<true, true>(p, num_sms, tiles, tw, tx, stream) : launch_rows<true, false>(p, num_sms, tiles, tw, tx, stream);
  }
  const int stage_bytes = kATile + bn * kBKBytes;
  const int max_stages = (227 * 1024 - 1024 - 8 * kStgWarp - static_cast<int>(sizeof(Tail)) - 256) / stage_bytes;
  if (stages <= 0 || stages > max_stages) stages = max_stages;
  if (stages > 8) stages = 8;
  p.stages = stages;
  CUtensorMap tw, tx;
  int rc = cached_tmap(&tw, Wq, N, K, K, kBM, 1);
  if (rc != MB_OK) return rc;
  rc = cached_tmap(&tx, Xq, M, K, K, bn, 1);
  if (rc != MB_OK) return rc;
  const size_t smem = static_cast<size_t>(stages) * stage_bytes + 8 * kStgWarp + sizeof(Tail) + 1024;
  const int kb_all = (K + 127) / 128;
  p.kb_per_split = (kb_all + splits - 1) / splits;
  p.splits = splits;
  p.partial = static_cast<float*>(workspace);
  p.expert_offsets = nullptr; p.w_rows = 0; p.sw_rows = 0; p.n_experts = 0;
  dim3 grid((M + bn - 1) / bn, (N + kBM - 1) / kBM, splits);
  const bool resid = (flags & 2) && splits == 1;
  static PerDeviceOnce configured;
  if (configured.needed()) {
    cudaFuncSetAttribute(gemm_fp8_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaFuncSetAttribute(gemm_fp8_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    configured.done();
  }
  if (resid)
    gemm_fp8_kernel<true><<<grid, kThreads, smem, stream>>>(tw, tx, p);
  else
    gemm_fp8_kernel<false><<<grid, kThreads, smem, stream>>>(tw, tx, p);
  if (splits > 1) {
    const size_t total4 = static_cast<size_t>(M) * N / 4;
    fp8_splitk_reduce_kernel<<<static_cast<unsigned>((total4 + 255) / 256), 256, 0, stream>>>(
        p.partial, (flags & 2) ? p.R : nullptr, p.Y, M, N, splits);
  }
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

// Whether a grouped product takes the form with tokens on M: where its 256-wide tiles keep half the SMs busy, or where the other form's
// grid, sized for any expert taking every row, is six waves and more of CTAs that mostly have nothing to do. Else the twice as many
// tiles of the other form are faster (148 SMs; 8 experts of 3072 x 7168, one row: 42 against 27 us; of 1536 x 2048, 128 rows: 17
// against 13; 64 experts of 2816 x 2048, 64 rows: 55 against 71; 256 of 4096 x 7168, 2048 rows: 1303 against 2936). Outputs of 128
// features fill half a tile (19 against 13 us). `avg` decides the other form's token tile.
extern "C" int mb_grouped_fp8_plan(int n_experts, int total_rows, int max_rows, int N, int num_sms, int* bn) {
  using namespace mb::f8;
  const int avg = (total_rows + n_experts - 1) / n_experts;
  *bn = avg <= 32 ? 32 : (avg <= 64 ? 64 : 128);
  if (N < kRowTileN || n_experts + total_rows / kBM > kMaxRowTiles) return 0;
  const long long tiles = static_cast<long long>((n_experts < total_rows ? n_experts : total_rows) + total_rows / kBM) * ((N + kRowTileN - 1) / kRowTileN);
  const long long ctas = static_cast<long long>(n_experts) * ((max_rows + *bn - 1) / *bn) * (N / kBM);
  return 2 * tiles >= num_sms || ctas >= 6ll * num_sms;
}

// Grouped block-scaled fp8 GEMM for mixture-of-experts layers: rows [offsets[e], offsets[e+1]) of Xq
// (tokens in expert order, scales Xs K-group-major over all `total_rows`) times expert e's weights
// Wq[e] ([N, K] e4m3 with 128x128 block scales Ws[e]). N % 128 == 0. `max_rows` bounds the rows of any
// expert (the grid is sized for it; CTAs past an expert's rows exit at once). `ldx` = byte stride of
// Xq rows (0 = K).
// Reference: max/python/max/nn/moe/moe_fp8.py:48 (MoEQuantized, fp8-blockwise strategy) over
// max/kernels/src/linalg/grouped_matmul_sm100_blockwise_fp8.mojo.
extern "C" int mb_grouped_gemm_fp8_blockscaled(const void* Xq, const float* Xs, const void* Wq, const float* Ws,
                                               void* Y, const int32_t* expert_offsets, int n_experts,
                                               int total_rows, int max_rows, int N, int K, int ldx, int bn,
                                               int stages, int* err, cudaStream_t stream) {
  using namespace mb::f8;
  if (total_rows <= 0 || N <= 0 || n_experts <= 0) return MB_OK;
  if (ldx <= 0) ldx = K;            // row stride of Xq in bytes (rows may carry trailing scale bytes)
  if (K % 16 || N % 128 || ldx % 16 || ldx < K) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(Xq) | reinterpret_cast<uintptr_t>(Wq) | reinterpret_cast<uintptr_t>(Y)) & 15)
    return MB_ERR_ALIGN;
  if (max_rows <= 0 || max_rows > total_rows) max_rows = total_rows;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // a caller that names a token tile (expert parallelism does, from the rows it expects) gets the form with weights on M
  const bool rows_form = bn <= 0 && mb_grouped_fp8_plan(n_experts, total_rows, max_rows, N, sms, &bn) != 0;
  if (bn % 32 || bn < 32 || bn > 128) return MB_ERR_SHAPE;
  Params p = {};
  p.Y = static_cast<__nv_bfloat16*>(Y);
  p.R = nullptr;
  p.sw = Ws; p.sx = Xs; p.err = err;
  p.M = total_rows; p.N = N; p.K = K; p.ldy = N; p.ldr = N; p.sw_ld = (K + 127) / 128; p.BN = bn;
  if (rows_form) {
    p.expert_offsets = expert_offsets;
    p.n_experts = n_experts;
    p.w_rows = N;
    p.sw_rows = N / 128;
    CUtensorMap tw, tx;
    int rc = cached_tmap(&tw, Wq, static_cast<uint64_t>(n_experts) * N, K, K, kBM, 1);
    if (rc != MB_OK) return rc;
    rc = cached_tmap(&tx, Xq, total_rows, K, ldx, kBM, 1);
    if (rc != MB_OK) return rc;
    return launch_rows<false, false>(p, sms, 1 << 30, tw, tx, stream);
  }
  const int stage_bytes = kATile + bn * kBKBytes;
  const int max_stages = (227 * 1024 - 1024 - 8 * kStgWarp - static_cast<int>(sizeof(Tail)) - 256) / stage_bytes;
  if (stages <= 0 || stages > max_stages) stages = max_stages;
  if (stages > 8) stages = 8;
  p.stages = stages;
  p.splits = 1;
  p.kb_per_split = (K + 127) / 128;
  p.partial = nullptr;
  p.expert_offsets = expert_offsets;
  p.n_experts = n_experts;
  p.w_rows = N;
  p.sw_rows = N / 128;
  CUtensorMap tw, tx;
  int rc = cached_tmap(&tw, Wq, static_cast<uint64_t>(n_experts) * N, K, K, kBM, 1);
  if (rc != MB_OK) return rc;
  rc = cached_tmap(&tx, Xq, total_rows, K, ldx, bn, 1);
  if (rc != MB_OK) return rc;
  const size_t smem = static_cast<size_t>(stages) * stage_bytes + 8 * kStgWarp + sizeof(Tail) + 1024;
  static PerDeviceOnce configured;
  if (configured.needed()) {
    cudaFuncSetAttribute(gemm_fp8_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    configured.done();
  }
  // an upper bound of the number of token tiles: every expert wastes less than one tile, and no expert has
  // more than max_rows rows
  long long tiles = (total_rows + bn - 1) / bn + n_experts;
  const long long by_expert = static_cast<long long>(n_experts) * ((max_rows + bn - 1) / bn);
  if (by_expert < tiles) tiles = by_expert;
  dim3 grid(static_cast<unsigned>(tiles), N / kBM, 1);
  gemm_fp8_kernel<false><<<grid, kThreads, smem, stream>>>(tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}
