// Prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): paged grouped-query heads of width 128, and
// latent heads projected up to keys of 192 and values of 128 (contiguous rows).
//
// A tile is 128 query rows of one (sequence, KV head): 128/G consecutive tokens x the G query heads that share the KV head (GQA
// packing puts them on the MMA M dimension). A CTA owns one tile (paged heads; two CTAs an SM) or two (latent heads, whose
// operands fill an SM's shared memory) and walks the sequence's keys 64 at a time:
//
//   warp 0      TMA producer: K tiles and V tiles (boxes of 64 rows x 64 columns, 128B swizzle) into a ring of five slots
//   warp 1      MMA issuer. One tile: S = Q . K^T of the next keys into the other of two score buffers, while the softmax has this
//               one; then O += P . V (P read from TMEM, V an MN-major operand straight from the row-major rows). Two tiles, for
//               tile g in turn: O_g += P_g . V, then S_g of the next keys into the columns P_g was read from. (MMAs of one
//               thread run in order.)
//   warps 4-7   softmax of tile 0, warps 8-11 of tile 1: one query row per thread (TMEM lane = row). Read S, mask, row
//               maximum, exponentials, P (bf16) back into the columns of S. The output stays in TMEM; it is rescaled only
//               when a row's maximum has grown by more than 2^8 since the reference maximum was taken (exact after the
//               final 1/l normalisation, because P is always computed against that reference)
//
// While one tile's softmax runs, the tensor pipe works for the other tile, of this CTA or of the other on the SM. Per 256 x 128 scores
// the four MMAs take 2048 cycles and the exponentials as many (16 a cycle and SM), so both pipes bound it together; what is lost is the
// chain between them. 32 heads over 8, causal: 8000 tokens 927 us with one tile an SM, P through shared memory and a third wait a tile;
// 570 with two tiles of 256 rows a CTA and 128 keys; 508 so, and short prompts, of which a pair of tiles was mostly empty, gain more
// (64 of 64 tokens 65, 65 and 48 us; 16 heads of 64 x 64 tokens 47, 54 and 29).
//
// (Exponentials of one tile under the products of another, and the lazy rescaling, are the schedule that FlashAttention-3 and -4
// published.)
//
// A sliding window of W keys (itself and the W - 1 before it) starts the walk at the first tile any row of the CTA
// sees and masks the edge; a sink score per head only adds exp(sink) to the denominator.
//
// All mbarrier waits are bounded; a timed-out wait raises the error word, and the CTA drains,
// frees its TMEM and leaves. Decode rows (one token per sequence) stay on the mma.sync kernel of
// attention_tma.cu: with one token only G of the 256 MMA rows would be used.
//
// Reference counterpart: max/kernels/src/nn/attention/gpu/nvidia/sm100/attention.mojo (FA4 prefill).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/api.h"
#include "../common/head_gate.cuh"
#include "../common/launch.h"
#include "../common/ptx.cuh"
#include "gemm_common.h"

namespace mb {
namespace atc {

typedef __nv_bfloat16 bf16;
constexpr int HD = 128;        // values, and keys without a rotated part of their own
constexpr int kSlots = 5;      // K and V tiles in turn

struct Params {
  const bf16* q;
  const bf16* q_rope;    // LATENT: the rotated 64 columns of a key's query, ld_rope between tokens, rope_head between heads
  bf16* out;
  const int32_t* block_table;
  const int32_t* kv_start;   // LATENT: first row of every sequence in the projected keys
  const int32_t* q_start;
  const int32_t* q_len;
  const int32_t* kv_len;
  const int32_t* tile_seq;
  const int32_t* tile_q0;
  int* err;
  long long k_off_rows, v_off_rows, page_rows;
  int ldq, ldo, bt_stride, page_size, n_tiles, G, q_head, ld_rope, rope_head;
  float scale_log2;
  int window;            // keys a query sees (0x7fffffff: all before it)
  const float* sink;     // per query head, or null
  HeadGate gate;
};

struct Bars {
  uint64_t full[kSlots];
  uint64_t empty[kSlots];
  uint64_t s_full[2];
  uint64_t p_full[2];
  uint64_t o_done[2];
  uint64_t pv_done[2];     // one tile: the products with V, in turn. A wait for one of them is not confused by the phases around it:
                           // the product two before it ended before the scores that the waiting warp has, the one two after cannot begin
  uint32_t tmem_base;
  int abort_word;
};

// MN-major operand with 128B swizzle: rows of 64 contiguous MN elements (128 B), 8 consecutive K rows
// form one 1024 B swizzle atom (SBO = stride between atoms along K), the next 64 MN elements live
// LBO bytes away.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(const void* smem_tile, uint32_t lbo_bytes,
                                                       uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_u32(smem_tile) & 0x3ffff) >> 4);
  d |= static_cast<uint64_t>(lbo_bytes >> 4) << 16;
  d |= static_cast<uint64_t>(sbo_bytes >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// D += A . B with A in TMEM (16-bit values, two a column) and B in shared memory
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool LATENT>
struct Shape {
  static constexpr int TILES = LATENT ? 2 : 1;                    // query tiles of a CTA
  static constexpr int NC = LATENT ? 3 : 2;                       // 64-column chunks of a key
  static constexpr int BN = 64;                                   // keys per tile
  static constexpr int kThreads = 128 + TILES * 128;              // warps 2 and 3 idle: register budgets belong to groups of four warps
  static constexpr uint32_t kTmemCols = TILES * 256;              // S / P of tile 0 | of tile 1 | O of tile 0 | of tile 1 (128 each)
  static constexpr int kScoreCols = TILES == 1 ? 64 : 128;        // one tile: S / P of even keys' tiles | of odd ones | O
  static constexpr int kQTile = NC * 128 * 128;                   // 128 rows
  static constexpr int kKBytes = NC * BN * 128, kVBytes = 2 * BN * 128;
  static constexpr int kSlot = kKBytes > kVBytes ? kKBytes : kVBytes;
  static constexpr size_t kSmem = TILES * kQTile + kSlots * kSlot + sizeof(Bars);
};

template <bool LATENT>
__global__ void __launch_bounds__(Shape<LATENT>::kThreads, LATENT ? 1 : 2)
attn_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmR, const __grid_constant__ CUtensorMap tmV,
               const Params p) {
  using Sh = Shape<LATENT>;
  constexpr int BN = Sh::BN, NC = Sh::NC, TILES = Sh::TILES;
  // No alignment slack. The dynamic shared memory window starts 1024-byte aligned (there is no static shared memory in
  // this kernel); should a future toolchain place it elsewhere the kernel reports it instead of computing garbage.
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if (smem_u32(smem_raw) & 1023u) {
    if (threadIdx.x == 0 && p.err) atomicCAS(p.err, 0, 799);
    return;
  }
  uint8_t* sQ = smem_raw;                           // [tile][chunk][128 rows x 128 B]
  uint8_t* sRing = sQ + TILES * Sh::kQTile;         // [slot][chunk][BN rows x 128 B]
  Bars* bars = reinterpret_cast<Bars*>(sRing + kSlots * Sh::kSlot);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kvh = blockIdx.x;
  const int G = p.G;
  const int tok_per_tile = 128 / G;

  // A CTA covers two tiles of the plan as a rule, and leaves at the second. First come those that have work (the even ones, where
  // sequences have even numbers of tiles), spread over all SMs; in each half the later tiles of a prompt, which see more keys.
  const int n_tiles = gridDim.y, even = (n_tiles + 1) >> 1, at = blockIdx.y;
  const int tile = at < even ? 2 * (even - 1 - at) : 2 * (n_tiles - 1 - at) + 1;
  const int seq = p.tile_seq[tile];
  if (seq < 0) return;                 // an unused tile of a plan made on the device
  const int tq0 = p.tile_q0[tile];
  if (tq0 % (TILES * tok_per_tile) != 0) return;  // covered by the CTA of a tile before it
  const int qs = p.q_start[seq], ql = p.q_len[seq], kl = p.kv_len[seq];
  const bool two = TILES == 2 && tq0 + tok_per_tile < ql;         // the second tile has rows
  const int last_tq = min(tq0 + TILES * tok_per_tile, ql);
  const int kv_hi = kl - ql + last_tq;
  const int kv_lo = kl - ql + tq0 - p.window + 1;        // first key the CTA's first row sees
  const int t_first = kv_lo > 0 ? kv_lo / BN : 0;
  const int ntiles = (kv_hi + BN - 1) / BN - t_first;

  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(&bars->s_full[g], 1);
      mbar_init(&bars->p_full[g], 4);
      mbar_init(&bars->o_done[g], 1);
      mbar_init(&bars->pv_done[g], 1);
    }
    bars->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, Sh::kTmemCols);
    tmem_relinquish();
  }
  if (warp >= 4) {
    // query rows of this CTA into shared memory, K-major with 128B swizzle (row r, 16 B piece c): a thread copies its own row
    const int g = (warp - 4) >> 2, r = (warp & 3) * 32 + lane;
    const int tq = tq0 + g * tok_per_tile + r / G, head = kvh * G + r % G;
    const bool valid = tq < ql;
    const int64_t row = qs + (valid ? tq : 0);
    const bf16* src = p.q + row * p.ldq + head * p.q_head;
#pragma unroll
    for (int ch = 0; ch < NC; ++ch) {
      const bf16* from = LATENT && ch == 2 ? p.q_rope + row * p.ld_rope + head * p.rope_head : src + ch * 64;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (valid) v = *reinterpret_cast<const uint4*>(from + c * 8);
        *reinterpret_cast<uint4*>(sQ + g * Sh::kQTile + ch * 16384 + r * 128 + ((c ^ (r & 7)) << 4)) = v;
      }
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  volatile int* abort_word = &bars->abort_word;

  // Two tiles: 384 x 168 registers at launch, four warps give theirs up, eight take them (128 x 56 + 256 x 224 is the same sum). One
  // tile: 256 x 128, of which four warps take 200 (128 x 56 + 128 x 200).
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0 && lane == 0) {
      // -------------------------------------------------------------- TMA producer
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      if (LATENT) tma_prefetch_desc(&tmR);
      const int32_t* bt = LATENT ? nullptr : p.block_table + static_cast<int64_t>(seq) * p.bt_stride;
      const int first_row = LATENT ? p.kv_start[seq] : 0;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = 0; t < ntiles && ok; ++t) {
        const int kv0 = (t_first + t) * BN;
        int row[BN / 64];              // first row of each 64-key part; parts beyond the keys repeat the first one (finite values)
#pragma unroll
        for (int h = 0; h < BN / 64; ++h) {
          const int k0 = h > 0 && kv0 + 64 * h >= kv_hi ? kv0 : kv0 + 64 * h;
          if (LATENT) row[h] = first_row + k0;
          else row[h] = static_cast<int>(static_cast<long long>(bt[k0 / p.page_size]) * p.page_rows + static_cast<long long>(kvh) * p.page_size + k0 % p.page_size);
        }
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          ok = ok && mbar_wait(&bars->empty[s], ph ^ 1, abort_word, p.err, 701);
          if (!ok) break;
          uint8_t* dst = sRing + s * Sh::kSlot;
          mbar_arrive_expect_tx(&bars->full[s], kv == 0 ? Sh::kKBytes : Sh::kVBytes);
          const long long off = kv == 0 ? p.k_off_rows : p.v_off_rows;
#pragma unroll
          for (int ch = 0; ch < (kv == 0 ? NC : 2); ++ch)
#pragma unroll
            for (int h = 0; h < BN / 64; ++h) {
              uint8_t* to = dst + ch * (BN * 128) + h * 8192;
              if (LATENT && kv == 0 && ch == 2) tma_load_2d(to, &tmR, &bars->full[s], 0, row[h]);
              else tma_load_2d(to, kv == 0 ? &tmK : &tmV, &bars->full[s], (LATENT ? kvh * HD : 0) + ch * 64,
                               static_cast<int32_t>(off + row[h]));
            }
          if (++s == kSlots) { s = 0; ph ^= 1; }
        }
      }
    } else if (warp == 1 && lane == 0) {
      // -------------------------------------------------------------- MMA issuer
      const uint32_t idesc_s = umma_idesc(128, BN, 1, 1);
      const uint32_t idesc_pv = umma_idesc(128, HD, 1, 1) | (1u << 16);   // B operand (V) is MN-major
      const int last = two ? 1 : 0;
      bool ok = true;
      auto wait_item = [&](int i) { ok = ok && mbar_wait(&bars->full[i % kSlots], (i / kSlots) & 1, abort_word, p.err, 702); };
      // S_g from ring item i; with one tile, S into buffer g
      auto scores = [&](int i, int g) {
        const uint8_t* sK = sRing + (i % kSlots) * Sh::kSlot;
#pragma unroll
        for (int k = 0; k < NC * 4; ++k) {
          const uint64_t da = umma_desc_sw128(sQ + (TILES == 2 ? g * Sh::kQTile : 0) + (k >> 2) * 16384) + static_cast<uint64_t>((k & 3) * 2);
          const uint64_t db = umma_desc_sw128(sK + (k >> 2) * (BN * 128)) + static_cast<uint64_t>((k & 3) * 2);
          umma_bf16(tmem_base + g * Sh::kScoreCols, da, db, idesc_s, k > 0 ? 1u : 0u);
        }
        tc_commit(&bars->s_full[g]);
        if (TILES == 1 || g == last) tc_commit(&bars->empty[i % kSlots]);
      };
      if (ntiles > 0) {
        wait_item(0);
        if (ok) {
          tc_fence_after();
          scores(0, 0);
          if (two) scores(0, 1);
        }
      }
      for (int t = 0; t < ntiles && ok && TILES == 1; ++t) {
        // the next scores go into the other buffer while the softmax has this one (the product that read P there was issued before)
        if (t + 1 < ntiles) {
          wait_item(2 * t + 2);
          if (!ok) break;
          tc_fence_after();
          scores(2 * t + 2, (t + 1) & 1);
        }
        wait_item(2 * t + 1);
        // (a barrier per buffer: the softmax may be through with the next tile before this one's values are there)
        ok = ok && mbar_wait(&bars->p_full[t & 1], (t >> 1) & 1, abort_word, p.err, 704);
        if (!ok) break;
        tc_fence_after();
        const uint8_t* sV = sRing + ((2 * t + 1) % kSlots) * Sh::kSlot;
#pragma unroll
        for (int k = 0; k < BN / 16; ++k)
          umma_bf16_ts(tmem_base + 128, tmem_base + (t & 1) * Sh::kScoreCols + k * 8, umma_desc_mn_sw128(sV + k * 2048, BN * 128, 1024), idesc_pv,
                       (t > 0 || k > 0) ? 1u : 0u);
        tc_commit(&bars->empty[(2 * t + 1) % kSlots]);
        tc_commit(&bars->pv_done[t & 1]);
        if (t + 1 == ntiles) tc_commit(&bars->o_done[0]);
      }
      for (int t = 0; t < ntiles && ok && TILES == 2; ++t) {
        for (int g = 0; g <= last && ok; ++g) {
          if (g == 0) wait_item(2 * t + 1);
          ok = ok && mbar_wait(&bars->p_full[g], t & 1, abort_word, p.err, 704);
          if (!ok) break;
          tc_fence_after();
          const uint8_t* sV = sRing + ((2 * t + 1) % kSlots) * Sh::kSlot;
#pragma unroll
          for (int k = 0; k < BN / 16; ++k)
            umma_bf16_ts(tmem_base + 256 + g * 128, tmem_base + g * 128 + k * 8, umma_desc_mn_sw128(sV + k * 2048, BN * 128, 1024), idesc_pv,
                         (t > 0 || k > 0) ? 1u : 0u);
          if (g == last) tc_commit(&bars->empty[(2 * t + 1) % kSlots]);
          if (t + 1 < ntiles) {
            if (g == 0) {
              wait_item(2 * t + 2);
              if (!ok) break;
              tc_fence_after();
            }
            scores(2 * t + 2, g);
          } else {
            tc_commit(&bars->o_done[g]);
          }
        }
      }
    }
  } else {
    if constexpr (TILES == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    // ---------------------------------------------------------------- softmax
    const int g = TILES == 1 ? 0 : (warp - 4) >> 2, quad = warp & 3, r = quad * 32 + lane;
    const int tq = tq0 + g * tok_per_tile + r / G, head = kvh * G + r % G;
    const int limit = tq < ql ? kl - ql + tq : -1;
    const uint32_t s_tile = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + g * 128, o_addr = s_tile + TILES * 128;
    float m_ref = 0.f, l = 0.f;       // P and l are relative to m_ref (a lagging running maximum)
    bool ok = true, unset = true;     // unset: no key has been visible to the row yet
    const int mine = g == 0 || two ? ntiles : 0;
    for (int t = 0; t < mine; ++t) {
      // the scores are there; with two tiles, so is everything issued before them: the last P . V has retired, O is at rest
      const uint32_t s_addr = TILES == 1 ? s_tile + (t & 1) * Sh::kScoreCols : s_tile;
      ok = TILES == 1 ? mbar_wait(&bars->s_full[t & 1], (t >> 1) & 1, abort_word, p.err, 706) : mbar_wait(&bars->s_full[g], t & 1, abort_word, p.err, 706);
      if (!ok) break;
      tc_fence_after();
      uint32_t sr[BN / 32][32];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32(s_addr + c * 32, sr[c]);
      tc_wait_ld();
      const int kv0 = (t_first + t) * BN;
      // row maximum of the raw scores (four independent chains); only tiles that touch the causal
      // diagonal, the end of the sequence or the edge of the window need the mask
      float mxa[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (!(kv0 + BN - 1 <= limit && limit - kv0 < p.window)) {
#pragma unroll
        for (int c = 0; c < BN; ++c)
          if (static_cast<uint32_t>(limit - (kv0 + c)) >= static_cast<uint32_t>(p.window)) sr[c >> 5][c & 31] = __float_as_uint(-INFINITY);
      }
#pragma unroll
      for (int c = 0; c < BN; ++c) mxa[c & 3] = fmaxf(mxa[c & 3], __uint_as_float(sr[c >> 5][c & 31]));
      const float mx = fmaxf(fmaxf(mxa[0], mxa[1]), fmaxf(mxa[2], mxa[3])) * p.scale_log2;   // scale > 0
      bool grow = false;
      if (unset) {                     // everything so far was masked: the sum and the accumulator are zero
        unset = mx == -INFINITY;
        m_ref = unset ? 0.f : mx;
      } else {
        grow = mx - m_ref > 8.0f;      // probabilities would exceed 2^8: move the reference
      }
      if (__any_sync(0xffffffffu, grow)) {
        if (TILES == 1) {              // the last P . V may still be adding (this tile's cannot have begun, the one before it is done)
          ok = t == 0 || mbar_wait(&bars->pv_done[(t - 1) & 1], ((t - 1) >> 1) & 1, abort_word, p.err, 707);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
          tc_fence_after();
        }
        // rescale this warp's 32 accumulator rows (factor 1 for rows whose reference stays)
        const float factor = grow ? exp2f(m_ref - mx) : 1.0f;
        if (grow) { m_ref = mx; l *= factor; }
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t tr[32];
          tmem_ld_32x32(o_addr + q4 * 32, tr);
          tc_wait_ld();
#pragma unroll
          for (int c = 0; c < 32; ++c) tr[c] = __float_as_uint(__uint_as_float(tr[c]) * factor);
          tmem_st_32x32(o_addr + q4 * 32, tr);
        }
      }
      float la[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < BN / 64; ++c) {
        uint32_t pk[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float p0 = ex2(fmaf(__uint_as_float(sr[2 * c + (j >> 4)][2 * (j & 15)]), p.scale_log2, -m_ref));
          const float p1 = ex2(fmaf(__uint_as_float(sr[2 * c + (j >> 4)][2 * (j & 15) + 1]), p.scale_log2, -m_ref));
          la[j & 3] += p0 + p1;
          const __nv_bfloat162 v2 = __floats2bfloat162_rn(p0, p1);
          pk[j] = *reinterpret_cast<const uint32_t*>(&v2);
        }
        tmem_st_32x32(s_addr + c * 32, pk);
      }
      l += (la[0] + la[1]) + (la[2] + la[3]);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full[TILES == 1 ? t & 1 : g]);
    }
    if (ok && mine > 0) ok = mbar_wait(&bars->o_done[g], 0, abort_word, p.err, 708);
    if (ok && mine > 0) {
      tc_fence_after();
      float w = 1.f;
      if (p.sink) {
        const float sink2 = p.sink[head] * 1.4426950408889634f;
        const float mm = fmaxf(l > 0.f ? m_ref : -INFINITY, sink2);
        w = l > 0.f ? exp2f(m_ref - mm) : 0.f;
        l = l * w + exp2f(sink2 - mm);
      }
      w = l > 0.f ? w / l : 0.f;
      if (tq < ql) w *= p.gate(qs + tq, head);
      bf16* orow = p.out + static_cast<int64_t>(qs + (tq < ql ? tq : 0)) * p.ldo + head * HD;
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        uint32_t ta[32];
        tmem_ld_32x32(o_addr + q4 * 32, ta);          // warp-collective: every lane takes part
        tc_wait_ld();
        if (tq < ql) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __nv_bfloat162 v2 = __floats2bfloat162_rn(__uint_as_float(ta[c * 8 + 2 * j]) * w, __uint_as_float(ta[c * 8 + 2 * j + 1]) * w);
              pk[j] = *reinterpret_cast<const uint32_t*>(&v2);
            }
            *reinterpret_cast<uint4*>(orow + q4 * 32 + c * 8) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Sh::kTmemCols);
  }
}

// An ordinary launch, and no early start of the next kernel either: both would hide a microsecond or two, and these CTAs take
// all registers and shared memory of their SM, so that a grid of them that waits for the kernel before it leaves no room for
// anything else.
template <bool LATENT>
static int launch(const CUtensorMap& tk, const CUtensorMap& tr, const CUtensorMap& tv, const Params& p, int heads, cudaStream_t stream) {
  static PerDeviceOnce configured;
  if (configured.needed()) {
    if (cudaFuncSetAttribute(attn_tc_kernel<LATENT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Shape<LATENT>::kSmem)) !=
        cudaSuccess)
      return MB_ERR_LAUNCH;
    configured.done();
  }
  using Sh = Shape<LATENT>;
  return launch_plain(attn_tc_kernel<LATENT>, dim3(heads, p.n_tiles), dim3(Sh::kThreads), Sh::kSmem, stream, tk, tr, tv, p) == cudaSuccess
             ? MB_OK
             : MB_ERR_LAUNCH;
}

}  // namespace atc
}  // namespace mb

using namespace mb;

// Prefill tiles of a ragged batch on the tcgen05 kernel. Same KV addressing as mb_paged_attention_tma
// (kv_base viewed as [total_rows, 128]); head_dim 128, G = n_q / n_kv in {1, 2, 4, 8, 16}, page_size % 64 == 0.
// tile_seq / tile_q0 is the plan of 64-row tiles (CTAs take two of them) or of 128-row tiles; a negative sequence is an unused
// tile.
extern "C" int mb_paged_attention_prefill_tc(const void* q, int ldq, void* out, int ldo, const void* kv_base,
                                             long long total_rows, long long k_off_rows, long long v_off_rows,
                                             long long page_rows, const int32_t* block_table, int bt_stride,
                                             const int32_t* q_start, const int32_t* q_len, const int32_t* kv_len,
                                             const int32_t* tile_seq, const int32_t* tile_q0, int n_tiles, int n_q,
                                             int n_kv, int head_dim, int page_size, float scale,
                                             const MbAttnOptions* opt, int* err, cudaStream_t stream) {
  using namespace mb::atc;
  if (n_tiles <= 0) return MB_OK;
  if (head_dim != 128 || n_kv <= 0 || n_q % n_kv || page_size % 64 || total_rows >= (1ll << 31)) return MB_ERR_SHAPE;
  const int G = n_q / n_kv;
  if (G > 16 || (G & (G - 1))) return MB_ERR_SHAPE;
  if (reinterpret_cast<uintptr_t>(kv_base) & 15 || ldq % 8 || ldo % 8) return MB_ERR_ALIGN;
  Params p = {};
  p.q = static_cast<const bf16*>(q);
  p.out = static_cast<bf16*>(out);
  p.block_table = block_table;
  p.q_start = q_start; p.q_len = q_len; p.kv_len = kv_len;
  p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
  p.err = err;
  p.k_off_rows = k_off_rows; p.v_off_rows = v_off_rows; p.page_rows = page_rows;
  p.ldq = ldq; p.ldo = ldo; p.bt_stride = bt_stride; p.page_size = page_size; p.n_tiles = n_tiles; p.G = G; p.q_head = head_dim;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.window = opt && opt->window > 0 ? opt->window : 0x7fffffff;
  p.sink = opt ? opt->sink : nullptr;
  p.gate = HeadGate(opt);
  CUtensorMap tm;
  const int rc = cached_tmap(&tm, kv_base, static_cast<uint64_t>(total_rows), head_dim, head_dim, 64, 2);
  if (rc != MB_OK) return rc;
  return launch<false>(tm, tm, tm, p, n_kv, stream);
}

// Latent attention of prompts in its plain form: keys [128 projected | 64 rotated, shared by the heads] and values [128]
// per head, rows of sequence s from kv_start[s] on. `kv` holds [rows, keys of all heads | values of all heads]. A query and
// a key meet in 192 + 128 products a head instead of the absorbed form's 576 + 512.
extern "C" int mb_latent_prefill_tc(const void* q, int ldq, int q_head, const void* q_rope, int ld_rope, int rope_head, void* out, int ldo,
                                    const void* kv, int ld_kv, const void* k_rope, long long rows, const int32_t* kv_start,
                                    const int32_t* q_start, const int32_t* q_len, const int32_t* kv_len, const int32_t* tile_seq,
                                    const int32_t* tile_q0, int n_tiles, int n_heads, float scale, const MbAttnOptions* opt, int* err,
                                    cudaStream_t stream) {
  using namespace mb::atc;
  if (n_tiles <= 0 || rows <= 0) return MB_OK;
  if (n_heads <= 0 || n_heads > 65535 || ld_kv < 2 * n_heads * HD || rows >= (1ll << 31)) return MB_ERR_SHAPE;
  if (((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(q_rope) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(kv) |
        reinterpret_cast<uintptr_t>(k_rope)) & 15) || (ldq | q_head | ld_rope | rope_head | ldo | ld_kv) % 8)
    return MB_ERR_ALIGN;
  Params p = {};
  p.q = static_cast<const bf16*>(q);
  p.q_rope = static_cast<const bf16*>(q_rope);
  p.out = static_cast<bf16*>(out);
  p.kv_start = kv_start;
  p.q_start = q_start; p.q_len = q_len; p.kv_len = kv_len;
  p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
  p.err = err;
  p.ldq = ldq; p.ldo = ldo; p.q_head = q_head; p.ld_rope = ld_rope; p.rope_head = rope_head; p.n_tiles = n_tiles; p.G = 1;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.window = opt && opt->window > 0 ? opt->window : 0x7fffffff;
  p.sink = opt ? opt->sink : nullptr;
  p.gate = HeadGate(opt);
  CUtensorMap tk, tr, tv;
  const int cols = n_heads * HD;
  int rc = cached_tmap(&tk, kv, static_cast<uint64_t>(rows), cols, ld_kv, 64, 2);
  if (rc != MB_OK) return rc;
  rc = cached_tmap(&tv, static_cast<const bf16*>(kv) + cols, static_cast<uint64_t>(rows), cols, ld_kv, 64, 2);
  if (rc != MB_OK) return rc;
  rc = cached_tmap(&tr, k_rope, static_cast<uint64_t>(rows), 64, 64, 64, 2);
  if (rc != MB_OK) return rc;
  return launch<true>(tk, tr, tv, p, n_heads, stream);
}

namespace mb {
namespace atc {
// Rows [0, kv_len[s]) of every sequence, out of the pages: latents [rows, R] and rotated parts [rows, 64], 16 bytes a thread.
// Rows between a sequence's end and the next one's start are zeros.
__global__ void latent_gather_kernel(const bf16* __restrict__ cache, long long page_stride, int ld, int page, const int32_t* __restrict__ block_table,
                                     int bt_stride, const int32_t* __restrict__ kv_start, const int32_t* __restrict__ kv_len, int B, int R,
                                     bf16* __restrict__ c, bf16* __restrict__ rope, long long rows) {
  const int per = (R + 64) / 8;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * per) return;
  const int row = static_cast<int>(i / per), col = static_cast<int>(i % per) * 8;
  int lo = 0, hi = B - 1;                            // the last sequence that starts at or before the row
  while (lo < hi) {
    const int m = (lo + hi + 1) >> 1;
    if (kv_start[m] <= row) lo = m; else hi = m - 1;
  }
  const int at = row - kv_start[lo];
  uint4 v = make_uint4(0, 0, 0, 0);
  if (at < kv_len[lo])
    v = *reinterpret_cast<const uint4*>(cache + block_table[static_cast<long long>(lo) * bt_stride + at / page] * page_stride +
                                        static_cast<long long>(at % page) * ld + col);
  bf16* dst = col < R ? c + static_cast<long long>(row) * R + col : rope + static_cast<long long>(row) * 64 + (col - R);
  *reinterpret_cast<uint4*>(dst) = v;
}

// Weights of the projection: out rows [h 128 | h 128] x R from w_uk [h, R, 128] (transposed per head, tiles of 64 x 64 through shared
// memory) and w_uv [h, 128, R] (as it is). Made anew for each layer of a step, in the step's scratch: kept, it would be a second copy of
// both (2 GB for 61 layers of 128 heads), and an old one once the weights change. 128 heads, R = 512: 48 us as three torch kernels.
__global__ void __launch_bounds__(256) latent_stack_kernel(const bf16* __restrict__ w_uk, const bf16* __restrict__ w_uv, bf16* __restrict__ out, int h, int R) {
  __shared__ bf16 tile[64][66];
  const int head = blockIdx.z, r0 = blockIdx.x * 64, n0 = (blockIdx.y & 1) * 64, tid = threadIdx.x, row = tid >> 3, c = (tid & 7) * 8;
  if (blockIdx.y >= 2) {                             // 64 value rows of a head
    const size_t at = (static_cast<size_t>(head) * 128 + n0) * R + r0;
#pragma unroll
    for (int q = 0; q < 64; q += 32)
      *reinterpret_cast<uint4*>(out + static_cast<size_t>(h) * 128 * R + at + static_cast<size_t>(row + q) * R + c) =
          *reinterpret_cast<const uint4*>(w_uv + at + static_cast<size_t>(row + q) * R + c);
    return;
  }
#pragma unroll
  for (int q = 0; q < 64; q += 32) {
    const uint4 v = *reinterpret_cast<const uint4*>(w_uk + (static_cast<size_t>(head) * R + r0 + row + q) * 128 + n0 + c);
    uint32_t* to = reinterpret_cast<uint32_t*>(&tile[row + q][c]);
    to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 64; q += 32) {
    __align__(16) bf16 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = tile[c + i][row + q];
    *reinterpret_cast<uint4*>(out + (static_cast<size_t>(head) * 128 + n0 + row + q) * R + r0 + c) = *reinterpret_cast<const uint4*>(v);
  }
}
}  // namespace atc
}  // namespace mb

extern "C" int mb_latent_stack(const void* w_uk, const void* w_uv, void* out, int heads, int R, cudaStream_t stream) {
  using namespace mb::atc;
  if (heads <= 0 || R <= 0) return MB_OK;
  if (R % 64 || heads > 65535) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(w_uk) | reinterpret_cast<uintptr_t>(w_uv) | reinterpret_cast<uintptr_t>(out)) & 15) return MB_ERR_ALIGN;
  latent_stack_kernel<<<dim3(R / 64, 4, heads), 256, 0, stream>>>(static_cast<const bf16*>(w_uk), static_cast<const bf16*>(w_uv), static_cast<bf16*>(out), heads, R);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}

extern "C" int mb_latent_gather(const void* cache, long long page_stride, int ld, int page, const int32_t* block_table, int bt_stride,
                                const int32_t* kv_start, const int32_t* kv_len, int B, int R, void* c, void* rope, long long rows,
                                cudaStream_t stream) {
  using namespace mb::atc;
  if (rows <= 0 || B <= 0) return MB_OK;
  if (R % 8 || ld % 8 || page_stride % 8) return MB_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(rope)) & 15) return MB_ERR_ALIGN;
  const long long work = rows * ((R + 64) / 8);
  latent_gather_kernel<<<static_cast<unsigned>((work + 255) / 256), 256, 0, stream>>>(
      static_cast<const bf16*>(cache), page_stride, ld, page, block_table, bt_stride, kv_start, kv_len, B, R, static_cast<bf16*>(c),
      static_cast<bf16*>(rope), rows);
  return cudaGetLastError() == cudaSuccess ? MB_OK : MB_ERR_LAUNCH;
}
