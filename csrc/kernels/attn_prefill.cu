// Paged flash-attention prefill on tcgen05 / TMEM (varlen, causal with bottom-right
// alignment, GQA, sliding window, soft-cap), head_dim 64, 128 or 256.
//
// One CTA = one 128-row query tile of one request and one query head; two CTAs share an SM.
// Per 64-token KV tile:  S = Q K^T  (tcgen05, A = Q smem, B = K smem, both K-major SW128,
// fp32 S in TMEM), softmax with one thread per query row (TMEM lane == row, so no
// cross-thread reductions), P written to smem as bf16 in the UMMA K-major swizzled layout,
// then  PV = P V  with V as an MN-major operand (the pages land in smem exactly as they sit
// in the cache, d contiguous). QK^T of tile j+1 and PV of tile j-1 run on the tensor pipe
// while the softmax warps work on tile j; S is double-buffered in TMEM; O is accumulated in
// TMEM by the tensor pipe and rescaled in place only when a row's reference max is raised
// (lazily, by more than 2^8).
//
// K and V tiles share one ring of three TMA slots, filled in the order the MMA warp consumes them
// (K0 K1 V0 K2 V1 ...); pages are fetched with 3-D TMA boxes
// (64 dims x 1 head x min(block_size, 64) tokens) straight from the paged cache
// [num_blocks, 2, block_size, Hkv, D].
//
// Warp roles (192 threads): warp 0 TMA producer, warp 1 MMA issuer + TMEM owner,
// warps 2..5 softmax + output.
//
// Replaces the reference prefill ladder (src/vt/cuda/cuda_paged_attn.cu:567 PagedFlashKernel,
// :720-1686 wmma variants, and the vendored FA2 path cuda_flash_attn_fa2.cu), none of which
// has an sm_100 tensor-core body.
#include <mutex>
#include <unordered_map>

#include "api.h"
#include "sm100.cuh"

namespace b200 {

static constexpr int kQT = 128;   // query rows per CTA
static constexpr int kKT = 64;    // kv tokens per tile
static constexpr int kRing = 3;   // K/V slots

struct PrefillParams {
  __nv_bfloat16* out;   // [T, Hq*D]
  int ldo;
  float* lse;           // optional [T, Hq] natural-log LSE
  const int32_t* block_table;  // [B, max_blocks]
  int max_blocks;
  const int32_t* seq_lens;     // [B]
  const int32_t* q_start;      // [B+1]
  const int32_t* tile_req;     // [num_tiles]
  const int32_t* tile_q0;      // [num_tiles] first query row of the tile inside its request
  int Hq, Hkv, block_size;
  float scale_log2;            // softmax scale * log2(e)
  float softcap2;              // soft-cap in the log2 domain, 0 = off
  int window;                  // > 0: sliding window (tokens to the left incl. self); < 0: chunked-local
                               // attention with chunks of -window tokens (a query sees its own chunk); 0 = off
  int causal;
  int* status;
};

struct alignas(8) PrefillBars {
  uint64_t q_full;
  uint64_t kv_full[kRing], kv_empty[kRing];
  uint64_t s_full[2], s_empty[2];
  uint64_t p_full, p_empty, o_full;
  uint32_t tmem_base;
};

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}


// D = 256 keeps two softmax threads per query row (warps w and w + 4 share a TMEM lane
// quarter): both reduce the full score row, each writes half of P and owns half of O.
template <int D>
__global__ void __launch_bounds__(64 + 128 * (D > 128 ? 2 : 1), D > 128 ? 1 : 2)
    attn_prefill_kernel(const __grid_constant__ CUtensorMap tmQ,
                        const __grid_constant__ CUtensorMap tmKV, PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  constexpr int kDH = D / 64;                     // 64-wide halves of the head dim
  constexpr int kSplit = D > 128 ? 2 : 1;         // softmax threads per query row
  constexpr int kDO = D / kSplit;                 // output dims owned by one thread
  constexpr uint32_t kTmemCols = D > 128 ? 512 : 256;
  constexpr int kQHalf = kQT * 128;               // 16 KB: 128 rows x 128 B
  constexpr int kKVHalf = kKT * 128;              // 8 KB: 64 tokens x 128 B
  constexpr int kQBytes = kDH * kQHalf;
  constexpr int kSlotBytes = kDH * kKVHalf;       // one K or V tile
  constexpr int kPBytes = kQT * kKT * 2;          // 16 KB: one K-major half-tile
  uint8_t* sQ = smem;
  uint8_t* sKV = sQ + kQBytes;
  uint8_t* sP = sKV + kRing * kSlotBytes;
  PrefillBars* bars = reinterpret_cast<PrefillBars*>(sP + kPBytes);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tile = blockIdx.x, h = blockIdx.y;
  const int hkv = h / (p.Hq / p.Hkv);
  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&bars->kv_full[i], 1);
      mbar_init(&bars->kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->s_empty[i], 4 * kSplit);
    }
    mbar_init(&bars->p_full, 4 * kSplit);
    mbar_init(&bars->p_empty, 1);
    mbar_init(&bars->o_full, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  const uint32_t tmem_s0 = tmem_base, tmem_o = tmem_base + 128;
  pdl_wait();
  pdl_launch_dependents();
  const int req = p.tile_req[tile];
  const int q0 = p.tile_q0[tile];
  const int q_begin = p.q_start[req];
  const int q_len = p.q_start[req + 1] - q_begin;
  const int seq_len = p.seq_lens[req];
  const int ctx_off = seq_len - q_len;          // position of query row 0
  const int rows = min(kQT, q_len - q0);
  // kv range needed by this tile
  const int last_pos = p.causal ? (ctx_off + q0 + rows - 1) : (seq_len - 1);
  int first_pos = 0;
  if (p.window > 0) first_pos = max(0, ctx_off + q0 - p.window + 1);
  else if (p.window < 0) first_pos = ((ctx_off + q0) / -p.window) * -p.window;   // chunk start of the first row
  const int kt0 = first_pos / kKT;
  const int kt1 = last_pos / kKT + 1;           // exclusive
  const int ntiles = kt1 - kt0;

  // The producer and the issuer walk their loops as whole warps and elect the lane that issues (mbar_wait_warp).
  if (warp == 0) {
    if (elect_one()) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmKV);
      mbar_expect_tx(&bars->q_full, kQBytes);
      for (int dh = 0; dh < kDH; ++dh)
        tma_load_2d(sQ + dh * kQHalf, &tmQ, &bars->q_full, h * D + dh * 64, q_begin + q0);
    }
    __syncwarp();
    const int32_t* bt = p.block_table + (size_t)req * p.max_blocks;
    const int nblk_valid = (seq_len + p.block_size - 1) / p.block_size;
    const int rows_per_load = min(p.block_size, kKT);
    const int loads = kKT / rows_per_load;                      // pages of a tile (at most 8): a lane each
    // Load order K0 K1 V0 K2 V1 K3 ... V(n-1): the order in which the MMA warp consumes the
    // tiles, with K one tile further ahead than V (V slots are held until the softmax of their
    // tile is done; K slots turn over as soon as QK^T has run).
    const int nseq = 2 * ntiles;
    int sl = 0;
    uint32_t ph = 1;
    for (int sq = 0; sq < nseq; ++sq) {
      int kv, j;
      if (sq == 0) { kv = 0; j = 0; }
      else if (sq == nseq - 1) { kv = 1; j = ntiles - 1; }
      else if (sq & 1) { kv = 0; j = (sq + 1) >> 1; }
      else { kv = 1; j = (sq - 2) >> 1; }
      int row = 0;
      if (lane < loads) {
        const int tk = (kt0 + j) * kKT + lane * rows_per_load, bi = tk / p.block_size;
        const int blk = max(0, bt[bi < nblk_valid ? bi : 0]);
        row = (blk * 2 + kv) * p.block_size + tk % p.block_size;
      }
      if (!mbar_wait_warp(&bars->kv_empty[sl], ph, p.status)) break;
      if (lane == 0) mbar_expect_tx(&bars->kv_full[sl], kSlotBytes);
      __syncwarp();
      if (lane < loads) {
        uint8_t* dst = sKV + sl * kSlotBytes + lane * rows_per_load * 128;
#pragma unroll
        for (int dh = 0; dh < kDH; ++dh) tma_load_3d(dst + dh * kKVHalf, &tmKV, &bars->kv_full[sl], dh * 64, hkv, row);
      }
      __syncwarp();
      if (++sl == kRing) { sl = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_qk = umma_idesc_bf16(kQT, kKT, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(kQT, D, 0, 1);  // B (V) is MN-major
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = mbar_wait_warp(&bars->q_full, 0, p.status);
    const uint32_t q_addr = smem_u32(sQ), p_addr = smem_u32(sP);
    for (int j = 0; j <= ntiles && ok; ++j) {
      if (j < ntiles) {
        const int it = j == 0 ? 0 : 2 * j - 1, sl = it % kRing, sb = j & 1;   // K(j) in load order
        if (!(ok = mbar_wait_warp(&bars->kv_full[sl], (it / kRing) & 1, p.status))) break;
        if (!(ok = mbar_wait_warp(&bars->s_empty[sb], ((j >> 1) & 1) ^ 1, p.status))) break;
        tc_fence_after_sync();
        const uint32_t k_addr = smem_u32(sKV + sl * kSlotBytes);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            umma_bf16_ss(tm + sb * kKT,
                         umma_desc_k_sw128(q_addr + (kk / 4) * kQHalf + (kk % 4) * 32, 1024),
                         umma_desc_k_sw128(k_addr + (kk / 4) * kKVHalf + (kk % 4) * 32, 1024),
                         idesc_qk, kk != 0);
          }
          umma_commit(&bars->kv_empty[sl]);
          umma_commit(&bars->s_full[sb]);
        }
        __syncwarp();
      }
      if (j >= 1) {
        const int i = j - 1;
        const int it = i == ntiles - 1 ? 2 * ntiles - 1 : 2 * i + 2, sl = it % kRing;       // V(i)
        if (!(ok = mbar_wait_warp(&bars->kv_full[sl], (it / kRing) & 1, p.status))) break;
        if (!(ok = mbar_wait_warp(&bars->p_full, i & 1, p.status))) break;
        tc_fence_after_sync();
        const uint32_t v_addr = smem_u32(sKV + sl * kSlotBytes);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kKT / 16; ++kk) {
            // V: MN-major; 64-dim blocks are kKVHalf apart, 8-token groups 1024 B apart,
            // 16 tokens per instruction = 2048 B.
            umma_bf16_ss(tm + 128, umma_desc_k_sw128(p_addr + kk * 32, 1024),
                         umma_desc_mn_sw128(v_addr + kk * 2048, kKVHalf, 1024), idesc_pv, (i | kk) != 0);
          }
          umma_commit(&bars->kv_empty[sl]);
          umma_commit(&bars->o_full);     // before p_empty: whoever sees p_empty has this arrival too
          umma_commit(&bars->p_empty);
        }
        __syncwarp();
      }
    }
  } else {
    // ---------------- softmax + output: one thread per query row ----------------
    const int quarter = warp & 3;
    const int part = (warp - 2) >> 2;               // which half of P / O this thread owns
    const int r = quarter * 32 + lane;              // row inside the tile
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const int q_pos = ctx_off + q0 + r;             // absolute position of this query row
    const int lo = (p.window > 0) ? (q_pos - p.window + 1) : (p.window < 0 ? (q_pos / -p.window) * -p.window : 0);
    const int hi = min(p.causal ? q_pos : (seq_len - 1), seq_len - 1);
    const float sc = p.scale_log2;
    const bool cap = p.softcap2 > 0.f;
    // m: reference maximum of the row in the scaled log2 domain. It is raised lazily: only when a
    // tile exceeds it by more than 2^8, so P stays below 256 and the rescale of O is rare. O is
    // accumulated by the tensor pipe in TMEM across tiles; a raise rescales this thread's row of
    // O in place (TMEM lane == query row, so no other thread is involved).
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    uint8_t* prow = sP + r * 128;
    for (int j = 0; j < ntiles && ok; ++j) {
      const int sb = j & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full[sb], (j >> 1) & 1, p.status));
      if (!ok) break;
      tc_fence_after_sync();
      const int kbase = (kt0 + j) * kKT;
      const uint32_t s_addr = tmem_s0 + sb * kKT + lane_off;
      const bool need_mask = (kbase + kKT - 1 > hi) || (kbase < lo);
      uint32_t s0[32], s1[32];
      tmem_ld_32x32b_x32(s_addr, s0);
      tmem_ld_32x32b_x32(s_addr + 32, s1);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->s_empty[sb]);   // S is in registers now
      // scaled scores (log2 domain), soft-cap, mask
      if (cap || need_mask) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          float a = __uint_as_float(s0[i]) * sc, b = __uint_as_float(s1[i]) * sc;
          if (cap) {
            a = p.softcap2 * tanhf(a / p.softcap2);
            b = p.softcap2 * tanhf(b / p.softcap2);
          }
          const int ka = kbase + i, kb = kbase + 32 + i;
          if (ka > hi || ka < lo) a = -INFINITY;
          if (kb > hi || kb < lo) b = -INFINITY;
          s0[i] = __float_as_uint(a);
          s1[i] = __float_as_uint(b);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          s0[i] = __float_as_uint(__uint_as_float(s0[i]) * sc);
          s1[i] = __float_as_uint(__uint_as_float(s1[i]) * sc);
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        mx0 = fmaxf(mx0, __uint_as_float(s0[i]));
        mx1 = fmaxf(mx1, __uint_as_float(s1[i]));
      }
      const float tile_max = fmaxf(mx0, mx1);
      float alpha = 1.f;
      bool rescale = false;
      if (tile_max > m + 8.f) {          // also the first finite tile: m == -inf
        if (m != -INFINITY) {
          alpha = ex2_fast(m - tile_max);
          rescale = j > 0;
        }
        m = tile_max;
      }
      const float m_use = (m == -INFINITY) ? 0.f : m;
      // PV of tile j-1 has completed: the P buffer is free and O holds every product so far
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->p_empty, (j & 1) ^ 1, p.status));
      if (!ok) break;
      if (__any_sync(0xffffffffu, rescale)) {
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < kDO / 32; ++c) {
          uint32_t rr[32];
          tmem_ld_32x32b_x32(tmem_o + lane_off + part * kDO + c * 32, rr);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) rr[i] = __float_as_uint(__uint_as_float(rr[i]) * alpha);
          tmem_st_32x32b_x32(tmem_o + lane_off + part * kDO + c * 32, rr);
        }
        tmem_st_wait();
      }
      float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {     // 8 chunks of 8 columns = 16 bytes each
        uint32_t pk[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = (c & 3) * 8 + e * 2;
          const float x0 = __uint_as_float(c < 4 ? s0[i] : s1[i]);
          const float x1 = __uint_as_float(c < 4 ? s0[i + 1] : s1[i + 1]);
          const float p0 = ex2_fast(x0 - m_use), p1 = ex2_fast(x1 - m_use);
          rs0 += p0;
          rs1 += p1;
          pk[e] = pack_bf16x2(p0, p1);
        }
        if (kSplit == 1 || (c >> 2) == part)
          *reinterpret_cast<uint4*>(prow + ((c ^ (r & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
      l = l * alpha + (rs0 + rs1);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full);
    }
    if (ok && ntiles > 0) {
      // o_full completes once per PV; p_empty of the last iteration showed PV(ntiles-2) complete,
      // so this parity wait can only be satisfied by the last product
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_full, (ntiles - 1) & 1, p.status));
      if (ok) tc_fence_after_sync();
    }
    if (ok) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + (size_t)(q_begin + q0 + r) * p.ldo + h * D + part * kDO;
#pragma unroll
      for (int c = 0; c < kDO / 32; ++c) {
        uint32_t rr[32];
        if (ntiles > 0) {
          tmem_ld_32x32b_x32(tmem_o + lane_off + part * kDO + c * 32, rr);   // (whole warp)
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) rr[i] = 0;
        }
        if (r < rows) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(rr[i + 0]) * inv, __uint_as_float(rr[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(rr[i + 2]) * inv, __uint_as_float(rr[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(rr[i + 4]) * inv, __uint_as_float(rr[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(rr[i + 6]) * inv, __uint_as_float(rr[i + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + i) = w;
          }
        }
      }
    }
    if (ok && r < rows) {
      if (p.lse && part == 0) {
        const float ln2 = 0.6931471805599453f;
        p.lse[(size_t)(q_begin + q0 + r) * p.Hq + h] = l > 0.f ? (m + log2f(l)) * ln2 : -INFINITY;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
}

// ---------------------------------------------------------------------------------------
// Two query heads of one kv head per CTA (head_dim 128): 2 x 128 query rows over 128-key tiles. K and V are staged once for
// both heads (half the L2 traffic of a CTA per head), and while the softmax of one head runs, the tensor pipe works on the
// other. P goes back to tensor memory over its own scores (the A operand of P V), so that shared memory holds nothing but
// Q and a ring of four K / V tiles.
//
// Measured against one head a CTA, 64-key tiles and P in shared memory (32 query / 8 kv heads, TFLOP/s of causal work):
// 4096 tokens 656 -> 1099, 8192 -> 1268, 7309 after 8192 cached -> 1263, 8 x 1000 496 -> 611. Shorter prompts, whose time
// is a CTA's start and end, stay with one head a CTA (b200_attn_prefill_keys).
//
// A tile of two heads is 32 MMAs of 64 cycles and 128 exponentials a row, 2048 cycles of the tensor pipe and as many of the
// special-function units; it takes 3500, as each head's chain S -> softmax -> P V -> S covers the other's only in part. What
// shortens the chain: S of the next tile is issued right behind P V, over P, which the tensor pipe (it takes one thread's
// instructions in their order) has read by then (984 -> 1207 at 8192 tokens, with pairs of floats in the softmax); P V starts on
// the first half of the keys (-> 1268; three quarters 1249). Order of issue, for tile j and both heads t:
//   P(t, j) written and V(j) there   ->  O(t) += P(t, j) V(j), then, with K(j+1) there, S(t) = Q(t) K(j+1)^T
//
// Tensor memory (512 columns): S0 | S1 | O0 | O1; P(t) is the first 64 columns of S(t).
// Warp roles (320 threads): warp 0 TMA, warp 1 MMA + TMEM owner, warps 2..5 / 6..9 softmax and output of head 0 / 1, one
// thread per query row.
// ---------------------------------------------------------------------------------------
static constexpr int kPT = 128;        // keys of a tile
static constexpr int kPRing = 4;
static constexpr int kPQBytes = 2 * 16384, kPSlotBytes = 2 * 16384;      // one head's Q, one K or V tile: two 64-dim halves
static constexpr int kPSmem = 2 * kPQBytes + kPRing * kPSlotBytes + 1024;

struct alignas(8) PairBars {
  uint64_t q_full, kv_full[kPRing], kv_empty[kPRing], s_full[2], p_first[2], p_full[2], pv_done[2];
  uint32_t tmem_base;
};

__global__ void __launch_bounds__(320, 1)
    attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ PairBars bars;
  uint8_t* sQ = smem;
  uint8_t* sKV = sQ + 2 * kPQBytes;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&bars.q_full, 1);
    for (int i = 0; i < kPRing; ++i) {
      mbar_init(&bars.kv_full[i], 1);
      mbar_init(&bars.kv_empty[i], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bars.s_full[t], 1);
      mbar_init(&bars.p_first[t], 4);
      mbar_init(&bars.p_full[t], 4);
      mbar_init(&bars.pv_done[t], 1);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars.tmem_base;
  pdl_wait();
  pdl_launch_dependents();
  const int tile = gridDim.y - 1 - blockIdx.y;                 // later tiles of a prompt see more keys: they start first
  const int h0 = blockIdx.x * 2, hkv = h0 / (p.Hq / p.Hkv);
  const int req = p.tile_req[tile], q0 = p.tile_q0[tile];
  const int q_begin = p.q_start[req], q_len = p.q_start[req + 1] - q_begin;
  const int seq_len = p.seq_lens[req];
  const int ctx_off = seq_len - q_len;
  const int rows = min(kQT, q_len - q0);
  const int last_pos = p.causal ? (ctx_off + q0 + rows - 1) : (seq_len - 1);
  int first_pos = 0;
  if (p.window > 0) first_pos = max(0, ctx_off + q0 - p.window + 1);
  else if (p.window < 0) first_pos = ((ctx_off + q0) / -p.window) * -p.window;
  const int kt0 = first_pos / kPT;
  const int ntiles = last_pos / kPT + 1 - kt0;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmKV);
      mbar_expect_tx(&bars.q_full, 2 * kPQBytes);
      for (int i = 0; i < 4; ++i) tma_load_2d(sQ + i * 16384, &tmQ, &bars.q_full, h0 * 128 + i * 64, q_begin + q0);
    }
    const int32_t* bt = p.block_table + (size_t)req * p.max_blocks;
    const int nblk = (seq_len + p.block_size - 1) / p.block_size;
    const int per = min(p.block_size, kPT), loads = kPT / per;   // pages of a tile (at most 16): a lane each
    for (int sq = 0; sq < 2 * ntiles; ++sq) {                    // K0 V0 K1 V1 ...
      const int sl = sq % kPRing;
      int row = 0;
      if (lane < loads) {
        const int tk = (kt0 + (sq >> 1)) * kPT + lane * per, bi = tk / p.block_size;
        const int blk = max(0, bt[bi < nblk ? bi : 0]);
        row = (blk * 2 + (sq & 1)) * p.block_size + tk % p.block_size;
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&bars.kv_empty[sl], ((sq / kPRing) & 1) ^ 1, p.status))) break;
      if (lane == 0) mbar_expect_tx(&bars.kv_full[sl], kPSlotBytes);
      __syncwarp();
      if (lane < loads) {
        uint8_t* dst = sKV + sl * kPSlotBytes + lane * per * 128;
        tma_load_3d(dst, &tmKV, &bars.kv_full[sl], 0, hkv, row);
        tma_load_3d(dst + 16384, &tmKV, &bars.kv_full[sl], 64, hkv, row);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_qk = umma_idesc_bf16(kQT, kPT, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(kQT, 128, 0, 1);      // B (V) is MN-major
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), q_addr = smem_u32(sQ);
    const auto qk = [&](int t, int n) {           // S(t) = Q(t) K(n)^T
      const int sl = (2 * n) % kPRing;
      const uint32_t k_addr = smem_u32(sKV + sl * kPSlotBytes);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_bf16_ss(tm + t * 128, umma_desc_k_sw128(q_addr + t * kPQBytes + (kk / 4) * 16384 + (kk % 4) * 32, 1024),
                       umma_desc_k_sw128(k_addr + (kk / 4) * 16384 + (kk % 4) * 32, 1024), idesc_qk, kk != 0);
        umma_commit(&bars.s_full[t]);
        if (t == 1) umma_commit(&bars.kv_empty[sl]);
      }
      __syncwarp();
    };
    bool ok = mbar_wait_warp(&bars.q_full, 0, p.status) && mbar_wait_warp(&bars.kv_full[0], 0, p.status);
    if (ok && ntiles > 0) {
      tc_fence_after_sync();
      qk(0, 0);
      qk(1, 0);
    }
    for (int j = 0; j < ntiles && ok; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int sv = 2 * j + 1, sk = 2 * j + 2, sl = sv % kPRing;
        if (t == 0 && !(ok = mbar_wait_warp(&bars.kv_full[sl], (sv / kPRing) & 1, p.status))) break;
        const uint64_t vd = umma_desc_mn_sw128(smem_u32(sKV + sl * kPSlotBytes), 16384, 1024);
        if (!(ok = mbar_wait_warp(&bars.p_first[t], j & 1, p.status))) break;
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kPT / 32; ++kk)
            umma_bf16_ts(tm + 256 + t * 128, tm + t * 128 + kk * 8, vd + kk * (2048 >> 4), idesc_pv, (j | kk) != 0);
        }
        __syncwarp();
        if (!(ok = mbar_wait_warp(&bars.p_full[t], j & 1, p.status))) break;
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int kk = kPT / 32; kk < kPT / 16; ++kk)
            umma_bf16_ts(tm + 256 + t * 128, tm + t * 128 + kk * 8, vd + kk * (2048 >> 4), idesc_pv, 1);
          if (t == 1) umma_commit(&bars.kv_empty[sl]);
          if (j == ntiles - 1) umma_commit(&bars.pv_done[t]);
        }
        __syncwarp();
        if (j + 1 < ntiles) {
          if (t == 0) {
            if (!(ok = mbar_wait_warp(&bars.kv_full[sk % kPRing], (sk / kPRing) & 1, p.status))) break;
            tc_fence_after_sync();
          }
          qk(t, j + 1);
        }
      }
    }
  } else {
    const int t = (warp - 2) >> 2;
    const int quarter = warp & 3, r = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr = tmem + t * 128 + lane_off, o_addr = tmem + 256 + t * 128 + lane_off;
    const int q_pos = ctx_off + q0 + r;
    const int lo = (p.window > 0) ? (q_pos - p.window + 1) : (p.window < 0 ? (q_pos / -p.window) * -p.window : 0);
    const int hi = min(p.causal ? q_pos : (seq_len - 1), seq_len - 1);
    const float sc = p.scale_log2;                 // > 0
    // m: reference maximum of the row in the scaled log2 domain, raised lazily (by more than 2^8), so that O, which the
    // tensor pipe accumulates, is rescaled rarely; P stays below 256
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < ntiles; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.s_full[t], j & 1, p.status));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t s[kPT];
#pragma unroll
      for (int c = 0; c < kPT / 32; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, s + c * 32);
      tmem_ld_wait();
      const int kbase = (kt0 + j) * kPT;
      if (kbase + kPT - 1 > hi || kbase < lo) {
#pragma unroll
        for (int i = 0; i < kPT; ++i)
          if (kbase + i > hi || kbase + i < lo) s[i] = 0xff800000u;       // -inf
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < kPT; i += 4)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], __uint_as_float(s[i + e]));
      const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc;
      float alpha = 1.f;
      bool rescale = false;
      if (tile_max > m + 8.f) {          // also the first finite tile: m == -inf
        if (m != -INFINITY) {
          alpha = ex2_fast(m - tile_max);
          rescale = j > 0;
        }
        m = tile_max;
      }
      const float m_use = (m == -INFINITY) ? 0.f : m;
      // O is at rest: S(j) is issued right behind P V(j - 1), by the same elected lane, and a commit covers all that its thread has issued
      // before. Whoever moves the commit of s_full, or gives the two products to different threads, has to wait for P V(j - 1) here.
      if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll 1
        for (int c = 0; c < 8; ++c) {
          uint32_t rr[16];
          tmem_ld_32x32b_x16(o_addr + c * 16, rr);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) rr[i] = __float_as_uint(__uint_as_float(rr[i]) * alpha);
          tmem_st_32x32b_x16(o_addr + c * 16, rr);
        }
      }
      // (two values an instruction: scale and offset, and the sums)
      const uint64_t sc2 = pack_f32x2(sc, sc), off2 = pack_f32x2(-m_use, -m_use);
      uint64_t sum2[2] = {0, 0};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float a, b;
          unpack_f32x2(fma_f32x2(pack_b32x2(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]), sc2, off2), a, b);
          a = ex2_fast(a);
          b = ex2_fast(b);
          sum2[i & 1] = add_f32x2(sum2[i & 1], pack_f32x2(a, b));
          pk[i] = pack_bf16x2(a, b);
        }
        tmem_st_32x32b_x16(s_addr + c * 16, pk);
        if (c == 1) {                  // P V of the first half of the keys may start
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.p_first[t]);
        }
      }
      float sum[4];
      unpack_f32x2(sum2[0], sum[0], sum[1]);
      unpack_f32x2(sum2[1], sum[2], sum[3]);
      l = l * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.p_full[t]);
    }
    // every P V before the last is complete (its successor's S has been seen)
    if (ok && ntiles > 0) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars.pv_done[t], 0, p.status));
      if (ok) tc_fence_after_sync();
    }
    if (ok) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + (size_t)(q_begin + q0 + r) * p.ldo + (h0 + t) * 128;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t rr[32];
        if (ntiles > 0) {
          tmem_ld_32x32b_x32(o_addr + c * 32, rr);   // (whole warp)
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) rr[i] = 0;
        }
        if (r < rows) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(rr[i + 0]) * inv, __uint_as_float(rr[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(rr[i + 2]) * inv, __uint_as_float(rr[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(rr[i + 4]) * inv, __uint_as_float(rr[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(rr[i + 6]) * inv, __uint_as_float(rr[i + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + i) = w;
          }
        }
      }
      if (r < rows && p.lse) {
        const float ln2 = 0.6931471805599453f;
        p.lse[(size_t)(q_begin + q0 + r) * p.Hq + h0 + t] = l > 0.f ? (m + log2f(l)) * ln2 : -INFINITY;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

struct KvMapKey {
  const void* p;
  uint64_t rows;
  int hkv, d, box_rows;
  bool operator==(const KvMapKey& o) const {
    return p == o.p && rows == o.rows && hkv == o.hkv && d == o.d && box_rows == o.box_rows;
  }
};
struct KvMapKeyHash {
  size_t operator()(const KvMapKey& k) const {
    return reinterpret_cast<size_t>(k.p) ^ (k.rows * 0x9e3779b97f4a7c15ull) ^
           ((size_t)k.hkv << 40) ^ ((size_t)k.d << 20) ^ (size_t)k.box_rows;
  }
};

template <int D>
static int launch_prefill(const CUtensorMap& tmQ, const CUtensorMap& tmKV, const PrefillParams& p,
                          dim3 grid, cudaStream_t stream) {
  constexpr int kDH = D / 64;
  constexpr size_t smem = (size_t)kDH * 16384 + (size_t)kRing * kDH * 8192 + 16384 + 1024 +
                          sizeof(PrefillBars);
  static PerDeviceOnce attr_once;
  if (attr_once.first()) {
    cudaFuncSetAttribute(attn_prefill_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
  }
  return launch_pdl(attn_prefill_kernel<D>, grid, dim3(64 + 128 * (D > 128 ? 2 : 1)), smem, stream, tmQ, tmKV, p) == cudaSuccess ? 0 : -2;
}

}  // namespace b200

using namespace b200;


extern "C" int b200_attn_prefill(const void* q, int ldq, void* out, int ldo, void* lse,
                                 const void* kv_cache, int64_t num_blocks, int block_size, int Hq,
                                 int Hkv, int D, const void* block_table, int max_blocks,
                                 const void* seq_lens, const void* q_start, const void* tile_req,
                                 const void* tile_q0, int num_tiles, int total_q, float scale,
                                 float softcap, int window, int causal, cudaStream_t stream) {
  return b200_attn_prefill_keys(q, ldq, out, ldo, lse, kv_cache, num_blocks, block_size, Hq, Hkv, D, block_table, max_blocks,
                                seq_lens, q_start, tile_req, tile_q0, num_tiles, total_q, 0, scale, softcap, window, causal,
                                stream);
}

// The same; tile_keys, the sum over the tiles of the positions up to a tile's last row, only chooses between the kernels.
extern "C" int b200_attn_prefill_keys(const void* q, int ldq, void* out, int ldo, void* lse,
                                      const void* kv_cache, int64_t num_blocks, int block_size, int Hq,
                                      int Hkv, int D, const void* block_table, int max_blocks,
                                      const void* seq_lens, const void* q_start, const void* tile_req,
                                      const void* tile_q0, int num_tiles, int total_q, long long tile_keys, float scale,
                                      float softcap, int window, int causal, cudaStream_t stream) {
  if (num_tiles <= 0) return 0;
  if (D != 64 && D != 128 && D != 256) return -1;
  if (block_size < 8 || (block_size & 7) || (block_size < kKT && kKT % block_size) ||
      (block_size > kKT && block_size % kKT))
    return -1;
  if ((ldq & 7) || (ldo & 7) || Hq % Hkv) return -1;
  static std::mutex mu;
  static std::unordered_map<KvMapKey, CUtensorMap, KvMapKeyHash> kv_cache_maps;
  CUtensorMap tmQ, tmKV;
  if (!encode_tmap_2d(&tmQ, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)total_q,
                      (uint64_t)Hq * D, (uint64_t)ldq, kQT, 64, CU_TENSOR_MAP_SWIZZLE_128B))
    return -3;
  // Pairs of heads need an even group, 128-dim heads, no soft-cap (it is applied to the scores one by one) and pages
  // that divide a tile or are whole tiles, and tiles that the grid's second dimension holds.
  // They pay where a CTA sees keys enough: the start and the end of a CTA that has an SM to itself are in the open, and of 128
  // keys a tile more are masked. About 250 keys a tile on average are the line, or 96 where the grid is a single wave, and so
  // is more than half a wave: two heads a CTA leave SMs idle that one head a CTA has work for. A window or chunk shorter than
  // 1024 ends at both sides within a tile. us, one / two heads a CTA, 32 query heads:
  //   120 x 64 tokens 78 / 109, 30 x 128 33 / 37, 60 x 275 (220 keys) 189 / 201, 25 x 300 (243) 86 / 90, 30 x 330 108 / 107,
  //   30 x 400 (292) 150 / 148, 16 x 512 93 / 86, 8 x 1000 132 / 107, 60 x 60 after 2000 317 / 257; one wave: 8 x 40 and 8 x 100
  //   within 3 %, 1 x 700 18.8 / 17.2; windows, when the line was laid: 8192 tokens, window 256 106 / 112, 512 144 / 144,
  //   1024 218 / 201
  if (tile_keys <= 0) {       // not known: half of a request's last tile is empty on average, and nothing came before
    const long long empty = (long long)num_tiles * kQT - total_q, reqs = empty > kQT / 2 ? empty / (kQT / 2) : 1;
    tile_keys = num_tiles * (total_q / reqs + kQT) / 2;
  }
  const long long ctas = (long long)num_tiles * (Hq / 2), sms = b200_num_sms();
  const bool pair = D == 128 && (Hq / Hkv) % 2 == 0 && softcap == 0.f && scale > 0.f &&
                    (block_size <= kPT ? kPT % block_size == 0 : block_size % kPT == 0) &&
                    (window == 0 || window >= 1024 || window <= -1024) && num_tiles <= 65535 && 2 * ctas > sms &&
                    tile_keys >= (ctas <= sms ? 96 : 250) * (long long)num_tiles;
  const int most = pair ? kPT : kKT;
  const int box_rows = block_size < most ? block_size : most;
  const uint64_t rows = (uint64_t)num_blocks * 2 * block_size;
  {
    KvMapKey key{kv_cache, rows, Hkv, D, box_rows};
    std::lock_guard<std::mutex> lock(mu);
    auto it = kv_cache_maps.find(key);
    if (it == kv_cache_maps.end()) {
      if (kv_cache_maps.size() > 4096) kv_cache_maps.clear();   // scratch caches come and go
      CUtensorMap m;
      if (!encode_tmap_3d(&m, kv_cache, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)D,
                          (uint64_t)Hkv, rows, (uint64_t)D * 2, (uint64_t)Hkv * D * 2, 64, 1,
                          (uint32_t)box_rows, CU_TENSOR_MAP_SWIZZLE_128B))
        return -3;
      it = kv_cache_maps.emplace(key, m).first;
    }
    tmKV = it->second;
  }
  PrefillParams p;
  p.out = (__nv_bfloat16*)out; p.ldo = ldo; p.lse = (float*)lse;
  p.block_table = (const int32_t*)block_table; p.max_blocks = max_blocks;
  p.seq_lens = (const int32_t*)seq_lens; p.q_start = (const int32_t*)q_start;
  p.tile_req = (const int32_t*)tile_req; p.tile_q0 = (const int32_t*)tile_q0;
  p.Hq = Hq; p.Hkv = Hkv; p.block_size = block_size;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.softcap2 = softcap * 1.4426950408889634f;
  p.window = window; p.causal = causal;
  p.status = device_status_word();
  if (pair) {
    static PerDeviceOnce attr_once;
    if (attr_once.first())
      cudaFuncSetAttribute(attn_prefill_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPSmem);
    return launch_pdl(attn_prefill_pair_kernel, dim3(Hq / 2, num_tiles), dim3(320), kPSmem, stream, tmQ, tmKV, p) == cudaSuccess
               ? 0 : -2;
  }
  dim3 grid(num_tiles, Hq);
  if (D == 256) return launch_prefill<256>(tmQ, tmKV, p, grid, stream);
  return D == 128 ? launch_prefill<128>(tmQ, tmKV, p, grid, stream)
                  : launch_prefill<64>(tmQ, tmKV, p, grid, stream);
}
