// Mixture-of-experts kernels: router top-k, expert sort (device-side counts, no host sync),
// grouped expert GEMM on tcgen05, weighted combine (optionally scattered to the row owners
// of a tensor-parallel group, i.e. combine + reduce-scatter in one pass).
//
// Grouped GEMM form: for each expert the weight tile is the 128-row MMA operand and the
// tokens routed to that expert are the N operand (up to 256 per chunk), so small per-expert
// batches (decode) stream every expert weight exactly once and large ones (prefill) still
// run full 128 x 256 tiles. Work items (expert, token chunk) are listed on the device.
//
// Reference kernels replaced: src/vt/cuda/cuda_moe.cu:62 (MoeRouterTopKKernel), :197
// (MoeRouterGroupedTopKKernel), :406/:484 (MoeCombine[Gate]Kernel), :547 (MoeSiluMulKernel);
// cuda_matmul_nvfp4.cu:631-676 (hist / offsets / scatter / tile map), :923-1165 (bf16
// grouped GEMM naive / split-K / wmma variants).
#include <float.h>

#include <mutex>
#include <unordered_map>

#include "api.h"
#include "sm100.cuh"

namespace b200 {

// --------------------------------------------------------------------------- router top-k
// One block per token. scoring: 0 softmax, 1 sigmoid. Grouped selection (n_group > 1): the
// experts are split into n_group groups, a group's score is the sum of its group_best (1 or 2) best
// (bias-corrected) scores, only the topk_group best groups stay eligible. Selection uses
// score + bias, the returned weight is the unbiased score. Ties break to the lowest index.
__global__ void __launch_bounds__(256)
    moe_router_topk_kernel(const float* __restrict__ logits, int ld, int E, int k, int renorm,
                           int scoring, const float* __restrict__ e_bias, int n_group,
                           int topk_group, int group_best, float routed_scale, int32_t* topk_ids, float* topk_w) {
  extern __shared__ float sh[];   // E scores, E selection scores
  float* score = sh;
  float* sel = sh + E;
  __shared__ float red[32];
  __shared__ int redi[32];
  const int t = blockIdx.x;
  const float* x = logits + (size_t)t * ld;
  if (scoring == 0) {
    float mx = -FLT_MAX;
    for (int i = threadIdx.x; i < E; i += blockDim.x) mx = fmaxf(mx, x[i]);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = -FLT_MAX;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmaxf(mx, red[w]);
    __syncthreads();
    float s = 0.f;
    for (int i = threadIdx.x; i < E; i += blockDim.x) {
      const float e = expf(x[i] - mx);
      score[i] = e;
      s += e;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    const float inv = 1.f / s;
    for (int i = threadIdx.x; i < E; i += blockDim.x) score[i] *= inv;
  } else {
    for (int i = threadIdx.x; i < E; i += blockDim.x) score[i] = 1.f / (1.f + expf(-x[i]));
  }
  __syncthreads();
  // plain sigmoid scores are ranked by their logits: the same order, without the ties that fp32
  // scores near 1 round to
  const bool by_logit = scoring == 1 && !e_bias && n_group <= 1;
  for (int i = threadIdx.x; i < E; i += blockDim.x)
    sel[i] = by_logit ? x[i] : score[i] + (e_bias ? e_bias[i] : 0.f);
  __syncthreads();
  if (n_group > 1 && topk_group < n_group) {
    // thread g scores group g (n_group is small), thread 0 masks the losers
    __shared__ float gscore[64];
    const int per = E / n_group;
    if ((int)threadIdx.x < n_group) {
      float b0 = -FLT_MAX, b1 = -FLT_MAX;
      for (int i = 0; i < per; ++i) {
        const float v = sel[threadIdx.x * per + i];
        if (v > b0) { b1 = b0; b0 = v; } else if (v > b1) { b1 = v; }
      }
      gscore[threadIdx.x] = group_best == 2 ? b0 + b1 : b0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int pick = 0; pick < n_group - topk_group; ++pick) {
        int worst = -1;
        float wv = FLT_MAX;
        for (int g = n_group - 1; g >= 0; --g)   // ties: drop the highest index first
          if (gscore[g] != FLT_MAX && gscore[g] < wv) { wv = gscore[g]; worst = g; }
        if (worst < 0) break;
        gscore[worst] = FLT_MAX;
        for (int i = 0; i < per; ++i) sel[worst * per + i] = -FLT_MAX;
      }
    }
    __syncthreads();
  }
  float wsum = 0.f;
  for (int j = 0; j < k; ++j) {
    float bv = -FLT_MAX;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < E; i += blockDim.x) {
      const float v = sel[i];
      if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = bv; redi[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
        if (red[w] > bv || (red[w] == bv && redi[w] < bi)) { bv = red[w]; bi = redi[w]; }
      if (bi >= E) bi = 0;
      topk_ids[(size_t)t * k + j] = bi;
      topk_w[(size_t)t * k + j] = score[bi];
      sel[bi] = -FLT_MAX;
      red[0] = score[bi];
    }
    __syncthreads();
    wsum += red[0];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float denom = (renorm && wsum > 0.f) ? wsum : 1.f;
    for (int j = 0; j < k; ++j) topk_w[(size_t)t * k + j] = topk_w[(size_t)t * k + j] / denom * routed_scale;
  }
}

// The same for ungrouped routers of up to 256 experts: one warp per token, E / 32 scores a lane, no barrier (a block
// needed two to three a choice: 9.7 us for 3 tokens, 128 experts, k = 8).
template <int PER>
__global__ void __launch_bounds__(128)
    moe_router_warp_kernel(const float* __restrict__ logits, int ld, int T, int E, int k, int renorm, int scoring,
                           const float* __restrict__ e_bias, float routed_scale, int32_t* topk_ids, float* topk_w) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= T) return;
  const float* x = logits + (size_t)t * ld;
  float v[PER], score[PER], sel[PER];
  float mx = -FLT_MAX;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    v[i] = lane + 32 * i < E ? x[lane + 32 * i] : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
  if (scoring == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      score[i] = lane + 32 * i < E ? expf(v[i] - mx) : 0.f;
      s += score[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
#pragma unroll
    for (int i = 0; i < PER; ++i) score[i] *= inv;
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i) score[i] = 1.f / (1.f + expf(-v[i]));
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    // plain sigmoid scores are ranked by their logits: no ties of fp32 scores near 1
    sel[i] = e >= E ? -FLT_MAX : scoring == 1 && !e_bias ? v[i] : score[i] + (e_bias ? e_bias[e] : 0.f);
  }
  float wsum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int j = 0; j < k; ++j) {
    float bv = -FLT_MAX, bs = 0.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (sel[i] > bv || (sel[i] == bv && lane + 32 * i < bi)) { bv = sel[i]; bi = lane + 32 * i; bs = score[i]; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o), os = __shfl_xor_sync(0xffffffffu, bs, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; bs = os; }
    }
    if (bi >= E) {                    // nothing comparable is left (NaN logits): expert 0, as in the block kernel
      bi = 0;
      bs = __shfl_sync(0xffffffffu, score[0], 0);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i == bi) sel[i] = -FLT_MAX;
    wsum += bs;
    if (lane == (j & 31)) { my_id = bi; my_w = bs; }
    if ((j & 31) == 31 || j == k - 1) {
      const int j0 = j & ~31;
      if (j0 + lane <= j) {
        topk_ids[(size_t)t * k + j0 + lane] = my_id;
        topk_w[(size_t)t * k + j0 + lane] = my_w;
      }
    }
  }
  const float denom = (renorm && wsum > 0.f) ? wsum : 1.f;
  __syncwarp();
  for (int j = lane; j < k; j += 32) topk_w[(size_t)t * k + j] = topk_w[(size_t)t * k + j] / denom * routed_scale;
}

// ------------------------------------------------------------------------------ expert sort
// meta layout (int32): [0, E) counts | [E, 2E] offsets | [2E+1, 3E+1) cursors | 3E+1 num_chunks
__global__ void moe_hist_kernel(const int32_t* __restrict__ topk_ids, int P, int e0, int e1,
                                int32_t* meta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int e = topk_ids[i];
  if (e >= e0 && e < e1) atomicAdd(&meta[e - e0], 1);
}
__global__ void moe_offsets_kernel(int32_t* meta, int E, int chunk_rows, int32_t* chunk_expert,
                                   int32_t* chunk_row0, int32_t* chunk_n, int max_chunks) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int off = 0, nc = 0;
  for (int e = 0; e < E; ++e) {
    meta[E + e] = off;
    meta[2 * E + 1 + e] = off;
    const int c = meta[e];
    for (int r = 0; r < c && nc < max_chunks; r += chunk_rows) {
      chunk_expert[nc] = e;
      chunk_row0[nc] = off + r;
      chunk_n[nc] = min(chunk_rows, c - r);
      ++nc;
    }
    off += c;
  }
  meta[2 * E] = off;
  meta[3 * E + 1] = nc;
}
// Decode-sized batches: histogram, offsets, chunk table and scatter in ONE block (counts and
// cursors in shared memory) instead of a memset and three launches, one of them a single thread
// walking the experts. E <= 256. The order of the rows inside an expert depends on the atomics,
// which is harmless: every row's product is independent and the combine goes through pair_pos.
__global__ void __launch_bounds__(1024)
    moe_sort_small_kernel(const int32_t* __restrict__ topk_ids, int P, int k, int e0, int e1, int32_t* meta,
                          int chunk_rows, int32_t* chunk_expert, int32_t* chunk_row0, int32_t* chunk_n,
                          int max_chunks, int32_t* sorted_token, int32_t* pair_pos) {
  __shared__ int cnt[256], off[256], cbase[256], cursor[256];
  __shared__ int wsum[8], wcsum[8];
  pdl_wait();
  pdl_launch_dependents();
  const int E = e1 - e0, tid = threadIdx.x;
  if (tid < 256) cnt[tid] = 0;
  __syncthreads();
  for (int i = tid; i < P; i += blockDim.x) {
    const int e = topk_ids[i];
    if (e >= e0 && e < e1) atomicAdd(&cnt[e - e0], 1);
  }
  __syncthreads();
  if (tid < 256) {
    // exclusive scans of the counts and of the chunk counts over 256 entries: warp scan + 8 totals
    const int c = tid < E ? cnt[tid] : 0;
    const int nch = (c + chunk_rows - 1) / chunk_rows;
    int a = c, b = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ta = __shfl_up_sync(0xffffffffu, a, o), tb = __shfl_up_sync(0xffffffffu, b, o);
      if ((tid & 31) >= o) { a += ta; b += tb; }
    }
    if ((tid & 31) == 31) { wsum[tid >> 5] = a; wcsum[tid >> 5] = b; }
    off[tid] = a - c;
    cbase[tid] = b - nch;
  }
  __syncthreads();
  if (tid < 256) {
    int pa = 0, pb = 0;
    for (int w = 0; w < (tid >> 5); ++w) { pa += wsum[w]; pb += wcsum[w]; }
    off[tid] += pa;
    cbase[tid] += pb;
  }
  __syncthreads();
  if (tid < E) {
    const int c = cnt[tid], o = off[tid];
    meta[tid] = c;
    meta[E + tid] = o;
    meta[2 * E + 1 + tid] = o + c;          // where the scatter's cursor ends
    cursor[tid] = o;
    int nc = cbase[tid];
    for (int r = 0; r < c && nc < max_chunks; r += chunk_rows, ++nc) {
      chunk_expert[nc] = tid;
      chunk_row0[nc] = o + r;
      chunk_n[nc] = min(chunk_rows, c - r);
    }
    if (tid == E - 1) {
      meta[2 * E] = o + c;
      meta[3 * E + 1] = min(max_chunks, cbase[tid] + (c + chunk_rows - 1) / chunk_rows);
    }
  }
  __syncthreads();
  for (int i = tid; i < P; i += blockDim.x) {
    const int e = topk_ids[i];
    if (e >= e0 && e < e1) {
      const int pos = atomicAdd(&cursor[e - e0], 1);
      sorted_token[pos] = i / k;
      pair_pos[i] = pos;
    } else {
      pair_pos[i] = -1;
    }
  }
}
__global__ void moe_scatter_kernel(const int32_t* __restrict__ topk_ids, int P, int k, int e0,
                                   int e1, int32_t* meta, int E, int32_t* sorted_token,
                                   int32_t* pair_pos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int e = topk_ids[i];
  if (e >= e0 && e < e1) {
    const int pos = atomicAdd(&meta[2 * E + 1 + (e - e0)], 1);
    sorted_token[pos] = i / k;
    pair_pos[i] = pos;
  } else {
    pair_pos[i] = -1;
  }
}
// xs[pos, :] = x[sorted_token[pos], :] for pos < total (read from meta), rows of H bf16. PDL: may start while its predecessor runs.
template <bool PDL>
__global__ void __launch_bounds__(128)
    moe_gather_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const int32_t* sorted_token,
                      const int32_t* meta, int E, __nv_bfloat16* xs, int H) {
  if constexpr (PDL) {
    pdl_wait();
    pdl_launch_dependents();
  }
  const int pos = blockIdx.x;
  if (pos >= meta[2 * E]) return;
  const uint4* s = reinterpret_cast<const uint4*>(x + (size_t)sorted_token[pos] * ldx);
  uint4* d = reinterpret_cast<uint4*>(xs + (size_t)pos * H);
  for (int i = threadIdx.x; i < (H >> 3); i += blockDim.x) d[i] = s[i];
}

// row_w[pos] = weight of the (token, expert) pair that was sorted to pos
__global__ void moe_row_weights_kernel(const int32_t* __restrict__ pair_pos, const float* __restrict__ topk_w, int P,
                                       float* row_w) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P && pair_pos[i] >= 0) row_w[pair_pos[i]] = topk_w[i];
}

// ------------------------------------------------------------------------------ grouped GEMM
static constexpr int kGBM = 128, kGBK = 64, kGMaxStages = 8;
struct GroupedParams {
  int N, K;                 // per expert: out[rows, N] = xs[rows, K] * W_e[N, K]^T
  __nv_bfloat16* out;       // [P, N] sorted order
  const int32_t* chunk_expert;
  const int32_t* chunk_row0;
  const int32_t* chunk_n;
  const int32_t* meta;
  int E;
  int stages;
  int sub_rows;             // sorted rows of a CTA: 256, or 128 (gated): blockIdx.x = part of the chunk * column tiles + column tile
  // Gated mode (act_fuse = activation kind + 1): W_e is [gate rows (N/2) | up rows (N/2)]; a CTA
  // takes 128 gate rows and the 128 up rows of the same outputs, keeps one accumulator for each in
  // TMEM (columns [0, np) and [sub_rows, sub_rows + np)) and writes act(gate) * up to out[rows, N / 2], so the
  // merged projection never reaches memory. Both values are rounded to bf16 first, as the separate
  // activation kernel would see them.
  int act_fuse;
  B200ClampedGate clamp;    // act_fuse == 4: clamped pair, applied to the fp32 accumulators
  int act;                  // not gated: activation of the result (act_epilogue)
  int* status;
};
struct alignas(8) GroupedBars {
  uint64_t full[kGMaxStages], empty[kGMaxStages], acc_full;
  uint32_t tmem_base;
  float row_w[256];        // clamped pair: routing weights of the chunk's rows
};

// grid: (column tiles x parts of a chunk, max_chunks). A CTA whose chunk index is past the device-side count exits. Two CTAs
// share an SM (96 KB of stages and 256 TMEM columns each), so that one stores its outputs while the other multiplies; a CTA
// alone, with twice the stages and, gated, the accumulators of 256 rows, leaves the tensor pipe idle during
// its epilogue (us at 8192 tokens, gated / down: 128 experts of 768, top 8, 608 / 525 -> 492 / 349; 64 of 1408, top 6,
// 799 / 511 -> 637 / 349). Where there are too few CTAs to pair up that form stays (moe_grouped_gemm_impl).
__global__ void __launch_bounds__(192, 2)
    moe_grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmW,
                            const __grid_constant__ CUtensorMap tmX, GroupedParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  const int tiles = (int)gridDim.x * p.sub_rows >> 8, chunk = blockIdx.y, first = (int)blockIdx.x / tiles * p.sub_rows;
  if (chunk >= p.meta[3 * p.E + 1] || first >= p.chunk_n[chunk]) return;
  const int e = p.chunk_expert[chunk], row0 = p.chunk_row0[chunk] + first, rows = min(p.sub_rows, p.chunk_n[chunk] - first);
  const int np = (rows + 15) & ~15;                 // UMMA N
  constexpr int kWBytes = kGBM * kGBK * 2;
  const int kXBytes = p.sub_rows * kGBK * 2;        // TMA box: always sub_rows rows
  const bool gated = p.act_fuse != 0;
  const int half_n = p.N >> 1;                      // gated: outputs per expert
  const int kStage = kWBytes * (gated ? 2 : 1) + kXBytes;
  const int stages = p.stages;
  GroupedBars* bars = reinterpret_cast<GroupedBars*>(smem + (size_t)stages * kStage);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tn = (int)blockIdx.x % tiles;
  const int nkb = (p.K + kGBK - 1) / kGBK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&bars->full[s], 1); mbar_init(&bars->empty[s], 1); }
    mbar_init(&bars->acc_full, 1);
    mbar_fence_init();
  }
  const uint32_t tmem_cols = gated ? 2 * p.sub_rows : 256;
  if (warp == 1) { tmem_alloc(&bars->tmem_base, tmem_cols); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  const int x_off = kWBytes * (gated ? 2 : 1);
  if (warp == 0) {          // (these two warps walk their loops whole, one elected lane issues)
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
    }
    __syncwarp();
    int s = 0;
    uint32_t ph = 1;
    for (int i = 0; i < nkb; ++i) {
      if (!mbar_wait_warp(&bars->empty[s], ph, p.status)) break;
      uint8_t* wd = smem + (size_t)s * kStage;
      if (elect_one()) {
        mbar_expect_tx(&bars->full[s], kStage);
        tma_load_3d(wd, &tmW, &bars->full[s], i * kGBK, tn * kGBM, e);
        if (gated) tma_load_3d(wd + kWBytes, &tmW, &bars->full[s], i * kGBK, half_n + tn * kGBM, e);
        tma_load_2d(wd + x_off, &tmX, &bars->full[s], i * kGBK, row0);
      }
      __syncwarp();
      if (++s == stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_bf16(kGBM, np), acc = __shfl_sync(0xffffffffu, tmem_base, 0);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int i = 0; i < nkb; ++i) {
      if (!(ok = mbar_wait_warp(&bars->full[s], ph, p.status))) break;
      tc_fence_after_sync();
      const uint32_t wa = smem_u32(smem + (size_t)s * kStage);
      const uint64_t wdesc = umma_desc_k_sw128(wa, 1024), udesc = umma_desc_k_sw128(wa + kWBytes, 1024),
                     xdesc = umma_desc_k_sw128(wa + x_off, 1024);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kGBK / 16; ++kk) {
          umma_bf16_ss(acc, wdesc + 2 * kk, xdesc + 2 * kk, idesc, (i | kk) != 0);
          if (gated) umma_bf16_ss(acc + p.sub_rows, udesc + 2 * kk, xdesc + 2 * kk, idesc, (i | kk) != 0);
        }
        umma_commit(&bars->empty[s]);
      }
      __syncwarp();
      if (++s == stages) { s = 0; ph ^= 1; }
    }
    if (ok && elect_one()) umma_commit(&bars->acc_full);
    __syncwarp();
  } else if (gated) {
    const int quarter = warp & 3;
    if (p.act_fuse == 4) {
      for (int i = threadIdx.x - 64; i < 256; i += 128)
        bars->row_w[i] = p.clamp.row_w && i < rows ? p.clamp.row_w[row0 + i] : 1.f;
      asm volatile("bar.sync 1, 128;" ::: "memory");      // the four epilogue warps
    }
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, 0, p.status));
    tc_fence_after_sync();
    const int n = tn * kGBM + quarter * 32 + lane;        // output column of this thread
    const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int kind = p.act_fuse - 1;
    if (ok && kind == 3) {
      for (int c = 0; c < np / 16; ++c) {
        uint32_t g[16], u[16];
        tmem_ld_32x32b_x16(ta + c * 16, g);
        tmem_ld_32x32b_x16(ta + p.sub_rows + c * 16, u);
        tmem_ld_wait();
        if (n < half_n) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int m = c * 16 + i;
            if (m < rows) {
              const float w = bars->row_w[m];
              const float gg = fminf(__uint_as_float(g[i]) * w, p.clamp.limit);
              const float uu = fminf(fmaxf(__uint_as_float(u[i]) * w, -p.clamp.limit), p.clamp.limit);
              p.out[(size_t)(row0 + m) * half_n + n] =
                  __float2bfloat16(__fdividef(gg, 1.f + __expf(-p.clamp.alpha * gg)) * (uu + p.clamp.up_offset));
            }
          }
        }
      }
    } else if (ok) {
      for (int c = 0; c < np / 16; ++c) {
        uint32_t g[16], u[16];
        tmem_ld_32x32b_x16(ta + c * 16, g);
        tmem_ld_32x32b_x16(ta + p.sub_rows + c * 16, u);
        tmem_ld_wait();
        if (n < half_n) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int m = c * 16 + i;
            if (m < rows) {
              const float gg = __bfloat162float(__float2bfloat16(__uint_as_float(g[i])));
              const float uu = __bfloat162float(__float2bfloat16(__uint_as_float(u[i])));
              p.out[(size_t)(row0 + m) * half_n + n] = __float2bfloat16(act_of(gg, kind) * uu);
            }
          }
        }
      }
    }
  } else {
    const int quarter = warp & 3;
    bool ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_full, 0, p.status));
    tc_fence_after_sync();
    const int n = tn * kGBM + quarter * 32 + lane;
    const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16);
    if (ok) {
      for (int c = 0; c < np / 16; ++c) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(ta + c * 16, r);
        tmem_ld_wait();
        if (n < p.N) {
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
          act_epilogue<true>(v, p.act);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int m = c * 16 + i;
            if (m < rows)
              p.out[(size_t)(row0 + m) * p.N + n] = __float2bfloat16(v[i]);
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
}

// Experts of many rows: CTA pairs as in gemm_bf16_pair_kernel, a tile of 256 sorted rows (128 a CTA) x 256 weight rows, gated 128
// gate rows (staged by the first CTA) and the 128 up rows of the same outputs (by the second). Persistent: a pair takes the tiles
// pair, pair + pairs, ... of the device-side list of chunks, weight tiles inside a chunk; two accumulators let the epilogue of a tile run
// under the products of the next, which with a K of 12 k-blocks takes about as long. A chunk's missing rows up to 256
// are multiplied and not stored.
static constexpr int kPStages = 6, kPStage = 32 * 1024, kPMostChunks = 1024, kPGroup = 16;
struct GroupedPairChunk {
  int expert, row0, rows, first, group;       // first: of the group that the chunk belongs to, group: its chunks
};
struct GroupedPairParams {
  int N, K, E, max_chunks, tiles;       // tiles: of 256 weight rows (gated: 128 outputs)
  int act_fuse, act;
  __nv_bfloat16* out;
  const int32_t *chunk_expert, *chunk_row0, *chunk_n, *meta;
  int* status;
};
struct alignas(8) GroupedPairBars {
  uint64_t full[kPStages], empty[kPStages], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};

__global__ void __launch_bounds__(192, 1)
    moe_grouped_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, GroupedPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ GroupedPairBars bars;
  GroupedPairChunk* table = reinterpret_cast<GroupedPairChunk*>(smem + kPStages * kPStage);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int nkb = (p.K + kGBK - 1) / kGBK, half_n = p.N >> 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPStages; ++s) { mbar_init(&bars.full[s], 1); mbar_init(&bars.empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&bars.acc_full[b], 1); mbar_init(&bars.acc_empty[b], 8); }
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc_pair(&bars.tmem_base, 512); tmem_relinquish_pair(); }
  pdl_wait();
  const int chunks = min(p.meta[3 * p.E + 1], p.max_chunks);
  // Up to kPGroup chunks of an expert take a weight tile one after the other, so that side by side pairs share it in L2 (8 experts
  // of 14336, width 4096, 4096 tokens: a chunk at a time 1779 us)
  for (int i = threadIdx.x; i < chunks; i += 192) {
    const int e = p.chunk_expert[i];
    int first = i, end = i + 1;
    while (first > 0 && p.chunk_expert[first - 1] == e) --first;
    first += (i - first) / kPGroup * kPGroup;
    while (end < chunks && end < first + kPGroup && p.chunk_expert[end] == e) ++end;
    table[i] = GroupedPairChunk{e, p.chunk_row0[i], p.chunk_n[i], first, end - first};
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();            // the peer's barriers exist before anything signals them
  tc_fence_after_sync();
  pdl_launch_dependents();       // (not before the columns are taken: a successor that took some first would wait for this kernel's end)
  const uint32_t tmem = __shfl_sync(0xffffffffu, bars.tmem_base, 0);
  const int total = chunks * p.tiles;
  const auto tile_of = [&](int t, int& tn) {
    const GroupedPairChunk& g = table[t / p.tiles];
    const int at = t - g.first * p.tiles;
    tn = at / g.group;
    return table[g.first + at - tn * g.group];
  };

  if (warp == 0) {
    if (lane == 0) { tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX); }
    int s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int t = pair; t < total && ok; t += pairs) {
      int tn;
      const GroupedPairChunk c = tile_of(t, tn);
      const int x_row = c.row0 + rank * 128;
      const int w_row = p.act_fuse ? rank * half_n + tn * 128 : tn * 256 + rank * 128;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!(ok = mbar_wait_warp(&bars.empty[s], ph, p.status))) break;
        uint8_t* dst = smem + s * kPStage;
        const uint32_t leader_bar = mapa_u32(smem_u32(&bars.full[s]), 0);
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&bars.full[s], 2 * kPStage);
          tma_load_2d_pair(dst, &tmX, leader_bar, kb * kGBK, x_row);
          tma_load_3d_pair(dst + kPStage / 2, &tmW, leader_bar, kb * kGBK, w_row, c.expert);
        }
        __syncwarp();
        if (++s == kPStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(256, 256);
      int s = 0;
      uint32_t ph = 0, n = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += pairs, ++n) {
        const int buf = n & 1;
        if (!(ok = mbar_wait_warp(&bars.acc_empty[buf], ((n >> 1) & 1) ^ 1, p.status))) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!(ok = mbar_wait_warp(&bars.full[s], ph, p.status))) break;
          tc_fence_after_sync();
          const uint32_t a = smem_u32(smem + s * kPStage);
          const uint64_t adesc = umma_desc_k_sw128(a, 1024), bdesc = umma_desc_k_sw128(a + kPStage / 2, 1024);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_ss_pair(tmem + buf * 256, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0);
            umma_commit_pair(&bars.empty[s], 3);
            if (kb == nkb - 1) umma_commit_pair(&bars.acc_full[buf], 3);
          }
          __syncwarp();
          if (++s == kPStages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else {
    const int quarter = warp & 3, r = rank * 128 + quarter * 32 + lane;
    uint32_t n = 0;
    for (int t = pair; t < total; t += pairs, ++n) {
      const int buf = n & 1;
      int tn;
      const GroupedPairChunk c = tile_of(t, tn);
      const bool in = r < c.rows;
      const size_t row = (size_t)(c.row0 + r);
      if (!mbar_wait_warp(&bars.acc_full[buf], (n >> 1) & 1, p.status)) break;
      tc_fence_after_sync();
      const uint32_t acc = tmem + buf * 256 + ((uint32_t)(quarter * 32) << 16);
      if (p.act_fuse) {
        __nv_bfloat16* o = p.out + row * half_n + tn * 128;
        const int kind = p.act_fuse - 1;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          uint32_t g[32], u[32];
          tmem_ld_32x32b_x32(acc + q * 32, g);
          tmem_ld_32x32b_x32(acc + 128 + q * 32, u);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            if (!in || tn * 128 + q * 32 + i >= half_n) continue;
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float gg = __bfloat162float(__float2bfloat16(__uint_as_float(g[i + j])));
              v[j] = act_of(gg, kind) * __bfloat162float(__float2bfloat16(__uint_as_float(u[i + j])));
            }
            *reinterpret_cast<uint4*>(o + q * 32 + i) =
                make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
          }
        }
      } else {
        __nv_bfloat16* o = p.out + row * p.N + tn * 256;
#pragma unroll 1
        for (int q = 0; q < 8; ++q) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(acc + q * 32, v);
          tmem_ld_wait();
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]);
          act_epilogue<true>(f, p.act);
#pragma unroll
          for (int i = 0; i < 32; i += 8)
            if (in && tn * 256 + q * 32 + i < p.N)
              *reinterpret_cast<uint4*>(o + q * 32 + i) = make_uint4(pack_bf16x2(f[i], f[i + 1]), pack_bf16x2(f[i + 2], f[i + 3]),
                                                                     pack_bf16x2(f[i + 4], f[i + 5]), pack_bf16x2(f[i + 6], f[i + 7]));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bars.acc_empty[buf]), 0));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();            // neither CTA frees while the other still reads its accumulators
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

// ---------------------------------------------------------------------------------- combine
// out[t, :] = sum_j w[t, j] * y[pair_pos[t, j], :] (+ shared[t, :] * shared_scale[t]) ;
// pairs routed to experts of other ranks (pair_pos < 0) are skipped. fp32 accumulation in
// ascending j, one bf16 rounding. With `peer_recv` set the row is stored into the receive
// slot of its owner rank (combine + reduce-scatter); signalled per 32-row group.
struct CombineParams {
  const __nv_bfloat16* y;
  const int32_t* pair_pos;
  const float* topk_w;
  int k, H, T;
  const __nv_bfloat16* shared;       // optional [T, H]
  const float* shared_gate;          // optional [T] (sigmoid applied by the caller)
  __nv_bfloat16* out;                // [T, H] when not scattering
  int tp_world, tp_rank, rows_per_rank;
  __nv_bfloat16* peer_recv[8];
  uint32_t* peer_rs_flags[8];
  long long recv_parity_stride;
  int rs_flag_parity_stride;
  const uint32_t* op_counter;
};
__global__ void __launch_bounds__(256) moe_combine_kernel(CombineParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int nv = p.H >> 3;
  __nv_bfloat16* dst;
  uint32_t par = 0;
  int owner = 0;
  if (p.tp_world > 1 && p.peer_recv[0]) {
    owner = t / p.rows_per_rank;
    par = *p.op_counter & 1;
    dst = p.peer_recv[owner] + par * p.recv_parity_stride +
          ((size_t)p.tp_rank * p.rows_per_rank + (t - owner * p.rows_per_rank)) * p.H;
  } else {
    dst = p.out + (size_t)t * p.H;
  }
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int j0 = 0; j0 < p.k; j0 += 4) {          // four expert rows on the way at a time
      int pos[4];
      float w[4];
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        pos[j] = j0 + j < p.k ? p.pair_pos[(size_t)t * p.k + j0 + j] : -1;
        w[j] = j0 + j < p.k ? p.topk_w[(size_t)t * p.k + j0 + j] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (pos[j] >= 0) v[j] = *reinterpret_cast<const uint4*>(p.y + (size_t)pos[j] * p.H + i * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (pos[j] < 0) continue;
        float2 f;
        f = unpack_bf16x2(v[j].x); acc[0] += w[j] * f.x; acc[1] += w[j] * f.y;
        f = unpack_bf16x2(v[j].y); acc[2] += w[j] * f.x; acc[3] += w[j] * f.y;
        f = unpack_bf16x2(v[j].z); acc[4] += w[j] * f.x; acc[5] += w[j] * f.y;
        f = unpack_bf16x2(v[j].w); acc[6] += w[j] * f.x; acc[7] += w[j] * f.y;
      }
    }
    uint4 o;
    o.x = pack_bf16x2(acc[0], acc[1]); o.y = pack_bf16x2(acc[2], acc[3]);
    o.z = pack_bf16x2(acc[4], acc[5]); o.w = pack_bf16x2(acc[6], acc[7]);
    if (p.shared) {
      // routed sum is rounded to bf16 first, then the shared expert is added (reference order)
      const float g = p.shared_gate ? p.shared_gate[t] : 1.f;
      const uint4 s = *reinterpret_cast<const uint4*>(p.shared + (size_t)t * p.H + i * 8);
      float2 a, b;
      a = unpack_bf16x2(o.x); b = unpack_bf16x2(s.x); o.x = pack_bf16x2(a.x + g * b.x, a.y + g * b.y);
      a = unpack_bf16x2(o.y); b = unpack_bf16x2(s.y); o.y = pack_bf16x2(a.x + g * b.x, a.y + g * b.y);
      a = unpack_bf16x2(o.z); b = unpack_bf16x2(s.z); o.z = pack_bf16x2(a.x + g * b.x, a.y + g * b.y);
      a = unpack_bf16x2(o.w); b = unpack_bf16x2(s.w); o.w = pack_bf16x2(a.x + g * b.x, a.y + g * b.y);
    }
    reinterpret_cast<uint4*>(dst)[i] = o;
  }
  if (p.tp_world > 1 && p.peer_recv[0]) {
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
      // every 32-row group receives exactly 32 arrivals per source rank: the last token also
      // covers the rows its (partial) group does not have
      uint32_t inc = 1;
      if (t == p.T - 1 && (p.T & 31)) inc += 32 - (p.T & 31);
      asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(
                       p.peer_rs_flags[owner] + par * p.rs_flag_parity_stride +
                       (t - owner * p.rows_per_rank) / 32),
                   "r"(inc)
                   : "memory");
    }
  }
}

// sigmoid(x . w) per row: gate of the shared expert (Qwen3.5 / 3.6 MoE)
__global__ void __launch_bounds__(128)
    shared_gate_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const __nv_bfloat16* w, int H,
                       float* out) {
  __shared__ float red[4];
  const int t = blockIdx.x;
  float s = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    s += __bfloat162float(x[(size_t)t * ldx + i]) * __bfloat162float(w[i]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float v = red[0] + red[1] + red[2] + red[3];
    out[t] = 1.f / (1.f + expf(-v));
  }
}

}  // namespace b200

using namespace b200;
typedef __nv_bfloat16 bf16;
#define RETL return cudaGetLastError() == cudaSuccess ? 0 : -2

extern "C" {

int b200_moe_router_topk(const void* logits_f32, int ld, int T, int E, int k, int renorm,
                         int scoring, const void* e_bias, int n_group, int topk_group, int group_best,
                         float routed_scale, void* topk_ids, void* topk_w, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (k > E || n_group > 64 || (n_group > 1 && E % n_group)) return -1;
  if (n_group <= 1 && E <= 256) {
    auto kernel = E <= 64 ? moe_router_warp_kernel<2> : E <= 128 ? moe_router_warp_kernel<4> : moe_router_warp_kernel<8>;
    return launch_pdl(kernel, dim3((T + 3) / 4), dim3(128), 0, stream, (const float*)logits_f32, ld, T, E, k, renorm, scoring,
                      (const float*)e_bias, routed_scale, (int32_t*)topk_ids, (float*)topk_w) == cudaSuccess ? 0 : -2;
  }
  moe_router_topk_kernel<<<T, 256, (size_t)2 * E * sizeof(float), stream>>>(
      (const float*)logits_f32, ld, E, k, renorm, scoring, (const float*)e_bias, n_group,
      topk_group, group_best, routed_scale, (int32_t*)topk_ids, (float*)topk_w);
  RETL;
}

// Sorts the (token, expert) pairs whose expert is in [e0, e1) by expert.
// meta: int32[3*E_local + 2] (zeroed here); chunk arrays: int32[max_chunks].
int b200_moe_sort(const void* topk_ids, int T, int k, int e0, int e1, void* meta,
                  void* sorted_token, void* pair_pos, void* chunk_expert, void* chunk_row0,
                  void* chunk_n, int max_chunks, cudaStream_t stream) {
  const int P = T * k, E = e1 - e0;
  if (P <= 0) return 0;
  if (E <= 256 && P <= 16384) {
    return launch_pdl(moe_sort_small_kernel, dim3(1), dim3(1024), 0, stream, (const int32_t*)topk_ids, P, k, e0, e1,
                      (int32_t*)meta, 256, (int32_t*)chunk_expert, (int32_t*)chunk_row0, (int32_t*)chunk_n, max_chunks,
                      (int32_t*)sorted_token, (int32_t*)pair_pos) == cudaSuccess ? 0 : -2;
  }
  cudaMemsetAsync(meta, 0, (size_t)(3 * E + 2) * sizeof(int32_t), stream);
  moe_hist_kernel<<<(P + 255) / 256, 256, 0, stream>>>((const int32_t*)topk_ids, P, e0, e1,
                                                       (int32_t*)meta);
  moe_offsets_kernel<<<1, 1, 0, stream>>>((int32_t*)meta, E, 256, (int32_t*)chunk_expert,
                                          (int32_t*)chunk_row0, (int32_t*)chunk_n, max_chunks);
  moe_scatter_kernel<<<(P + 255) / 256, 256, 0, stream>>>((const int32_t*)topk_ids, P, k, e0, e1,
                                                          (int32_t*)meta, E, (int32_t*)sorted_token,
                                                          (int32_t*)pair_pos);
  RETL;
}

int b200_moe_gather(const void* x, int ldx, const void* sorted_token, const void* meta, int E,
                    void* xs, int H, int max_rows, cudaStream_t stream) {
  if (max_rows <= 0) return 0;
  // A CTA is one row, about a microsecond: over several waves of them the two instructions of an early start cost more than the
  // start gains, also where the launch is an ordinary one (us without / with them, rows of 2048: 3840 rows 4.9 / 4.8, 6400 6.6 / 7.9,
  // 16384 14.1 / 18.4; with the sort ahead, rows of 1024: 5600 rows 10.4 / 12.3; rows of 4096: 5600 14.8 / 14.6).
  if (max_rows >= 4096) {
    moe_gather_kernel<false><<<max_rows, 128, 0, stream>>>((const bf16*)x, ldx, (const int32_t*)sorted_token, (const int32_t*)meta, E,
                                                           (bf16*)xs, H);
    RETL;
  }
  return launch_pdl(moe_gather_kernel<true>, dim3(max_rows), dim3(128), 0, stream, (const bf16*)x, ldx, (const int32_t*)sorted_token,
                    (const int32_t*)meta, E, (bf16*)xs, H) == cudaSuccess ? 0 : -2;
}

// out[P, N] = grouped(xs[P, K], W[E, N, K]); xs must have at least max_rows + 256 rows allocated.
static int moe_grouped_gemm_impl(const void* xs, int max_rows, const void* W, int E, int N, int K,
                                 void* out, const void* chunk_expert, const void* chunk_row0,
                                 const void* chunk_n, const void* meta, int max_chunks, int act_fuse,
                                 cudaStream_t stream, const B200ClampedGate* clamp = nullptr, int act = 0) {
  if (max_rows <= 0) return 0;
  if ((K & 7) || (N & 7) || act < 0 || act > 4) return -1;
  if (act_fuse && ((N & 1) || ((N / 2) & 7) || act_fuse < 1 || act_fuse > 4 || (act_fuse == 4) != (clamp != nullptr)))
    return -1;
  // up to 64 rows an expert on average: weight-bound, see gemm_cluster.cu (us, gated + down, against the kernel above:
  // 3 tokens of 128 experts of 768, top 8, 28 + 31 -> 29 + 19; 64 tokens 150 + 132 -> 132 + 71; 1024 tokens 194 + 158 ->
  // 166 + 94; from there on the wider tiles win: 2048 tokens 250 + 130 against 240 + 188, less with two CTAs per SM)
  if (act_fuse != 4 && max_rows <= 64 * E && !(reinterpret_cast<uintptr_t>(out) & 15)) {
    ExpertsCluster g{};
    g.xs = xs; g.W = W; g.out = out;
    g.chunk_expert = (const int32_t*)chunk_expert; g.chunk_row0 = (const int32_t*)chunk_row0;
    g.chunk_n = (const int32_t*)chunk_n; g.num_chunks = (const int32_t*)meta + 3 * E + 1;
    g.max_rows = max_rows; g.max_chunks = max_chunks; g.E = E; g.N = N; g.K = K; g.gated = act_fuse; g.act = act;
    return launch_experts_cluster(g, stream);
  }
  // Experts of many rows go to CTA pairs, which read the weights once for 256 rows and multiply at twice the rate, padded to 256
  // rows an expert: from 160 rows on average on, plain from 128. us, the kernel below / pairs, gated and plain: 128 experts of
  // 768, width 2048, 68 rows 152 / 181 and 99 / 94, 128 rows 183 / 186 and 117 / 106, 187 rows 228 / 189 and 131 / 110, 512 rows
  // 473 / 407 and 292 / 247; 64 of 1408, 768 rows 619 / 487 and 323 / 241; 8 of 1792, width 4096, 150 rows 68 / 72 and 37 / 34,
  // 1024 rows 268 / 181 and 129 / 96; 8 of 14336, 300 rows 756 / 649 and 363 / 347, 1024 rows 2143 / 1443 and 958 / 766;
  // 32 of 2880, 75 rows 209 / 248 and 133 / 142.
  if (act_fuse != 4 && max_rows >= (act_fuse ? 160 : 128) * (long long)E && max_chunks <= kPMostChunks &&
      !(reinterpret_cast<uintptr_t>(out) & 15)) {
    GroupedPairParams q{};
    q.N = N; q.K = K; q.E = E; q.max_chunks = max_chunks; q.tiles = act_fuse ? (N / 2 + 127) / 128 : (N + 255) / 256;
    q.act_fuse = act_fuse; q.act = act; q.out = (bf16*)out;
    q.chunk_expert = (const int32_t*)chunk_expert; q.chunk_row0 = (const int32_t*)chunk_row0;
    q.chunk_n = (const int32_t*)chunk_n; q.meta = (const int32_t*)meta; q.status = device_status_word();
    CUtensorMap tW, tX;
    if (!encode_tmap_3d(&tW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)N, (uint64_t)E, (uint64_t)K * 2,
                        (uint64_t)N * K * 2, kGBK, 128, 1, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_tmap_2d(&tX, xs, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)max_rows + 256, (uint64_t)K, (uint64_t)K, 128, kGBK,
                        CU_TENSOR_MAP_SWIZZLE_128B))
      return -3;
    const size_t bytes = (size_t)kPStages * kPStage + (size_t)max_chunks * sizeof(GroupedPairChunk) + 1024;
    static PerDeviceOnce once;
    if (once.first())
      cudaFuncSetAttribute(moe_grouped_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kPStages * kPStage + kPMostChunks * (int)sizeof(GroupedPairChunk) + 1024);
    const long long tiles = (long long)max_chunks * q.tiles;
    const int pairs = (int)(tiles < b200_num_sms() / 2 ? tiles : b200_num_sms() / 2);
    return launch_cluster_pdl(moe_grouped_pair_kernel, dim3(2 * pairs), 2, 192, bytes, stream, tW, tX, q) == cudaSuccess ? 0 : -2;
  }
  // Gated: 128 rows a CTA and two CTAs an SM, or 256 rows, a CTA with three stages of 64 KB alone on its SM. The smaller CTA
  // hides its epilogue behind its neighbour, but reads the weights once for every 128 rows and has two stages of 48 KB.
  //  - Few CTAs (about 1.35 an SM; an expert's last 128 rows are half full on average) have no neighbour. us, 256 / 128 rows:
  //    8 experts of 1792, width 4096, 70 and 190 rows each 55 / 81, 73 / 91; 16 of 1024, width 2048, 70 rows 39 / 51. With
  //    more than 192 rows an expert the second CTA halves the time all the same: 4 of 2048, width 2048, 256 rows 53 / 44.
  //  - Long products (K of 4096 on) have little epilogue: 8 of 14336, width 4096, 150 rows 459 / 551, 400 rows 902 / 1056;
  //    16 of 8192, width 5120, 150 rows 560 / 699, 1024 rows 2740 / 3024. Up to 128 rows there is no second reading: 70 rows
  //    386 / 344 and 479 / 442.
  //  - Shorter ones: 128 of 768, width 2048, 70 rows 202 / 162, 1024 rows 1128 / 917; 32 of 2880, width 2880, 512 rows 670 / 595.
  const int tiles = ((act_fuse ? N / 2 : N) + kGBM - 1) / kGBM;
  const long long sms = b200_num_sms(), per128 = (long long)tiles * E * ((max_rows + 128 * E - 1) / (128 * E));
  const bool few = max_rows <= 192 * E ? 20LL * tiles * (max_rows / 128 + E / 2) < 27 * sms : per128 <= 2 * sms;
  const bool pairs = act_fuse && (max_rows <= 192 * E ? !few && (K < 4096 || max_rows <= 128 * E) : few || K < 4096);
  const int sub_rows = pairs ? 128 : 256;
  CUtensorMap tmW, tmX;
  if (!encode_tmap_3d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)N,
                      (uint64_t)E, (uint64_t)K * 2, (uint64_t)N * K * 2, kGBK, kGBM, 1,
                      CU_TENSOR_MAP_SWIZZLE_128B))
    return -3;
  if (!encode_tmap_2d(&tmX, xs, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)max_rows + 256,
                      (uint64_t)K, (uint64_t)K, sub_rows, kGBK, CU_TENSOR_MAP_SWIZZLE_128B))
    return -3;
  GroupedParams p;
  p.sub_rows = sub_rows;
  p.N = N; p.K = K; p.out = (bf16*)out;
  p.chunk_expert = (const int32_t*)chunk_expert; p.chunk_row0 = (const int32_t*)chunk_row0;
  p.chunk_n = (const int32_t*)chunk_n; p.meta = (const int32_t*)meta; p.E = E;
  const int stage = kGBM * kGBK * 2 * (act_fuse ? 2 : 1) + sub_rows * kGBK * 2;
  // Plain product: two stages and a neighbour on the SM, or, where the grid leaves no SM two CTAs, four stages (an expert's last 256
  // rows are half full on average): 8 experts of 14336, width 1024, us, four / two stages: 66 rows each 123 / 158 (64 CTAs), 400 rows
  // 130 / 181 (132), 700 rows 256 / 192 (207); 16 of 4096, width 512, 256 rows 47 / 62, 700 rows 89 / 68.
  const long long most = max_rows / 256 + E / 2, ctas = (long long)tiles * (most > E ? most : E);
  const bool alone = act_fuse ? !pairs : ctas <= sms;
  int stages = (alone ? 200 : 96) * 1024 / stage;
  if (stages > kGMaxStages) stages = kGMaxStages;
  const int nkb = (K + kGBK - 1) / kGBK;
  if (stages > nkb) stages = nkb < 2 ? 2 : nkb;
  p.stages = stages; p.act_fuse = act_fuse; p.act = act; p.status = device_status_word();
  if (clamp) p.clamp = *clamp;
  const size_t smem = (size_t)stages * stage + 1024 + sizeof(GroupedBars);
  static PerDeviceOnce attr_once;
  if (attr_once.first()) {
    cudaFuncSetAttribute(moe_grouped_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         220 * 1024);
  }
  dim3 grid((unsigned)(tiles * (256 / sub_rows)), (unsigned)max_chunks);
  moe_grouped_gemm_kernel<<<grid, 192, smem, stream>>>(tmW, tmX, p);
  RETL;
}

int b200_moe_grouped_gemm(const void* xs, int max_rows, const void* W, int E, int N, int K,
                          void* out, const void* chunk_expert, const void* chunk_row0,
                          const void* chunk_n, const void* meta, int max_chunks,
                          cudaStream_t stream) {
  return moe_grouped_gemm_impl(xs, max_rows, W, E, N, K, out, chunk_expert, chunk_row0, chunk_n, meta, max_chunks, 0,
                               stream);
}
// Gate / up projection with the gated activation in the epilogue: W [E, 2 I, K] with rows
// [gate (I) | up (I)], out[P, I] = act(xs W_gate^T) * (xs W_up^T). kind: 0 SiLU, 1 GELU-tanh, 2 GELU-erf.
int b200_moe_grouped_gemm_gated(const void* xs, int max_rows, const void* W, int E, int N, int K,
                                void* out, const void* chunk_expert, const void* chunk_row0,
                                const void* chunk_n, const void* meta, int max_chunks, int kind,
                                cudaStream_t stream) {
  return moe_grouped_gemm_impl(xs, max_rows, W, E, N, K, out, chunk_expert, chunk_row0, chunk_n, meta, max_chunks,
                               kind + 1, stream);
}
// Same with the clamped pair as the activation (B200ClampedGate); a routing weight that scales the
// expert's input is applied here, to the accumulators: W (w x) = w (W x).
int b200_moe_grouped_gemm_clamped(const void* xs, int max_rows, const void* W, int E, int N, int K,
                                  void* out, const void* chunk_expert, const void* chunk_row0,
                                  const void* chunk_n, const void* meta, int max_chunks,
                                  const B200ClampedGate* act, cudaStream_t stream) {
  if (!act) return -1;
  return moe_grouped_gemm_impl(xs, max_rows, W, E, N, K, out, chunk_expert, chunk_row0, chunk_n, meta, max_chunks, 4,
                               stream, act);
}
// The plain product with an activation of the result (act_epilogue).
int b200_moe_grouped_gemm_act(const void* xs, int max_rows, const void* W, int E, int N, int K,
                              void* out, const void* chunk_expert, const void* chunk_row0,
                              const void* chunk_n, const void* meta, int max_chunks, int act,
                              cudaStream_t stream) {
  return moe_grouped_gemm_impl(xs, max_rows, W, E, N, K, out, chunk_expert, chunk_row0, chunk_n, meta, max_chunks, 0,
                               stream, nullptr, act);
}
int b200_moe_row_weights(const void* pair_pos, const void* topk_w, int P, void* row_w, cudaStream_t stream) {
  if (P <= 0) return 0;
  moe_row_weights_kernel<<<(P + 255) / 256, 256, 0, stream>>>((const int32_t*)pair_pos, (const float*)topk_w, P,
                                                            (float*)row_w);
  RETL;
}


int b200_moe_combine(const void* y, const void* pair_pos, const void* topk_w, int T, int k, int H,
                     const void* shared, const void* shared_gate, void* out,
                     const B200MoeScatter* sc, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return -1;
  CombineParams p{};
  p.y = (const bf16*)y; p.pair_pos = (const int32_t*)pair_pos; p.topk_w = (const float*)topk_w;
  p.k = k; p.H = H; p.T = T; p.shared = (const bf16*)shared; p.shared_gate = (const float*)shared_gate;
  p.out = (bf16*)out;
  if (sc && sc->world > 1) {
    p.tp_world = sc->world; p.tp_rank = sc->rank; p.rows_per_rank = sc->rows_per_rank;
    for (int i = 0; i < sc->world; ++i) {
      p.peer_recv[i] = (bf16*)sc->peer_recv[i];
      p.peer_rs_flags[i] = (uint32_t*)sc->peer_rs_flags[i];
    }
    p.recv_parity_stride = sc->recv_parity_stride;
    p.rs_flag_parity_stride = sc->rs_flag_parity_stride;
    p.op_counter = (const uint32_t*)sc->op_counter;
  }
  if (sc && sc->world > 1) {
    moe_combine_kernel<<<T, 128, 0, stream>>>(p);
    RETL;
  }
  return launch_pdl(moe_combine_kernel, dim3(T), dim3(H >= 2048 ? 256 : 128), 0, stream, p) == cudaSuccess ? 0 : -2;
}

int b200_shared_gate(const void* x, int ldx, const void* w, int T, int H, void* out,
                     cudaStream_t stream) {
  if (T <= 0) return 0;
  shared_gate_kernel<<<T, 128, 0, stream>>>((const bf16*)x, ldx, (const bf16*)w, H, (float*)out);
  RETL;
}

}  // extern "C"
