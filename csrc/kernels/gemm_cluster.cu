// Small-batch bf16 product  C[M,N] = A[M,K] * W[N,K]^T  for M <= 128, split over K inside a thread-block cluster.
//
// The weights are the 128-row operand of tcgen05.mma and the batch, padded to 16, its N, so every weight is read once.
// What bounds it is the weight stream: a CTA holds about 100 KB of shared memory, so that two CTAs share an SM and the
// grid (row tiles x splits) stays in one wave; HBM, not the number of tiles, then shares the work out, and the next
// kernel's CTAs move in while the last tiles drain. The CTAs of a cluster take the parts of K of one row tile (with a
// gated activation: of the gate tile and of the up tile). Each leaves its fp32 partial tile in its own shared memory, and
// every CTA sums a share of the batch rows over the cluster, in the order of the splits, applies what follows the
// product and writes whole 256-byte rows: no partials in global memory, no second kernel.
//
// Measured on B200, launches in a chain over weights beyond L2, us at M = 1 / 13 / 40 / 120, against split-K with its
// partials in global memory, one CTA per SM and a reducing kernel:
//   6144 x 4096    16.1 / 17.5 / 20.5 / 30.2  ->  10.6 / 10.8 / 12.5 / 15.2   (4.7 TB/s at M = 1)
//   4096 x 4096    13.7 / 14.9 / 18.2 / 27.7  ->   8.6 /  8.8 / 10.3 / 13.7   (3.9)
//   4096 x 14336   28.1 / 29.6 / 33.0 / 43.2  ->  22.5 / 22.8 / 24.0 / 28.5   (5.2)
//   1024 x 2048     6.5 /  7.7 / 11.0 / 20.5  ->   4.6 /  5.0 /  5.8 /  7.2
//   28672 x 4096 and the gated activation, against 128 x 256 tiles and its own kernel: 53.6 / 53.0 / 48.2 / 50.7 ->
//   40.8 / 41.9 / 44.8 / 51.3 (5.8)
// What is left at the small sizes is the start of a kernel and the cluster's exchange, about 3 us.
//
// Warp roles (192 threads): warp 0 TMA producer, warp 1 TMEM owner + MMA issuer, warps 2..5 read the accumulator;
// all six sum the cluster's partials.
//
// Replaces the library GEMM calls of the reference (src/vt/cuda/cuda_matmul.cu:284-355 "MatmulBT", :219-274) for
// decode-sized batches.
#include "api.h"
#include "rope.cuh"
#include "sm100.cuh"

namespace b200 {

static constexpr int kRows = 128;          // weight rows of a tile
static constexpr int kRowBytes = 128;      // bytes of a row in a stage: 64 bf16 or 128 e4m3 k-elements
static constexpr int kThreads = 192;
static constexpr int kRingStages = 8;
static constexpr int kSmemPerCta = 109 * 1024;      // two CTAs per SM
static constexpr int kMostRows = 128;      // batch rows of one pass

enum ClusterKind { kDense, kExperts, kFp8 };
// The batch as the product reads it: boxes of all its padded rows, or, where the rows of a product are only known on the
// device, of 16, 32, 64 and 128.
template <ClusterKind KIND>
struct BatchMaps {
  CUtensorMap m[KIND == kExperts ? 4 : 1];
};

struct ClusterParams {
  int M, N, K;
  int mp;                    // M padded to 16: N of the MMA
  int ring_bytes, kblocks;
  int splits;                // CTAs of a row tile
  int gated;                 // 1 + kind of the gated activation: cluster = 2 x splits, the gate tile's CTAs and the up tile's
  int up_rows;               // gated: weight rows from a gate tile to its up tile (128: interleaved blocks)
  void* out;
  long long ldo;
  int out_f32, act, w_early;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int ldr;
  int batch_a_cols;          // batched (blockIdx.z): first A column of batch b is b * batch_a_cols,
  long long batch_out;       // its output starts at out + b * batch_out, its weights at row b * N
  // experts (blockIdx.y): rows chunk_row0 .. + chunk_n of the sorted batch, weights of chunk_expert
  const int32_t *chunk_expert, *chunk_row0, *chunk_n, *num_chunks;
  // fp8: the sums times a_scale (of the tensor, or per row) and w_scale (of the tensor, or per output column)
  const float *a_scale, *w_scale;
  int a_per_row, w_per_col;
  RopeOut rope;              // (ROPE) a tile is a head
  int* status;
};

struct alignas(8) ClusterBars {
  uint64_t full[kRingStages], empty[kRingStages], acc;
  uint32_t tmem_base;
};

__device__ __forceinline__ float rounded(float x) { return __bfloat162float(__float2bfloat16(x)); }

// act(gate) * up; both are rounded first, as where the product and the activation are two kernels
__device__ __forceinline__ float4 gated4(const float4& g, const float4& u, int kind) {
  return make_float4(act_of(rounded(g.x), kind) * rounded(u.x), act_of(rounded(g.y), kind) * rounded(u.y),
                     act_of(rounded(g.z), kind) * rounded(u.z), act_of(rounded(g.w), kind) * rounded(u.w));
}
// The sums' scales, bias, residual and activation. col: first of the lane's four columns of the output, m: row of the output
__device__ __forceinline__ float4 finished(const ClusterParams& p, float4 a, int m, int col) {
  if (p.a_scale) {
    const float sa = p.a_scale[p.a_per_row ? m : 0];
    const float* sw = p.w_scale + (p.w_per_col ? col : 0);
    const int one = p.w_per_col ? 1 : 0;
    a.x = a.x * sa * __ldg(sw); a.y = a.y * sa * __ldg(sw + one); a.z = a.z * sa * __ldg(sw + 2 * one); a.w = a.w * sa * __ldg(sw + 3 * one);
  }
  if (p.bias) {
    const uint2 b = *reinterpret_cast<const uint2*>(p.bias + col);
    const float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y);
    a.x += f0.x; a.y += f0.y; a.z += f1.x; a.w += f1.y;
  }
  if (p.residual) {
    const uint2 b = *reinterpret_cast<const uint2*>(p.residual + (size_t)m * p.ldr + col);
    const float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y);
    a.x += f0.x; a.y += f0.y; a.z += f1.x; a.w += f1.y;
  }
  if (p.act) {
    a.x = act_epilogue<true>(a.x, p.act); a.y = act_epilogue<true>(a.y, p.act);
    a.z = act_epilogue<true>(a.z, p.act); a.w = act_epilogue<true>(a.w, p.act);
  }
  return a;
}
__device__ __forceinline__ void finish_row(const ClusterParams& p, float4 a, int m, int col) {
  if (col >= (p.gated ? p.N >> 1 : p.N)) return;                     // (a multiple of 8)
  a = finished(p, a, m, col);
  const size_t at = blockIdx.z * p.batch_out + (size_t)m * p.ldo + col;
  if (p.out_f32)
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at) = a;
  else
    *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + at) = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
}

// With a rotation: what a warp needs of its next row, fetched ahead of it.
struct RopeRow {
  float4 c, s;
  int64_t slot;
};
__device__ __forceinline__ RopeRow rope_row(const RopeOut& r, int m, int head, int lane) {
  RopeRow o;
  o.slot = head >= r.Hq ? r.slot_mapping[m] : -1;
  if (head < r.Hq + r.Hkv) {
    const float* cs = r.cos_sin + (size_t)r.positions[m] * 128 + (lane & 15) * 4;
    o.c = *reinterpret_cast<const float4*>(cs);
    o.s = *reinterpret_cast<const float4*>(cs + 64);
  }
  return o;
}
// The row's head as the product would have stored it, rounded, then b200_rope_kv's arithmetic.
__device__ __forceinline__ void finish_head(const ClusterParams& p, float4 a, int m, int head, const RopeRow& row, int lane) {
  const RopeOut& r = p.rope;
  a = finished(p, a, m, head * 128 + lane * 4);
  uint2 o = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
  const int v0 = r.Hq + r.Hkv;
  if (head < v0) {
    const float2 lo = unpack_bf16x2(o.x), hi = unpack_bf16x2(o.y);
    const float x[4] = {lo.x, lo.y, hi.x, hi.y};
    o = rope_head(x, row.c, row.s, head < r.Hq ? r.q_norm : r.k_norm, r.eps, r.gemma, lane);
  }
  if (head >= r.Hq) {
    const RopeCacheSlot cache = rope_cache_slot(row.slot, r.kv_cache, r.block_size, r.Hkv);
    __nv_bfloat16* dst = head < v0 ? cache.k : cache.v;
    if (dst) *reinterpret_cast<uint2*>(dst + (head < v0 ? head - r.Hq : head - v0) * 128 + lane * 4) = o;
  }
  *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)m * p.ldo + head * 128 + lane * 4) = o;
}

// Batch rows rank, rank + ranks, ... of the pass, dealt to the six warps, four columns a lane.
template <int S, bool ROPE>
__device__ __forceinline__ void reduce_rows(const ClusterParams& p, uint32_t partial, int rank, int ranks, int rows, int row0,
                                            int col, int warp, int lane, RopeRow next) {
  if constexpr (ROPE) {                    // (one pass, row0 = 0)
    const int head = col >> 7;
    for (int m = rank + warp * ranks; m < rows; m += 6 * ranks) {
      const RopeRow row = next;
      if (m + 6 * ranks < rows) next = rope_row(p.rope, m + 6 * ranks, head, lane);
      finish_head(p, sum_of<S>(partial + (uint32_t)m * (kRows * 4) + lane * 16, 0), m, head, row, lane);
    }
    return;
  }
  for (int m = rank + warp * ranks; m < rows; m += 6 * ranks) {
    const uint32_t addr = partial + (uint32_t)m * (kRows * 4) + lane * 16;
    float4 x = sum_of<S>(addr, 0);
    if (p.gated) x = gated4(x, sum_of<S>(addr, S), p.gated - 1);
    finish_row(p, x, row0 + m, col);
  }
}

template <ClusterKind KIND, bool ROPE = false>
__global__ void __launch_bounds__(kThreads, 2)
    gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ BatchMaps<KIND> tmA, ClusterParams p,
                        uint32_t tmem_cols) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ ClusterBars bars;
  constexpr int kWBytes = kRows * kRowBytes, kKB = KIND == kFp8 ? 128 : 64;
  constexpr bool EXPERTS = KIND == kExperts;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int ranks = (p.gated ? 2 : 1) * p.splits;
  const int rank = ranks > 1 ? (int)cluster_ctarank() : 0;
  const int split = rank % p.splits, half = rank / p.splits;           // half 1: the up tile
  const int tile = blockIdx.x / ranks;                                 // of the output
  const int kb0 = (int)((long long)p.kblocks * split / p.splits);
  const int nkb = (int)((long long)p.kblocks * (split + 1) / p.splits) - kb0;
  const int w_row = blockIdx.z * p.N + (p.gated && p.up_rows == kRows ? 2 * tile : tile) * kRows + half * p.up_rows;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRingStages; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    mbar_init(&bars.acc, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars.tmem_base, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = bars.tmem_base;


  int box = p.mp, total = p.M, row_base = 0, expert = 0;
  int stage_bytes = kWBytes + box * kRowBytes;
  int stages = min(kRingStages, p.ring_bytes / stage_bytes);
  // weights that nothing in the stream writes are fetched while the predecessor still runs
  int npre = 0;
  if (!EXPERTS && warp == 0 && p.w_early) {
    npre = min(nkb, stages);
    if (elect_one()) {
      tma_prefetch_desc(&tmW);
      for (int i = 0; i < npre; ++i) {
        mbar_expect_tx(&bars.full[i], stage_bytes);
        tma_load_2d(smem + (size_t)i * stage_bytes, &tmW, &bars.full[i], (kb0 + i) * kKB, w_row);
      }
    }
    __syncwarp();
  }
  pdl_wait();
  pdl_launch_dependents();
  int map = 0;
  if (EXPERTS) {
    const int chunk = blockIdx.y;
    total = chunk < *p.num_chunks ? p.chunk_n[chunk] : 0;               // 0 for the whole cluster: nothing to do
    if (total > 0) {
      row_base = p.chunk_row0[chunk];
      expert = p.chunk_expert[chunk];
      box = total <= 16 ? 16 : total <= 32 ? 32 : total <= 64 ? 64 : kMostRows;
      map = total <= 16 ? 0 : total <= 32 ? 1 : total <= 64 ? 2 : 3;
      stage_bytes = kWBytes + box * kRowBytes;
      stages = min(kRingStages, p.ring_bytes / stage_bytes);
    }
  }

  // (the warps that load and multiply fetch theirs when they are through: it is a chain of two loads)
  RopeRow rope{};
  const bool rotates = ROPE && rank + warp * ranks < total;
  if (rotates && warp >= 2) rope = rope_row(p.rope, rank + warp * ranks, tile, lane);

  int slot = 0;                             // of the ring, for the warps that load and multiply (over the passes)
  uint32_t turn = 0;                        // parity of its use
  for (int first = 0, pass = 0; first < total; first += kMostRows, ++pass) {
    const int rows = min(kMostRows, total - first);
    const int np = EXPERTS ? (rows + 15) & ~15 : p.mp;
    if (warp == 0) {
      for (int i = 0; i < nkb; ++i) {
        if (!mbar_wait_warp(&bars.empty[slot], turn ^ 1, p.status)) break;
        uint8_t* w_dst = smem + (size_t)slot * stage_bytes;
        if (elect_one()) {
          if (i >= npre) {
            mbar_expect_tx(&bars.full[slot], stage_bytes);
            if (EXPERTS) tma_load_3d(w_dst, &tmW, &bars.full[slot], (kb0 + i) * kKB, w_row, expert);
            else tma_load_2d(w_dst, &tmW, &bars.full[slot], (kb0 + i) * kKB, w_row);
          }
          tma_load_2d(w_dst + kWBytes, &tmA.m[map], &bars.full[slot], blockIdx.z * p.batch_a_cols + (kb0 + i) * kKB, row_base + first);
        }
        __syncwarp();
        if (++slot == stages) { slot = 0; turn ^= 1; }
      }
    } else if (warp == 1) {
      const uint32_t idesc = KIND == kFp8 ? umma_idesc_e4m3(kRows, np) : umma_idesc_bf16(kRows, np);
      const uint32_t acc = __shfl_sync(0xffffffffu, tmem, 0);
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        if (!(ok = mbar_wait_warp(&bars.full[slot], turn, p.status))) break;
        tc_fence_after_sync();
        const uint32_t w_addr = smem_u32(smem + (size_t)slot * stage_bytes);
        const uint64_t wdesc = umma_desc_k_sw128(w_addr, 1024), adesc = umma_desc_k_sw128(w_addr + kWBytes, 1024);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {       // 32 bytes of a row each
            if (KIND == kFp8) umma_f8f6f4_ss(acc, wdesc + 2 * k, adesc + 2 * k, idesc, (i | k) != 0);
            else umma_bf16_ss(acc, wdesc + 2 * k, adesc + 2 * k, idesc, (i | k) != 0);
          }
          umma_commit(&bars.empty[slot]);
          if (i == nkb - 1) umma_commit(&bars.acc);
        }
        __syncwarp();
        if (++slot == stages) { slot = 0; turn ^= 1; }
      }
    } else {
      // accumulator (lane = weight row, column = batch row) -> this CTA's partial tile [rows][128] over the ring, whose
      // loads and products have all completed
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bars.acc, pass & 1, p.status));
      tc_fence_after_sync();
      if (ok) {
        const int quarter = warp & 3;
        float* dst = reinterpret_cast<float*>(smem) + quarter * 32 + lane;
        const uint32_t t_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        int c = 0;
        for (; c + 32 <= np; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(t_addr + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) dst[(c + i) * kRows] = __uint_as_float(r[i]);
        }
        if (c < np) {
          uint32_t r[16];
          tmem_ld_32x32b_x16(t_addr + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) dst[(c + i) * kRows] = __uint_as_float(r[i]);
        }
      }
    }
    if (rotates && warp < 2) rope = rope_row(p.rope, rank + warp * ranks, tile, lane);
    tc_fence_before_sync();
    __syncthreads();
    if (ranks > 1) cluster_sync_all();       // every partial tile of the cluster is in place
    tc_fence_after_sync();
    const uint32_t partial = smem_u32(smem);
    const int col = tile * kRows + lane * 4, row0 = row_base + first;
    switch (p.splits) {
      case 1: reduce_rows<1, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 2: reduce_rows<2, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 3: reduce_rows<3, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 4: reduce_rows<4, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 5: reduce_rows<5, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 6: reduce_rows<6, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      case 7: reduce_rows<7, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
      default: reduce_rows<8, ROPE>(p, partial, rank, ranks, rows, row0, col, warp, lane, rope); break;
    }
    fence_proxy_async_smem();                // (a further pass loads over the partial tile)
    if (ranks > 1) cluster_sync_all();       // nobody reads this CTA's partial any more
    else __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, tmem_cols);
}

// How many clusters of `ranks` CTAs run at once at least, two CTAs to an SM. A cluster stays within a GPC, so that fewer
// of the larger ones fit. The driver counts one CTA to an SM for a kernel that allocates tensor memory (74 clusters of 2,
// 33 of 4, 15 of 8 on a B200; a kernel of the same size without it 148, 71, 33), so its answer is doubled. 0: it has none.
static int clusters_at_once(int ranks) {
  static std::atomic<int> known[64][9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  const int k = known[dev][ranks].load(std::memory_order_relaxed);
  if (k) return k;
  if (ranks == 1) return 2 * b200_num_sms();
  if (cudaFuncSetAttribute(gemm_cluster_kernel<kDense>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta) != cudaSuccess)
    return 0;                       // (the query below refuses more than the limit)
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(ranks * b200_num_sms()));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemPerCta;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_cluster_kernel<kDense>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  known[dev][ranks].store(2 * n, std::memory_order_relaxed);
  return 2 * n;
}

// CTAs of a row tile: as many as leave the whole grid in one wave, of eight in a cluster at most, with at least two
// stages of K each. A grid that needs a second wave loses more than the finer split gains (us at M = 1, splits 4 / 5 / 6 / 8):
//   6144 x 4096 (48 tiles)   12.6 / 10.7 / 17.7 / 15.2     4096 x 4096 (32)   11.9 / 10.4 / 8.5 / 8.7
//   5120 x 4096 (40 tiles)   12.2 / 10.3 /  9.4 / 14.8     6144 x 1024 (48)    6.0 /  5.8 / 9.8 / 9.4
// Up to four stages of K are fetched sooner than they are exchanged, once there are row tiles enough (us at 3 / 64 rows, one
// part / two: 8192 x 256 3.5 / 4.1, 5.8 / 6.4; 14336 x 256 3.6 / 5.1, 5.8 / 7.7; 4096 x 256 3.6 / 3.6, 5.7 / 5.6). A gated tile
// is exchanged in any case (12288 x 256 at 64 rows 9.5 / 8.4).
static int choose_splits(int clusters, int kblocks, int gated) {
  if (!gated && kblocks <= 4 && clusters >= 64) return 1;
  int s = gated ? 4 : 8;
  while (s > 1 && (s * 2 > kblocks || clusters > clusters_at_once(gated ? 2 * s : s))) --s;
  return s;
}

int cluster_splits(int tiles, int most) {
  int s = most < 8 ? most : 8;
  while (s > 1 && tiles > clusters_at_once(s)) --s;
  return s < 1 ? 1 : s;
}

template <ClusterKind KIND, bool ROPE = false>
static int launch(const CUtensorMap& tmW, const BatchMaps<KIND>& tmA, const ClusterParams& p, dim3 grid, int ranks,
                  uint32_t tmem_cols, cudaStream_t stream) {
  static PerDeviceOnce attr_once;
  if (attr_once.first())
    cudaFuncSetAttribute(gemm_cluster_kernel<KIND, ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta);
  return launch_cluster_pdl(gemm_cluster_kernel<KIND, ROPE>, grid, ranks, kThreads, p.ring_bytes + 1024, stream, tmW, tmA, p, tmem_cols) ==
                 cudaSuccess ? 0 : -2;
}

// Bytes of a CTA's ring, for `mp` rows (padded to 16) and its `longest` k-blocks, which the partial tile takes afterwards, and its columns of
// tensor memory. One k-block of 65 to 80 rows would let five CTAs onto an SM that has columns for four.
static int cluster_ring(int mp, int longest, int ranks, uint32_t* tmem_cols) {
  const int stage_bytes = (kRows + mp) * kRowBytes;
  int stages = (kSmemPerCta - 1024) / stage_bytes;
  if (stages > kRingStages) stages = kRingStages;
  if (stages > longest) stages = longest;
  int bytes = stages * stage_bytes;
  if (bytes < mp * kRows * 4) bytes = mp * kRows * 4;
  int cols = 32;
  while (cols < mp) cols <<= 1;
  *tmem_cols = (uint32_t)cols;
  return ranks > 1 ? (int)tmem_bound_smem(bytes, 512 / cols + 1, cols) : bytes;
}

int launch_gemm_cluster(const GemmCluster& g, cudaStream_t stream) {
  if (g.M < 1 || g.M > kMostRows || (g.gated && (g.N & 255))) return -1;
  if (g.rope && (g.gated || g.batch > 1 || g.out_f32 || g.N != (g.rope->Hq + 2 * g.rope->Hkv) * kRows)) return -1;
  ClusterParams p{};
  p.M = g.M; p.N = g.N; p.K = g.K;
  p.mp = (g.M + 15) & ~15;
  const int kb = g.a_scale ? 128 : 64;
  p.kblocks = (g.K + kb - 1) / kb;
  p.gated = g.gated; p.up_rows = kRows;
  p.a_scale = g.a_scale; p.w_scale = g.w_scale; p.a_per_row = g.a_per_row; p.w_per_col = g.w_per_col;
  p.out = g.out; p.ldo = g.ldo; p.out_f32 = g.out_f32; p.act = g.act; p.w_early = g.w_early;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias);
  p.residual = reinterpret_cast<const __nv_bfloat16*>(g.residual);
  p.ldr = g.ldr;
  p.batch_a_cols = g.batch_a_cols;
  p.batch_out = g.batch_out;
  if (g.rope) p.rope = *g.rope;
  p.status = device_status_word();
  const int tiles = ((g.gated ? g.N / 2 : g.N) + kRows - 1) / kRows;
  p.splits = g.splits > 0 ? g.splits : choose_splits(tiles * g.batch, p.kblocks, g.gated);
  if (p.splits > p.kblocks) p.splits = p.kblocks;
  const int ranks = (g.gated ? 2 : 1) * p.splits;
  if (ranks > 8) return -1;
  uint32_t tmem_cols = 0;
  p.ring_bytes = cluster_ring(p.mp, (p.kblocks + p.splits - 1) / p.splits, ranks, &tmem_cols);
  CUtensorMap tmW;
  const dim3 grid((unsigned)(tiles * ranks), 1, (unsigned)g.batch);
  if (g.a_scale) {
    BatchMaps<kFp8> tm8;
    if (!encode_tmap_2d(&tmW, g.W, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g.N, g.K, g.ldw, kRows, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_tmap_2d(&tm8.m[0], g.A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, g.M, g.K, g.lda, p.mp, 128, CU_TENSOR_MAP_SWIZZLE_128B))
      return -3;
    return (g.rope ? launch<kFp8, true> : launch<kFp8>)(tmW, tm8, p, grid, ranks, tmem_cols, stream);
  }
  BatchMaps<kDense> tmA;
  if (!get_tmap_bf16(&tmW, g.W, (uint64_t)g.batch * g.N, g.K, g.ldw, kRows, 64)) return -3;
  if (!get_tmap_bf16(&tmA.m[0], g.A, g.M, g.batch > 1 ? (uint64_t)g.lda : (uint64_t)g.K, g.lda, p.mp, 64)) return -3;
  return (g.rope ? launch<kDense, true> : launch<kDense>)(tmW, tmA, p, grid, ranks, tmem_cols, stream);
}

// out[P, N] = grouped(xs[P, K], W[E, N, K]) for chunks of few rows; gated: W_e = [gate (N / 2) | up (N / 2)], out[P, N / 2].
// Every chunk holds a row at least, so there are max_rows of them at most.
int launch_experts_cluster(const ExpertsCluster& g, cudaStream_t stream) {
  ClusterParams p{};
  p.N = g.N; p.K = g.K; p.mp = kMostRows;
  p.kblocks = (g.K + 63) / 64;
  p.gated = g.gated; p.up_rows = g.N / 2;
  p.out = g.out; p.ldo = g.gated ? g.N / 2 : g.N; p.act = g.act;
  p.chunk_expert = g.chunk_expert; p.chunk_row0 = g.chunk_row0; p.chunk_n = g.chunk_n; p.num_chunks = g.num_chunks;
  p.status = device_status_word();
  const int chunks = g.max_chunks < g.max_rows ? g.max_chunks : g.max_rows;
  const int tiles = ((g.gated ? g.N / 2 : g.N) + kRows - 1) / kRows;
  p.splits = choose_splits(tiles * chunks, p.kblocks, g.gated);
  const int ranks = (g.gated ? 2 : 1) * p.splits;
  p.ring_bytes = kSmemPerCta - 1024;
  CUtensorMap tmW;
  BatchMaps<kExperts> tmA;
  if (!encode_tmap_3d(&tmW, g.W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.E,
                      (uint64_t)g.K * 2, (uint64_t)g.N * g.K * 2, 64, kRows, 1, CU_TENSOR_MAP_SWIZZLE_128B))
    return -3;
  for (int i = 0; i < 4; ++i)
    if (!get_tmap_bf16(&tmA.m[i], g.xs, (uint64_t)g.max_rows + 256, g.K, g.K, 16 << i, 64)) return -3;
  return launch<kExperts>(tmW, tmA, p, dim3((unsigned)(tiles * ranks), (unsigned)chunks), ranks, kMostRows, stream);
}

}  // namespace b200

extern "C" size_t b200_gemm_cluster_smem(int mp, int longest, int ranks) {
  uint32_t cols = 0;
  return (size_t)b200::cluster_ring(mp, longest, ranks, &cols) + 1024;
}
