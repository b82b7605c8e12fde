// Sampler kernels over fp32 logits [n, V] (row stride ld). All reductions are fixed-order
// tree reductions (no float atomics), argmax breaks ties towards the lowest index, and the
// random draw is an exponential race driven by a SplitMix64 counter RNG that the host
// sampler reproduces bit for bit.
//
// Covers the reference's src/vt/cuda/cuda_sample.cu (ApplyTemperature :62, two-stage argmax
// :102/:130, Softmax :220, RandomSample :270, ApplyTopKTopP :367, ApplyPenalties :510,
// ApplyMinP :544, bias / mask / allowed ids :588-621, greedy rejection :647/:671) and
// cuda_combine_tokens.cu (async-scheduling input splice).
#include <float.h>

#include "api.h"
#include "sm100.cuh"

namespace b200 {

static constexpr int kSB = 256;  // threads per block for row kernels
static constexpr float kEps = 1e-5f;

struct ArgPair { float v; int i; };
__device__ __forceinline__ ArgPair arg_better(ArgPair a, ArgPair b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}
__device__ __forceinline__ ArgPair block_argmax(ArgPair a, ArgPair* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = arg_better(a, b);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) sh[warp] = a;
  __syncthreads();
  ArgPair r = (lane < nw) ? sh[lane] : ArgPair{-FLT_MAX, 0x7fffffff};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, r.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, r.i, o);
    r = arg_better(r, b);
  }
  __syncthreads();
  return r;
}
__device__ __forceinline__ float block_reduce_max(float v, float* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float r = (lane < nw) ? sh[lane] : -FLT_MAX;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
  __syncthreads();
  return r;
}
__device__ __forceinline__ int block_reduce_sum_int(int v, int* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  int r = (lane < nw) ? sh[lane] : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  __syncthreads();
  return r;
}

// ---- two-stage argmax ----
__global__ void __launch_bounds__(kSB)
    argmax_partial_kernel(const float* __restrict__ logits, int ld, int V, int blocks_per_row,
                          float* pv, int* pi) {
  __shared__ ArgPair sh[32];
  const int row = blockIdx.y, blk = blockIdx.x;
  const int per = (((V + blocks_per_row - 1) / blocks_per_row) + 3) & ~3;   // multiple of 4
  const int lo = blk * per, hi = min(V, lo + per);
  const float* x = logits + (size_t)row * ld;
  ArgPair a{-FLT_MAX, 0x7fffffff};
  int i0 = lo;
  if (!(ld & 3) && !(reinterpret_cast<uintptr_t>(logits) & 15)) {
    // 16-byte loads over the aligned part of the slice (lo is a multiple of 4)
    const int hi4 = lo + ((hi - lo) & ~3);
    for (int i = lo + threadIdx.x * 4; i < hi4; i += blockDim.x * 4) {
      const float4 q = *reinterpret_cast<const float4*>(x + i);
      const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) a = arg_better(a, ArgPair{v[k] != v[k] ? -FLT_MAX : v[k], i + k});
    }
    i0 = max(lo, hi4);
  }
  for (int i = i0 + threadIdx.x; i < hi; i += blockDim.x) {
    float v = x[i];
    if (v != v) v = -FLT_MAX;
    a = arg_better(a, ArgPair{v, i});
  }
  a = block_argmax(a, sh);
  if (threadIdx.x == 0) {
    pv[row * blocks_per_row + blk] = a.v;
    pi[row * blocks_per_row + blk] = a.i;
  }
}
__global__ void __launch_bounds__(32)
    argmax_final_kernel(const float* __restrict__ pv, const int* __restrict__ pi,
                        int blocks_per_row, int64_t* out, int V) {
  const int row = blockIdx.x;
  ArgPair a{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < blocks_per_row; i += 32)
    a = arg_better(a, ArgPair{pv[row * blocks_per_row + i], pi[row * blocks_per_row + i]});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = arg_better(a, b);
  }
  if (threadIdx.x == 0) out[row] = (a.i >= V || a.i < 0) ? 0 : a.i;
}

// Vocabulary-parallel greedy sampling: each rank reduces its own logits shard to one
// (value, global index) candidate per row; after the candidates of all ranks have been gathered
// ([n][world] pairs, 8 bytes each) the best one wins, ties going to the lowest index, so the
// result equals the argmax over the full row.
__global__ void __launch_bounds__(32)
    argmax_candidate_kernel(const float* __restrict__ pv, const int* __restrict__ pi,
                            int blocks_per_row, int V, int index_base, int2* __restrict__ out) {
  const int row = blockIdx.x;
  ArgPair a{-FLT_MAX, 0x7fffffff};
  for (int i = threadIdx.x; i < blocks_per_row; i += 32)
    a = arg_better(a, ArgPair{pv[row * blocks_per_row + i], pi[row * blocks_per_row + i]});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgPair b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = arg_better(a, b);
  }
  if (threadIdx.x == 0) {
    const bool ok = a.i >= 0 && a.i < V;
    out[row] = make_int2(__float_as_int(ok ? a.v : -FLT_MAX), ok ? index_base + a.i : 0x7fffffff);
  }
}
__global__ void argmax_combine_kernel(const int2* __restrict__ cand, int n, int world, int V_total,
                                      int64_t* __restrict__ out) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= n) return;
  ArgPair a{-FLT_MAX, 0x7fffffff};
  for (int r = 0; r < world; ++r) {
    const int2 c = cand[(size_t)r * n + row];     // rank-major, as an all-gather along dim 0 lays it out
    a = arg_better(a, ArgPair{__int_as_float(c.x), c.y});
  }
  out[row] = (a.i < 0 || a.i >= V_total) ? 0 : a.i;
}

// ---- temperature: rows with temperature < eps are left untouched (greedy rows) ----
__global__ void temperature_kernel(float* logits, int ld, int V, const float* __restrict__ temp) {
  const int row = blockIdx.y;
  const float t = temp[row];
  if (t < kEps) return;
  const float inv = 1.f / t;
  float* x = logits + (size_t)row * ld;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
    x[i] *= inv;
}

// ---- penalties over (row, token, output_count) triples; every triple is unique ----
__global__ void penalties_kernel(float* logits, int ld, int V, const int* __restrict__ rows,
                                 const int* __restrict__ toks, const int* __restrict__ out_cnt,
                                 int n, const float* __restrict__ rep,
                                 const float* __restrict__ freq, const float* __restrict__ pres) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], t = toks[i];
  if (t < 0 || t >= V) return;
  float v = logits[(size_t)r * ld + t];
  const float rp = rep[r];
  v = v > 0.f ? v / rp : v * rp;
  const int c = out_cnt[i];
  v -= freq[r] * (float)c;
  if (c > 0) v -= pres[r];
  logits[(size_t)r * ld + t] = v;
}

// ---- sparse edits: mode 0 add bias, 1 set -inf ----
__global__ void sparse_edit_kernel(float* logits, int ld, int V, const int* __restrict__ rows,
                                   const int* __restrict__ toks, const float* __restrict__ vals,
                                   int n, int mode) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i], t = toks[i];
  if (t < 0 || t >= V) return;
  if (mode == 0) logits[(size_t)r * ld + t] += vals[i];
  else logits[(size_t)r * ld + t] = -INFINITY;
}

// ---- packed bit mask [n, ceil(V/32)] : bit = 1 keeps the token. row_ids maps mask rows to
// logits rows (grammar requests only); allowed-token-ids use the same kernel. ----
__global__ void bitmask_kernel(float* logits, int ld, int V, const int32_t* __restrict__ mask,
                               int words, const int* __restrict__ row_ids) {
  const int mr = blockIdx.y;
  const int row = row_ids ? row_ids[mr] : mr;
  if (row < 0) return;
  float* x = logits + (size_t)row * ld;
  const int32_t* m = mask + (size_t)mr * words;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
    if (!((m[i >> 5] >> (i & 31)) & 1)) x[i] = -INFINITY;
}

// ---- min-p: drop tokens whose prob < min_p * max prob  <=> logit < max + ln(min_p) ----
__global__ void __launch_bounds__(kSB)
    min_p_kernel(float* logits, int ld, int V, const float* __restrict__ min_p) {
  __shared__ float sh[32];
  const int row = blockIdx.x;
  const float mp = min_p[row];
  if (mp <= 0.f) return;
  float* x = logits + (size_t)row * ld;
  float mx = -FLT_MAX;
  for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, x[i]);
  mx = block_reduce_max(mx, sh);
  const float thr = mx + logf(mp);
  for (int i = threadIdx.x; i < V; i += blockDim.x)
    if (x[i] < thr) x[i] = -INFINITY;
}

// ---- top-k / top-p without a sort ----
// Monotone key: larger float -> larger uint.
__device__ __forceinline__ uint32_t fkey(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}
// A row belongs to a cluster of CTAS CTAs: eight for a long row, as one SM alone reads a vocabulary of 150000 logits at the
// pace of its own loads; one for a short row, whose passes are all barrier (row_ctas). Each CTA keeps its slice in shared
// memory (rows too long for that are read from memory again), sums are taken within the CTA in a fixed order and then over
// the cluster in the order of its CTAs.
static constexpr int kMostStaged = 200 * 1024;      // bytes of a slice in shared memory

struct RowSlice {
  float* x;         // the slice in memory
  const float* v;   // where to read it (shared memory, or x)
  int lo, n;        // first column, columns
};
__host__ __device__ __forceinline__ int row_slice_cols(int V, int ctas) { return ((V + ctas - 1) / ctas + 3) & ~3; }
template <int CTAS>
__device__ __forceinline__ int row_rank() {
  if constexpr (CTAS > 1) return (int)cluster_ctarank();
  return 0;
}
template <int CTAS>
__device__ __forceinline__ void row_sync() {
  if constexpr (CTAS > 1) cluster_sync_all();
}
// Loads this CTA's slice of its row (blockIdx.x / CTAS). Every CTA of the cluster runs when it returns.
template <int CTAS, int T>
__device__ __forceinline__ RowSlice load_row_slice(float* row, int V, float* stage) {
  row_sync<CTAS>();
  const int per = row_slice_cols(V, CTAS), rank = row_rank<CTAS>();
  RowSlice s;
  s.lo = min(V, rank * per);
  s.n = min(V, s.lo + per) - s.lo;
  s.x = row + s.lo;
  s.v = s.x;
  if (per * 4 <= kMostStaged) {
    if (!(reinterpret_cast<uintptr_t>(s.x) & 15)) {
      const int n4 = s.n & ~3;
#pragma unroll 4
      for (int i = threadIdx.x * 4; i < n4; i += T * 4)
        *reinterpret_cast<float4*>(stage + i) = *reinterpret_cast<const float4*>(s.x + i);
      for (int i = n4 + threadIdx.x; i < s.n; i += T) stage[i] = s.x[i];
    } else {
#pragma unroll 4
      for (int i = threadIdx.x; i < s.n; i += T) stage[i] = s.x[i];
    }
    s.v = stage;
    __syncthreads();
  }
  return s;
}
// Exchange of W words per CTA: each CTA stores its own into every CTA of the cluster, and after one cluster barrier all
// threads read them at home. Two buffers in turn, so that one barrier a call is enough.
template <int CTAS, int W>
struct RowExchange {
  float slot[2][CTAS][W];
};
template <int CTAS, int W>
__device__ __forceinline__ void row_gather(RowExchange<CTAS, W>& ex, int turn, const float (&mine)[W], float (&all)[CTAS][W]) {
  if constexpr (CTAS == 1) {
#pragma unroll
    for (int w = 0; w < W; ++w) all[0][w] = mine[w];
    return;
  }
  if (threadIdx.x < CTAS) {
    const uint32_t to = mapa_u32(smem_u32(&ex.slot[turn & 1][cluster_ctarank()][0]), threadIdx.x);
#pragma unroll
    for (int w = 0; w < W; ++w) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4 * w), "f"(mine[w]) : "memory");
  }
  cluster_sync_all();
#pragma unroll
  for (int r = 0; r < CTAS; ++r)
#pragma unroll
    for (int w = 0; w < W; ++w) all[r][w] = ex.slot[turn & 1][r][w];
}
// Sums of W numbers a thread over the whole row (counts stay exact up to 2^24).
template <int CTAS, int T, int W>
__device__ __forceinline__ void row_sum(RowExchange<CTAS, W>& ex, int turn, float (&v)[W], float (&sh)[T / 32][W]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int w = 0; w < W; ++w)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[w] += __shfl_xor_sync(0xffffffffu, v[w], o);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int w = 0; w < W; ++w) sh[warp][w] = v[w];
  __syncthreads();
#pragma unroll
  for (int w = 0; w < W; ++w) {
    float r = lane < T / 32 ? sh[lane][w] : 0.f;
#pragma unroll
    for (int o = T / 64; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    v[w] = __shfl_sync(0xffffffffu, r, 0);
  }
  float all[CTAS][W];
  row_gather<CTAS, W>(ex, turn, v, all);
#pragma unroll
  for (int w = 0; w < W; ++w) {
    v[w] = all[0][w];
#pragma unroll
    for (int r = 1; r < CTAS; ++r) v[w] += all[r][w];
  }
}
template <int CTAS>
__device__ __forceinline__ float row_max(RowExchange<CTAS, 1>& ex, int turn, float v, float* sh) {
  const float mine[1] = {block_reduce_max(v, sh)};
  float all[CTAS][1];
  row_gather<CTAS, 1>(ex, turn, mine, all);
  v = all[0][0];
#pragma unroll
  for (int r = 1; r < CTAS; ++r) v = fmaxf(v, all[r][0]);
  return v;
}

// Values of the whole row whose key is `least` or more, in the order of their columns, into every CTA's list (`list` has room for
// them); their number. counts: one word per CTA of the cluster, warp_n: one per warp.
static constexpr int kMostKept = 1024;
template <int CTAS, int T>
__device__ __forceinline__ int gather_kept(const RowSlice& s, uint32_t least, float* list, int* counts, int* warp_n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = T / 32, rank = row_rank<CTAS>();
  const int lo = (int)((long long)s.n * warp / warps), hi = (int)((long long)s.n * (warp + 1) / warps);
  int n = 0;
  for (int i = lo; i < hi; i += 32) n += __popc(__ballot_sync(0xffffffffu, i + lane < hi && fkey(s.v[i + lane]) >= least));
  if (lane == 0) warp_n[warp] = n;
  __syncthreads();
  int before = 0, mine = 0;
  for (int w = 0; w < warps; ++w) {
    if (w < warp) before += warp_n[w];
    mine += warp_n[w];
  }
  if constexpr (CTAS > 1) {
    if (threadIdx.x < CTAS) {
      const uint32_t to = mapa_u32(smem_u32(counts + rank), threadIdx.x);
      asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(to), "r"(mine) : "memory");
    }
    cluster_sync_all();
  } else {
    if (threadIdx.x == 0) counts[0] = mine;
    __syncthreads();
  }
  int total = 0;
  for (int r = 0; r < CTAS; ++r) {
    if (r < rank) before += counts[r];
    total += counts[r];
  }
  for (int i = lo; i < hi; i += 32) {
    const bool in = i + lane < hi && fkey(s.v[i + lane]) >= least;
    const uint32_t who = __ballot_sync(0xffffffffu, in);
    const int at = before + __popc(who & ((1u << lane) - 1));
    before += __popc(who);
    if (!in || at >= kMostKept) continue;
    if constexpr (CTAS > 1) {
      for (int r = 0; r < CTAS; ++r)
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_u32(smem_u32(list + at), r)), "f"(s.v[i + lane]) : "memory");
    } else {
      list[at] = s.v[i + lane];
    }
  }
  if constexpr (CTAS > 1) cluster_sync_all();
  else __syncthreads();
  return total;
}

// top-k: radix select of the k-th largest key, two bits a pass (count based). top-p: the same search
// for the largest threshold whose kept mass is >= p. Ties at the threshold are all kept (same as the sort-based rule for
// distinct logits). A pass over the row is bound by its barriers and shared-memory reads, about 2 us, and there are 32 of them; once
// no more than kMostKept values are at or above the top-k search's prefix, every CTA of the cluster gets them all and goes on
// by itself, a fraction of a microsecond a pass. 40 rows of 151936 with k = 50, p = 0.95: 107 us, with all passes over the
// row 264, with a block of 256 threads per row that read the row from L2 for every bit 7717.
template <int CTAS, int T>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(T)
    top_k_top_p_kernel(float* logits, int ld, int V, const int* __restrict__ top_k,
                       const float* __restrict__ top_p) {
  extern __shared__ float4 stage_raw[];
  __shared__ RowExchange<CTAS, 1> ex1;
  __shared__ RowExchange<CTAS, 3> ex3;
  __shared__ RowExchange<1, 1> own1;
  __shared__ RowExchange<1, 3> own3;
  __shared__ float sh1[T / 32][1], sh3[T / 32][3], shm[32];
  __shared__ float list[kMostKept];
  __shared__ int counts[CTAS], warp_n[T / 32];
  const int row = blockIdx.x / CTAS;
  const int k = top_k ? top_k[row] : 0;
  const float pth = top_p ? top_p[row] : 1.f;
  const bool do_k = (k > 0 && k < V);
  const bool do_p = (pth < 1.f);
  if (!do_k && !do_p) return;                          // (the whole cluster)
  const RowSlice s = load_row_slice<CTAS, T>(logits + (size_t)row * ld, V, reinterpret_cast<float*>(stage_raw));
  uint32_t thr_key = 0;
  int turn = 0;
  // what is searched: the CTA's slice, its sums over the cluster, or the row's kept values, its sums within the CTA
  const float* v = s.v;
  int n = s.n;
  constexpr bool kLists = CTAS > 1 || T > 256;         // (the rows that 256 threads pass are as short as a list)
  bool alone = false;
  const auto sum3 = [&](float (&c)[3]) {
    if (kLists && alone) row_sum<1, T, 3>(own3, 0, c, sh3);
    else row_sum<CTAS, T, 3>(ex3, turn++, c, sh3);
  };
  if (do_k) {
    // find the largest key T such that count(key >= T) >= k
    uint32_t prefix = 0;
    float kept = (float)V;
    for (int bit = 30; bit >= 0; bit -= 2) {
      if (kLists && !alone && kept <= (float)kMostKept && (CTAS > 1 || n > 2 * kMostKept)) {
        n = gather_kept<CTAS, T>(s, prefix, list, counts, warp_n);
        v = list;
        alone = true;
      }
      const uint32_t c1 = prefix | (1u << bit), c2 = prefix | (2u << bit), c3 = prefix | (3u << bit);
      int n1 = 0, n2 = 0, n3 = 0;
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += T) {
        const uint32_t kk = fkey(v[i]);
        n1 += kk >= c1; n2 += kk >= c2; n3 += kk >= c3;
      }
      float c[3] = {(float)n1, (float)n2, (float)n3};
      sum3(c);
      if (c[2] >= (float)k) { prefix = c3; kept = c[2]; }
      else if (c[1] >= (float)k) { prefix = c2; kept = c[1]; }
      else if (c[0] >= (float)k) { prefix = c1; kept = c[0]; }
    }
    thr_key = prefix;
  }
  if (do_p) {
    float mx = -FLT_MAX;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += T) {
      const float x = v[i];
      if (fkey(x) >= thr_key) mx = fmaxf(mx, x);
    }
    mx = alone ? row_max<1>(own1, 0, mx, shm) : row_max<CTAS>(ex1, 0, mx, shm);
    float tot[1] = {0.f};
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += T) {
      const float x = v[i];
      if (fkey(x) >= thr_key) tot[0] += __expf(x - mx);
    }
    if (alone) row_sum<1, T, 1>(own1, 1, tot, sh1);
    else row_sum<CTAS, T, 1>(ex1, 1, tot, sh1);
    const float need = pth * tot[0];
    // largest key T (>= thr_key) with mass(key >= T) >= need
    uint32_t prefix = 0;
    for (int bit = 30; bit >= 0; bit -= 2) {
      const uint32_t c1 = prefix | (1u << bit), c2 = prefix | (2u << bit), c3 = prefix | (3u << bit);
      const uint32_t least = c1 > thr_key ? c1 : thr_key;
      float m[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += T) {
        const float x = v[i];
        const uint32_t kk = fkey(x);
        if (kk >= least) {
          const float e = __expf(x - mx);
          m[0] += e;
          m[1] += kk >= c2 ? e : 0.f;
          m[2] += kk >= c3 ? e : 0.f;
        }
      }
      sum3(m);
      if (m[2] >= need) prefix = c3;
      else if (m[1] >= need) prefix = c2;
      else if (m[0] >= need) prefix = c1;
    }
    if (prefix > thr_key) thr_key = prefix;
  }
#pragma unroll 4
  for (int i = threadIdx.x; i < s.n; i += T)
    if (fkey(s.v[i]) < thr_key) s.x[i] = -INFINITY;
}

// ---- softmax / log-softmax (out may alias in) ----
// (40 rows of 151936: 331 us with a block of 256 threads per row, 15 with a cluster.)
template <int CTAS, int T>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(T)
    softmax_kernel(const float* logits, int ld, float* out, int ldo, int V, int log_mode) {
  extern __shared__ float4 stage_raw[];
  __shared__ RowExchange<CTAS, 1> ex;
  __shared__ float sh[T / 32][1], shm[32];
  const int row = blockIdx.x / CTAS;
  const RowSlice s = load_row_slice<CTAS, T>(const_cast<float*>(logits) + (size_t)row * ld, V, reinterpret_cast<float*>(stage_raw));
  float* o = out + (size_t)row * ldo + s.lo;
  float mx = -FLT_MAX;
#pragma unroll 4
  for (int i = threadIdx.x; i < s.n; i += T) mx = fmaxf(mx, s.v[i]);
  mx = row_max<CTAS>(ex, 0, mx, shm);
  float sum[1] = {0.f};
#pragma unroll 4
  for (int i = threadIdx.x; i < s.n; i += T) sum[0] += __expf(s.v[i] - mx);
  row_sum<CTAS, T, 1>(ex, 1, sum, sh);
  if (log_mode) {
    const float lz = mx + logf(sum[0]);
#pragma unroll 4
    for (int i = threadIdx.x; i < s.n; i += T) o[i] = s.v[i] - lz;
  } else {
    const float inv = 1.f / sum[0];
#pragma unroll 4
    for (int i = threadIdx.x; i < s.n; i += T) o[i] = __expf(s.v[i] - mx) * inv;
  }
}

// ---- seeded exponential-race sample: argmax_i p_i / (-log u_i) ----
__host__ __device__ inline uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float race_key(float prob, uint64_t seed, uint64_t step, int col) {
  const uint64_t z = splitmix64(seed ^ splitmix64(step * 0x100000001B3ull + (uint64_t)col));
  const double u = ((double)(z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
  const float e = (float)(-log(u));
  return prob / e;
}
// (40 rows of 151936 dense probabilities: 314 us with a block of 256 threads per row, 52 with a cluster.)
template <int CTAS, int T>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(T)
    random_sample_kernel(const float* __restrict__ probs, int ld, int V,
                         const uint64_t* __restrict__ seeds, const uint64_t* __restrict__ steps,
                         int64_t* out) {
  __shared__ ArgPair sh[32];
  __shared__ RowExchange<CTAS, 2> ex;
  const int row = blockIdx.x / CTAS, per = row_slice_cols(V, CTAS), lo = min(V, row_rank<CTAS>() * per), hi = min(V, lo + per);
  row_sync<CTAS>();                                    // (before the first store into another CTA)
  const float* x = probs + (size_t)row * ld;
  const uint64_t seed = seeds[row], step = steps[row];
  ArgPair a{-FLT_MAX, 0x7fffffff};
#pragma unroll 4
  for (int i = lo + threadIdx.x; i < hi; i += T) {
    const float pr = x[i];
    if (pr > 0.f) a = arg_better(a, ArgPair{race_key(pr, seed, step, i), i});
  }
  a = block_argmax(a, sh);
  const float mine[2] = {a.v, __int_as_float(a.i)};
  float all[CTAS][2];
  row_gather<CTAS, 2>(ex, 0, mine, all);
  if (row_rank<CTAS>() == 0 && threadIdx.x == 0) {
    a = ArgPair{all[0][0], __float_as_int(all[0][1])};
    for (int r = 1; r < CTAS; ++r) a = arg_better(a, ArgPair{all[r][0], __float_as_int(all[r][1])});
    out[row] = (a.i >= V || a.i < 0) ? 0 : a.i;
  }
}

// out[row] = is_greedy ? greedy[row] : random[row]
__global__ void merge_greedy_random_kernel(const int64_t* g, const int64_t* r,
                                           const float* __restrict__ temp, int64_t* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = temp[i] < kEps ? g[i] : r[i];
}

// ---- logprob + rank of chosen tokens from log-softmax rows ----
__global__ void __launch_bounds__(kSB)
    token_rank_kernel(const float* __restrict__ logprobs, int ld, int V,
                      const int64_t* __restrict__ toks, float* out_lp, int* out_rank) {
  __shared__ int shi[32];
  const int row = blockIdx.x;
  const float* x = logprobs + (size_t)row * ld;
  const int64_t t = toks[row];
  const float v = (t >= 0 && t < V) ? x[t] : -INFINITY;
  int c = 0;
  for (int i = threadIdx.x; i < V; i += blockDim.x) c += (x[i] > v);
  c = block_reduce_sum_int(c, shi);
  if (threadIdx.x == 0) {
    out_lp[row] = v;
    out_rank[row] = c + 1;
  }
}

// ---- greedy rejection sampling for speculative decoding ----
// target_argmax: [sum(draft)+n] argmax of the target logits at every draft position plus the
// bonus position; cu: [n+1] prefix offsets of draft tokens. out: [n, max_spec+1], -1 padded.
__global__ void greedy_reject_kernel(const int64_t* __restrict__ target_argmax,
                                     const int64_t* __restrict__ draft,
                                     const int* __restrict__ cu_draft, int n, int max_spec,
                                     int64_t* out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int d0 = cu_draft[r], nd = cu_draft[r + 1] - d0;
  const int t0 = d0 + r;  // target rows: nd draft positions + 1 bonus per request
  int64_t* o = out + (size_t)r * (max_spec + 1);
  for (int i = 0; i <= max_spec; ++i) o[i] = -1;
  int i = 0;
  for (; i < nd; ++i) {
    const int64_t tg = target_argmax[t0 + i];
    o[i] = tg;
    if (tg != draft[d0 + i]) return;  // replacement token emitted, stop
  }
  o[nd] = target_argmax[t0 + nd];  // all accepted: bonus token
}

// ---- async-scheduling input splice ----
// input_ids[dst_idx[i]] = last_sampled[src_row[i]]
__global__ void splice_sampled_kernel(int64_t* input_ids, const int* __restrict__ dst_idx,
                                      const int* __restrict__ src_row,
                                      const int64_t* __restrict__ last_sampled, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) input_ids[dst_idx[i]] = last_sampled[src_row[i]];
}
// last_sampled[row_of[i]] = sampled[i]
__global__ void scatter_sampled_kernel(int64_t* last_sampled, const int* __restrict__ row_of,
                                       const int64_t* __restrict__ sampled, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && row_of[i] >= 0) last_sampled[row_of[i]] = sampled[i];
}

// CTAs of a row. A pass of eight CTAs ends in a cluster barrier, which takes the longer the more clusters there are, one of
// a single CTA reads the whole row: us with one / eight CTAs, and with a block of 256 threads that reads the row from L2
// for every bit. top-k with top-p, 4000 columns: 1 row 32 / 41 (84), 120 rows 34 / 200 (86); 16000: 1 row 69 / 48 (278), 40 rows
// 70 / 111 (282), 120 rows 71 / 236 (283); 32000: 40 rows 119 / 121, 120 rows 122 / 265. Softmax, 1000: 40 rows 3.3 / 5.1
// (3.8); 32000: 40 rows 9.5 / 6.5, 120 rows 10 / 14. The draw's logarithms are a CTA's whole time: 1000: 120 rows 3.9 / 9.5 (4.9);
// 2000: 1 row 6.0 / 3.4, 40 rows 6.4 / 4.5, 80 rows 6.3 / 7.4 (6.4). More rows than SMs need no second CTA each.
static constexpr int kMostOneCta = kMostStaged / 4;       // columns
static int row_ctas(int n, int V, int base, int per_row) {
  return V <= kMostOneCta && (n > b200_num_sms() || V <= base + per_row * n) ? 1 : 8;
}
static size_t row_stage_bytes(int V, int ctas) {
  const size_t bytes = (size_t)row_slice_cols(V, ctas) * 4;
  return bytes <= kMostStaged ? bytes : 0;
}
template <typename... KArgs, typename... Args>
static int launch_rows(void (*kernel)(KArgs...), int n, int ctas, int threads, size_t smem, cudaStream_t stream, PerDeviceOnce& once,
                       Args... args) {
  if (smem > 32 * 1024 && once.first())             // (48 KB with the static part go without)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostStaged);
  kernel<<<n * ctas, threads, smem, stream>>>(args...);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace b200

using namespace b200;
#define RET_LAUNCH return cudaGetLastError() == cudaSuccess ? 0 : -2

extern "C" {

int b200_argmax_blocks_per_row(int n, int V) {
  int target = b200_num_sms() * 2;
  int bpr = (target + n - 1) / n;
  int maxb = (V + 4095) / 4096;
  if (bpr > maxb) bpr = maxb;
  if (bpr < 1) bpr = 1;
  if (bpr > 64) bpr = 64;
  return bpr;
}

// scratch: float[n*64] + int[n*64]
int b200_argmax(const void* logits, int ld, int n, int V, void* out_i64, void* scratch_f,
                void* scratch_i, cudaStream_t stream) {
  if (n <= 0) return 0;
  const int bpr = b200_argmax_blocks_per_row(n, V);
  dim3 grid(bpr, n);
  argmax_partial_kernel<<<grid, kSB, 0, stream>>>((const float*)logits, ld, V, bpr,
                                                  (float*)scratch_f, (int*)scratch_i);
  argmax_final_kernel<<<n, 32, 0, stream>>>((const float*)scratch_f, (const int*)scratch_i, bpr,
                                            (int64_t*)out_i64, V);
  RET_LAUNCH;
}

// Local stage of the vocabulary-parallel argmax: cand_out[n] (8 bytes each) = best (value,
// index_base + column) of this rank's logits[n, V]; columns at or beyond v_valid are ignored
// (padding of the last shard).
int b200_argmax_candidates(const void* logits, int ld, int n, int V, int v_valid, int index_base,
                           void* cand_out, void* scratch_f, void* scratch_i, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (v_valid > V) v_valid = V;
  if (v_valid <= 0) {   // nothing of the vocabulary lives here: candidates that never win
    argmax_candidate_kernel<<<n, 32, 0, stream>>>(nullptr, nullptr, 0, 0, index_base, (int2*)cand_out);
    RET_LAUNCH;
  }
  const int bpr = b200_argmax_blocks_per_row(n, v_valid);
  dim3 grid(bpr, n);
  argmax_partial_kernel<<<grid, kSB, 0, stream>>>((const float*)logits, ld, v_valid, bpr,
                                                  (float*)scratch_f, (int*)scratch_i);
  argmax_candidate_kernel<<<n, 32, 0, stream>>>((const float*)scratch_f, (const int*)scratch_i, bpr, v_valid,
                                                index_base, (int2*)cand_out);
  RET_LAUNCH;
}
// Final stage: cand[world][n] pairs -> out[n] int64 token ids.
int b200_argmax_combine(const void* cand, int n, int world, int V_total, void* out_i64,
                        cudaStream_t stream) {
  if (n <= 0) return 0;
  argmax_combine_kernel<<<(n + 127) / 128, 128, 0, stream>>>((const int2*)cand, n, world, V_total,
                                                             (int64_t*)out_i64);
  RET_LAUNCH;
}

int b200_apply_temperature(void* logits, int ld, int n, int V, const void* temp,
                           cudaStream_t stream) {
  if (n <= 0) return 0;
  dim3 grid(min(64, (V + 255) / 256), n);
  temperature_kernel<<<grid, 256, 0, stream>>>((float*)logits, ld, V, (const float*)temp);
  RET_LAUNCH;
}

int b200_apply_penalties(void* logits, int ld, int V, const void* rows, const void* toks,
                         const void* out_cnt, int n_entries, const void* rep, const void* freq,
                         const void* pres, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  penalties_kernel<<<(n_entries + 255) / 256, 256, 0, stream>>>(
      (float*)logits, ld, V, (const int*)rows, (const int*)toks, (const int*)out_cnt, n_entries,
      (const float*)rep, (const float*)freq, (const float*)pres);
  RET_LAUNCH;
}

int b200_sparse_edit(void* logits, int ld, int V, const void* rows, const void* toks,
                     const void* vals, int n_entries, int mode, cudaStream_t stream) {
  if (n_entries <= 0) return 0;
  sparse_edit_kernel<<<(n_entries + 255) / 256, 256, 0, stream>>>(
      (float*)logits, ld, V, (const int*)rows, (const int*)toks, (const float*)vals, n_entries,
      mode);
  RET_LAUNCH;
}

int b200_apply_bitmask(void* logits, int ld, int V, const void* mask, int n_mask_rows,
                       const void* row_ids, cudaStream_t stream) {
  if (n_mask_rows <= 0) return 0;
  dim3 grid(min(64, (V + 255) / 256), n_mask_rows);
  bitmask_kernel<<<grid, 256, 0, stream>>>((float*)logits, ld, V, (const int32_t*)mask,
                                           (V + 31) / 32, (const int*)row_ids);
  RET_LAUNCH;
}

int b200_apply_min_p(void* logits, int ld, int n, int V, const void* min_p, cudaStream_t stream) {
  if (n <= 0) return 0;
  min_p_kernel<<<n, kSB, 0, stream>>>((float*)logits, ld, V, (const float*)min_p);
  RET_LAUNCH;
}

int b200_apply_top_k_top_p(void* logits, int ld, int n, int V, const void* top_k,
                           const void* top_p, cudaStream_t stream) {
  if (n <= 0) return 0;
  // (up to 1024 columns, a few a thread, 256 threads pass the search's barriers sooner: 256 rows of 256 columns 31 -> 23 us)
  static PerDeviceOnce once[3];
  const int ctas = row_ctas(n, V, 6500, 420), form = ctas == 8 ? 2 : V > 1024 ? 1 : 0;
  return launch_rows(form == 2 ? top_k_top_p_kernel<8, 512> : form ? top_k_top_p_kernel<1, 512> : top_k_top_p_kernel<1, 256>, n,
                     ctas, form ? 512 : 256, row_stage_bytes(V, ctas), stream, once[form], (float*)logits, ld, V,
                     (const int*)top_k, (const float*)top_p);
}

int b200_softmax(const void* logits, int ld, void* out, int ldo, int n, int V, int log_mode,
                 cudaStream_t stream) {
  if (n <= 0) return 0;
  static PerDeviceOnce once[2];
  const int ctas = row_ctas(n, V, 6500, 420);
  return launch_rows(ctas == 8 ? softmax_kernel<8, 512> : softmax_kernel<1, 512>, n, ctas, 512, row_stage_bytes(V, ctas), stream,
                     once[ctas == 8], (const float*)logits, ld, (float*)out, ldo, V, log_mode);
}

int b200_random_sample(const void* probs, int ld, int n, int V, const void* seeds,
                       const void* steps, void* out_i64, cudaStream_t stream) {
  if (n <= 0) return 0;
  static PerDeviceOnce once;
  const int ctas = row_ctas(n, V, 600, 30);
  return launch_rows(ctas == 8 ? random_sample_kernel<8, 512> : random_sample_kernel<1, 512>, n, ctas, 512, 0, stream, once,
                     (const float*)probs, ld, V, (const uint64_t*)seeds, (const uint64_t*)steps, (int64_t*)out_i64);
}

int b200_merge_greedy_random(const void* g, const void* r, const void* temp, void* out, int n,
                             cudaStream_t stream) {
  if (n <= 0) return 0;
  merge_greedy_random_kernel<<<(n + 255) / 256, 256, 0, stream>>>(
      (const int64_t*)g, (const int64_t*)r, (const float*)temp, (int64_t*)out, n);
  RET_LAUNCH;
}

int b200_token_rank(const void* logprobs, int ld, int n, int V, const void* toks, void* out_lp,
                    void* out_rank, cudaStream_t stream) {
  if (n <= 0) return 0;
  token_rank_kernel<<<n, kSB, 0, stream>>>((const float*)logprobs, ld, V, (const int64_t*)toks,
                                           (float*)out_lp, (int*)out_rank);
  RET_LAUNCH;
}

int b200_greedy_reject(const void* target_argmax, const void* draft, const void* cu_draft, int n,
                       int max_spec, void* out, cudaStream_t stream) {
  if (n <= 0) return 0;
  greedy_reject_kernel<<<(n + 127) / 128, 128, 0, stream>>>(
      (const int64_t*)target_argmax, (const int64_t*)draft, (const int*)cu_draft, n, max_spec,
      (int64_t*)out);
  RET_LAUNCH;
}

int b200_splice_sampled(void* input_ids, const void* dst_idx, const void* src_row,
                        const void* last_sampled, int n, cudaStream_t stream) {
  if (n <= 0) return 0;
  splice_sampled_kernel<<<(n + 255) / 256, 256, 0, stream>>>(
      (int64_t*)input_ids, (const int*)dst_idx, (const int*)src_row, (const int64_t*)last_sampled,
      n);
  RET_LAUNCH;
}
int b200_scatter_sampled(void* last_sampled, const void* row_of, const void* sampled, int n,
                         cudaStream_t stream) {
  if (n <= 0) return 0;
  scatter_sampled_kernel<<<(n + 255) / 256, 256, 0, stream>>>(
      (int64_t*)last_sampled, (const int*)row_of, (const int64_t*)sampled, n);
  RET_LAUNCH;
}

uint64_t b200_splitmix64(uint64_t z) { return splitmix64(z); }

}  // extern "C"
