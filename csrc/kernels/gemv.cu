// bf16 products of one or two rows  C[M,N] = A[M,K] * W[N,K]^T  on the CUDA cores, and the same with the residual addition
// and RMSNorm of the row in front.
//
// A single request's step is a chain of such products, each a few microseconds of weights; what bounds it is what comes
// after the predecessor's last store: start-up, first loads, exchange, last store. This form keeps that short. A warp
// multiplies two weight rows (with a gated activation: the gate and the up row of one output) straight from registers, the
// first of which are loaded while the predecessor still runs; nothing is exchanged but warp sums, and a split over K stays
// within a block. At two multiply-adds a weight the CUDA cores keep up with HBM (about a third of their issue slots per
// row); from three rows on the tensor cores' form (gemm_cluster.cu) is the faster one.
//
// Every block normalises the row for itself (16 KB from L2 at a width of 4096), which costs less than a kernel boundary; the
// sum with the residual is stored once, to another buffer than the one it is read from.
//
// Measured on B200 (chained launches of one row over weights beyond L2, us, against the cluster kernel):
//   4096 x 1024  5.4 -> 2.8    1024 x 2048  4.5 -> 2.8    6144 x 1024  6.0 -> 3.5    1024 x 3072  5.3 -> 3.1
//   6144 x 4096 10.9 -> 9.6    4096 x 4096  8.4 -> 8.5    28672 x 4096 38.8 -> 38.9  128256 x 4096 155 -> 151
// One token of the 0.6B shape, a block of six launches instead of eight: 27.8 -> 17.4 ms for 24 tokens.
#include "api.h"
#include "sm100.cuh"

namespace b200 {

static constexpr int kVThreads = 256, kVWarps = 8;
static constexpr int kVChunk = 256;        // k-elements of a warp's load: 16 bytes a lane
static constexpr int kVAhead = 4;          // chunks of both rows on the way

struct GemvParams {
  int N, K;
  const __nv_bfloat16 *A, *W;
  long long lda, ldw, ldo;
  int ksplit;                // warps that share two rows (1, 2, 4, 8)
  int groups;                // pairs of rows (gated: outputs), over the pairs of a block
  int gated;                 // 1 + kind; W rows in blocks of [128 gate | 128 up]
  void* out;
  int out_f32, act, w_early;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  // norm in front (norm_w set): rows of K = A (+ res_in), stored to res_out, then RMSNorm
  const __nv_bfloat16 *norm_w, *res_in;
  __nv_bfloat16* res_out;
  float eps;
  int gemma;
};

__device__ __forceinline__ uint4 ld_weights(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

template <int M>
__global__ void __launch_bounds__(kVThreads, 3) gemv_kernel(GemvParams p) {
  extern __shared__ uint4 act_raw[];                       // [M][K] bf16
  __shared__ float part[kVWarps][2 * M];
  __shared__ float norm_sum[M][kVWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_block = kVWarps / p.ksplit, ks = warp % p.ksplit, pair = warp / p.ksplit;
  const int chunks = (p.K + kVChunk - 1) / kVChunk;
  const int c0 = chunks * ks / p.ksplit, c1 = chunks * (ks + 1) / p.ksplit;

  // weight rows of group g: r0, r1 (a row past the end repeats the last one)
  auto rows_of = [&](int g, const __nv_bfloat16*& w0, const __nv_bfloat16*& w1) {
    int r0, r1;
    const int i = g * per_block + pair;
    if (p.gated) {
      const int o = min(i, p.N / 2 - 1);
      r0 = (o >> 7) * 256 + (o & 127);
      r1 = r0 + 128;
    } else {
      r0 = min(2 * i, p.N - 1);
      r1 = min(2 * i + 1, p.N - 1);
    }
    w0 = p.W + (long long)r0 * p.ldw + lane * 8;
    w1 = p.W + (long long)r1 * p.ldw + lane * 8;
  };
  uint4 a0[kVAhead], a1[kVAhead];
  auto fetch = [&](const __nv_bfloat16* x0, const __nv_bfloat16* x1, int c, uint4& v0, uint4& v1) {
    const bool in = c < c1 && c * kVChunk + lane * 8 < p.K;                      // K is a multiple of 8
    v0 = in ? ld_weights(x0 + c * kVChunk) : make_uint4(0, 0, 0, 0);
    v1 = in ? ld_weights(x1 + c * kVChunk) : make_uint4(0, 0, 0, 0);
  };

  const __nv_bfloat16 *w0, *w1;
  int g = blockIdx.x;
  rows_of(g, w0, w1);
  if (p.w_early)
#pragma unroll
    for (int u = 0; u < kVAhead; ++u) fetch(w0, w1, c0 + u, a0[u], a1[u]);
  pdl_wait();
  pdl_launch_dependents();
  if (!p.w_early)
#pragma unroll
    for (int u = 0; u < kVAhead; ++u) fetch(w0, w1, c0 + u, a0[u], a1[u]);

  // the rows of the batch, normed where asked for, into shared memory
  const int nv = p.K >> 3;
  if (p.norm_w) {
    float ss[M];
#pragma unroll
    for (int m = 0; m < M; ++m) ss[m] = 0.f;
    for (int i = threadIdx.x; i < nv; i += kVThreads) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        uint4 v = reinterpret_cast<const uint4*>(p.A + m * p.lda)[i];
        if (p.res_in) {
          const uint4 r = reinterpret_cast<const uint4*>(p.res_in + (long long)m * p.K)[i];
          float x[8], y[8];
          unpack8(v, x);
          unpack8(r, y);
          v = make_uint4(pack_bf16x2(x[0] + y[0], x[1] + y[1]), pack_bf16x2(x[2] + y[2], x[3] + y[3]),
                         pack_bf16x2(x[4] + y[4], x[5] + y[5]), pack_bf16x2(x[6] + y[6], x[7] + y[7]));
        }
        if (blockIdx.x == 0) reinterpret_cast<uint4*>(p.res_out + (long long)m * p.K)[i] = v;
        act_raw[m * nv + i] = v;
        const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {                 // (sums in rmsnorm_kernel's order: the same bits)
          const float2 f = unpack_bf16x2(q[e]);
          ss[m] += f.x * f.x + f.y * f.y;
        }
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
      if (lane == 0) norm_sum[m][warp] = ss[m];
    }
    __syncthreads();
    float inv[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float t = lane < kVWarps ? norm_sum[m][lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      inv[m] = rsqrtf(t / (float)p.K + p.eps);
    }
    const float one = p.gemma ? 1.f : 0.f;
    for (int i = threadIdx.x; i < nv; i += kVThreads) {                 // (each thread reads what it wrote)
      float w[8];
      unpack8(reinterpret_cast<const uint4*>(p.norm_w)[i], w);
#pragma unroll
      for (int m = 0; m < M; ++m) {
        float x[8];
        unpack8(act_raw[m * nv + i], x);
        act_raw[m * nv + i] = make_uint4(
            pack_bf16x2(x[0] * inv[m] * (w[0] + one), x[1] * inv[m] * (w[1] + one)),
            pack_bf16x2(x[2] * inv[m] * (w[2] + one), x[3] * inv[m] * (w[3] + one)),
            pack_bf16x2(x[4] * inv[m] * (w[4] + one), x[5] * inv[m] * (w[5] + one)),
            pack_bf16x2(x[6] * inv[m] * (w[6] + one), x[7] * inv[m] * (w[7] + one)));
      }
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += kVThreads)
#pragma unroll
      for (int m = 0; m < M; ++m) act_raw[m * nv + i] = reinterpret_cast<const uint4*>(p.A + m * p.lda)[i];
  }
  __syncthreads();

  while (g < p.groups) {
    float s0[M], s1[M];
#pragma unroll
    for (int m = 0; m < M; ++m) s0[m] = s1[m] = 0.f;
    for (int c = c0; c < c1; c += kVAhead) {
      const bool last = c + kVAhead >= c1;                // then the next rows' first chunks are fetched
      int next = c + kVAhead;
      if (last && g + (int)gridDim.x < p.groups) {
        rows_of(g + gridDim.x, w0, w1);
        next = c0;
      }
#pragma unroll
      for (int u = 0; u < kVAhead; ++u) {
        const uint4 b0 = a0[u], b1 = a1[u];
        fetch(w0, w1, next + u, a0[u], a1[u]);
        const int k8 = (c + u) * (kVChunk / 8) + lane;
        if (c + u >= c1 || k8 >= nv) continue;
        float f0[8], f1[8];
        unpack8(b0, f0);
        unpack8(b1, f1);
#pragma unroll
        for (int m = 0; m < M; ++m) {
          float x[8];
          unpack8(act_raw[m * nv + k8], x);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            s0[m] = fmaf(f0[e], x[e], s0[m]);
            s1[m] = fmaf(f1[e], x[e], s1[m]);
          }
        }
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        s0[m] += __shfl_xor_sync(0xffffffffu, s0[m], o);
        s1[m] += __shfl_xor_sync(0xffffffffu, s1[m], o);
      }
    if (p.ksplit > 1) {
      __syncthreads();                                    // (the last pair's sums have been read)
      if (lane == 0)
#pragma unroll
        for (int m = 0; m < M; ++m) { part[warp][2 * m] = s0[m]; part[warp][2 * m + 1] = s1[m]; }
      __syncthreads();
      if (ks == 0)
#pragma unroll
        for (int m = 0; m < M; ++m)
          for (int w = 1; w < p.ksplit; ++w) { s0[m] += part[warp + w][2 * m]; s1[m] += part[warp + w][2 * m + 1]; }
    }
    if (ks == 0 && lane < M) {
      float v0 = s0[0], v1 = s1[0];
#pragma unroll
      for (int m = 1; m < M; ++m)
        if (lane == m) { v0 = s0[m]; v1 = s1[m]; }
      const int i = g * per_block + pair;
      if (p.gated) {
        if (i < p.N / 2) {
          const float gg = __bfloat162float(__float2bfloat16(v0)), uu = __bfloat162float(__float2bfloat16(v1));
          reinterpret_cast<__nv_bfloat16*>(p.out)[lane * p.ldo + i] = __float2bfloat16(act_of(gg, p.gated - 1) * uu);
        }
      } else if (2 * i < p.N) {                           // N is even
        const long long at = lane * p.ldo + 2 * i;
        if (p.bias) { v0 += __bfloat162float(p.bias[2 * i]); v1 += __bfloat162float(p.bias[2 * i + 1]); }
        if (p.residual) {
          v0 += __bfloat162float(p.residual[lane * p.ldr + 2 * i]);
          v1 += __bfloat162float(p.residual[lane * p.ldr + 2 * i + 1]);
        }
        v0 = act_epilogue<true>(v0, p.act);
        v1 = act_epilogue<true>(v1, p.act);
        if (p.out_f32) *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.out) + at) = make_float2(v0, v1);
        else *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.out) + at) = pack_bf16x2(v0, v1);
      }
    }
    g += gridDim.x;
  }
}

// One row: all but the longest K, where the cluster kernel's deeper ring keeps HBM busier (4096 x 14336: 22.2 against 23.7
// us). Two rows: small matrices (1024 x 3072 5.3 -> 3.6 us, 5120 x 2048 7.2 -> 5.7; 4096 x 4096 8.5 against 9.5). A block that
// takes several pairs of rows in turn pays for each turn's first loads, which a short K does not cover (us, this kernel / the
// cluster kernel: 6144 x 256, one turn, 2.4 / 3.5; 8192 x 128 3.8 / 2.8; 14336 x 256 5.3 / 3.6; 16376 x 512, three, 6.2 / 6.3;
// 24576 x 512, four, 7.9 / 6.6; 57344 x 1024 22.6 / 24.6; two rows: 12288 x 512 5.0 / 5.9, 16376 x 512 6.8 / 6.3).
bool gemv_takes(int M, int N, int K) {
  if (M < 1 || M > 2 || K > 8192 || (M == 2 && (long long)N * K > (12 << 20))) return false;
  const long long warps = 3LL * b200_num_sms() * kVWarps, turns = ((N + 1) / 2 + warps - 1) / warps;
  return turns == 1 || K >= 1024 || (K >= 512 && turns <= 4 - M);
}

int launch_gemv(const GemmCluster& g, const GemvNorm* norm, cudaStream_t stream) {
  if (!gemv_takes(g.M, g.N, g.K) || (g.K & 7) || (g.gated && (g.N & 255))) return -1;
  GemvParams p{};
  p.N = g.N; p.K = g.K;
  p.A = (const __nv_bfloat16*)g.A; p.W = (const __nv_bfloat16*)g.W;
  p.lda = g.lda; p.ldw = g.ldw; p.ldo = g.ldo;
  p.gated = g.gated; p.out = g.out; p.out_f32 = g.out_f32; p.act = g.act; p.w_early = g.w_early;
  p.bias = (const __nv_bfloat16*)g.bias; p.residual = (const __nv_bfloat16*)g.residual; p.ldr = g.ldr;
  if (norm) {
    p.norm_w = (const __nv_bfloat16*)norm->weight; p.res_in = (const __nv_bfloat16*)norm->res_in;
    p.res_out = (__nv_bfloat16*)norm->res_out; p.eps = norm->eps; p.gemma = norm->gemma;
  }
  // 24 warps an SM are resident. Few rows: several warps share a pair, each with at least two chunks of K
  const int blocks = 3 * b200_num_sms(), pairs = g.gated ? g.N / 2 : (g.N + 1) / 2, chunks = (g.K + kVChunk - 1) / kVChunk;
  p.ksplit = 1;
  while (p.ksplit < kVWarps && (long long)pairs * p.ksplit * 2 <= (long long)blocks * kVWarps && chunks >= 4 * p.ksplit) p.ksplit *= 2;
  const int per_block = kVWarps / p.ksplit;
  p.groups = (pairs + per_block - 1) / per_block;
  const int turns = (p.groups + blocks - 1) / blocks;                 // every block takes about as many
  const int grid = (p.groups + turns - 1) / turns;
  const size_t smem = (size_t)g.M * g.K * 2;            // (at most 32 KB)
  auto kernel = g.M == 1 ? gemv_kernel<1> : gemv_kernel<2>;
  return launch_pdl(kernel, dim3(grid), dim3(kVThreads), smem, stream, p) == cudaSuccess ? 0 : -2;
}

}  // namespace b200
