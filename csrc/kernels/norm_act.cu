// Row-wise normalisation and element-wise activation kernels (HBM-bound; every access is a
// 16-byte vector, one pass over the data, fp32 math, bf16 storage).
//
//   rmsnorm / fused residual-add + rmsnorm (std and gemma "1+w")   reference:
//       src/vt/cuda/cuda_ops.cu:63 (RmsNormRowKernel), :165 (RmsNormRowFastKernel)
//   layernorm                                                      cuda_layernorm.cu:68
//   silu_and_mul, gelu_tanh_and_mul, relu, add, mul_scalar, softcap, casts
//       cuda_ops.cu:417,463,510,550; cuda_layernorm.cu:164,200; cuda_glue.cu:47-100
//   embedding gather with a bounds flag in the status word         cuda_ops.cu:600
//   gather_rows (logits-row gather before lm_head)
#include "api.h"
#include "quant_codec.cuh"
#include "sm100.cuh"

namespace b200 {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

// A row's norm: V vectors a thread (0: as many as it takes, through shared memory), all of whose loads - the row, the residual, the
// weights - are on their way before the first is used. Few rows are bound by such round trips to L2, many by memory. us, chained, against a
// loop over the vectors: 13 rows of 4096 2.4 -> 1.8, of 7168 3.4 -> 2.2; 8192 rows of 2048 23.9 -> 19.0 (7.1 TB/s), of 4096 44.0 -> 40.6.
__device__ __forceinline__ uint4 add_bf16x8(const uint4& x, const uint4& r) {
  const uint32_t p[4] = {x.x, x.y, x.z, x.w}, q[4] = {r.x, r.y, r.z, r.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = unpack_bf16x2(p[j]), b = unpack_bf16x2(q[j]);
    o[j] = pack_bf16x2(a.x + b.x, a.y + b.y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ float add_squares(float ss, const uint4& v) {
  const uint32_t p[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(p[j]);
    ss += f.x * f.x + f.y * f.y;
  }
  return ss;
}
__device__ __forceinline__ uint4 scale_bf16x8(const uint4& v, float inv, const uint4& w, float g) {
  const uint32_t p[4] = {v.x, v.y, v.z, v.w}, q[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = unpack_bf16x2(p[j]), b = unpack_bf16x2(q[j]);
    o[j] = pack_bf16x2(a.x * inv * (b.x + g), a.y * inv * (b.y + g));
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// RMSNorm of row t; every normed vector i of the calling thread goes to put(i, value).
template <int V, typename Put>
__device__ __forceinline__ void norm_row(const uint4* __restrict__ xr, uint4* rr, const uint4* __restrict__ wr, uint4* row_cache, float* red,
                                         int nv, float width, float eps, float g, Put&& put) {
  float ss = 0.f;
  if constexpr (V > 0) {
    uint4 v[V], r[V], w[V];
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if (i < nv) {
        v[j] = xr[i];
        if (rr) r[j] = rr[i];
        w[j] = wr[i];
      }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if (i < nv) {
        if (rr) rr[i] = v[j] = add_bf16x8(v[j], r[j]);
        ss = add_squares(ss, v[j]);
      }
    }
    const float inv = rsqrtf(block_sum(ss, red) / width + eps);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if (i < nv) put(i, scale_bf16x8(v[j], inv, w[j], g));
    }
  } else {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      uint4 v = xr[i];
      if (rr) rr[i] = v = add_bf16x8(v, rr[i]);
      row_cache[i] = v;
      ss = add_squares(ss, v);
    }
    const float inv = rsqrtf(block_sum(ss, red) / width + eps);
    for (int i = threadIdx.x; i < nv; i += blockDim.x) put(i, scale_bf16x8(row_cache[i], inv, wr[i], g));
  }
}
static inline int norm_vectors(int width, int threads) {
  const int v = (width / 8 + threads - 1) / threads;
  return v <= 2 ? v : v <= 4 ? 4 : 0;
}

// x: [T, H] bf16 (row stride ldx). If residual != nullptr: residual += x (bf16-rounded) and
// the norm is taken over the updated residual. out may alias x.
template <int V>
__global__ void __launch_bounds__(256)
    rmsnorm_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* residual,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* out, int ldo, int H,
                   float eps, int gemma) {
  __shared__ float red[32];
  extern __shared__ uint4 row_cache[];  // (V = 0) H/8 vectors
  pdl_wait();                 // predecessor grid complete, its writes visible
  pdl_launch_dependents();    // the successor may become resident (it waits the same way)
  const int t = blockIdx.x;
  uint4* orow = reinterpret_cast<uint4*>(out + (size_t)t * ldo);
  norm_row<V>(reinterpret_cast<const uint4*>(x + (size_t)t * ldx),
              residual ? reinterpret_cast<uint4*>(residual + (size_t)t * H) : nullptr, reinterpret_cast<const uint4*>(w), row_cache, red,
              H >> 3, (float)H, eps, gemma ? 1.f : 0.f, [&](int i, const uint4& o) { orow[i] = o; });
}

// LayerNorm with affine weight and optional bias; scalar loop (any H).
__global__ void __launch_bounds__(256)
    layernorm_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                     const __nv_bfloat16* __restrict__ b, __nv_bfloat16* out, int H, float eps) {
  __shared__ float red[32];
  const int t = blockIdx.x;
  const __nv_bfloat16* xr = x + (size_t)t * H;
  float s = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) s += __bfloat162float(xr[i]);
  const float mean = block_sum(s, red) / (float)H;
  float v = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float d = __bfloat162float(xr[i]) - mean;
    v += d * d;
  }
  const float inv = rsqrtf(block_sum(v, red) / (float)H + eps);
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float y = (__bfloat162float(xr[i]) - mean) * inv * __bfloat162float(w[i]);
    if (b) y += __bfloat162float(b[i]);
    out[(size_t)t * H + i] = __float2bfloat16(y);
  }
}

// x: [T, 2*I] = [gate | up] (or, with kind | 0x100, blocks of [128 gate | 128 up]);
// out: [T, I] = act(gate) * up.
__global__ void __launch_bounds__(256)
    act_and_mul_kernel(const __nv_bfloat16* __restrict__ x, int ldx, __nv_bfloat16* out, int I,
                       int T, int kind_flags) {
  pdl_wait();                 // predecessor grid complete, its writes visible
  pdl_launch_dependents();    // the successor may become resident (it waits the same way)
  const int kind = kind_flags & 0xff;
  const bool il = (kind_flags & 0x100) != 0;
  const int nv = I >> 3;
  const size_t total = (size_t)T * nv;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int t = (int)(idx / nv), i = (int)(idx % nv);
    // interleaved input: blocks of [128 gate | 128 up] instead of [all gate | all up]
    const int goff = il ? ((i * 8) >> 7) * 256 + ((i * 8) & 127) : i * 8;
    const int uoff = il ? goff + 128 : I + i * 8;
    const uint4 g = *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + goff);
    const uint4 u = *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + uoff);
    uint4 o;
    float2 a, b;
    a = unpack_bf16x2(g.x); b = unpack_bf16x2(u.x); o.x = pack_bf16x2(act_of(a.x, kind) * b.x, act_of(a.y, kind) * b.y);
    a = unpack_bf16x2(g.y); b = unpack_bf16x2(u.y); o.y = pack_bf16x2(act_of(a.x, kind) * b.x, act_of(a.y, kind) * b.y);
    a = unpack_bf16x2(g.z); b = unpack_bf16x2(u.z); o.z = pack_bf16x2(act_of(a.x, kind) * b.x, act_of(a.y, kind) * b.y);
    a = unpack_bf16x2(g.w); b = unpack_bf16x2(u.w); o.w = pack_bf16x2(act_of(a.x, kind) * b.x, act_of(a.y, kind) * b.y);
    *reinterpret_cast<uint4*>(out + (size_t)t * I + i * 8) = o;
  }
}

// Row-wise dynamic fp8: each token row gets its own scale (max|v| / 448), written to scales[t]
// for the GEMM's epilogue, and the producer of the row runs in the same pass:
//   mode 0  v = x
//   mode 1  v = RMSNorm(x (+ residual, written back)) -- the arithmetic of rmsnorm_kernel, so the
//           normalised row has the bytes the bf16 path would hand to its GEMM
//   mode 2  v = act(gate) * up from [gate | up] rows (kind_flags as act_and_mul_kernel takes them)
// The row (bf16) stays in shared memory between the producer and the quantisation. One kernel per mode and activation,
// packed maxima and conversions: bound by instructions, then by memory (8192 rows, us: plain 4096 31.0 -> 21.9, 4.6 TB/s;
// act 14336 163 -> 145 with the SiLU that needs no general division).
template <int MODE, int KIND, int V = 0>
__global__ void __launch_bounds__(MODE == 1 ? 256 : 1024)
    rowquant_fp8_kernel(const __nv_bfloat16* __restrict__ x, long ldx, __nv_bfloat16* residual,
                        const __nv_bfloat16* __restrict__ w, float eps, int gemma, int interleaved,
                        uint8_t* __restrict__ out, long ldo, float* __restrict__ scales, int K) {
  __shared__ float red[32];
  extern __shared__ uint4 row_cache[];  // K/8 vectors
  pdl_wait();
  pdl_launch_dependents();
  const long t = blockIdx.x;
  const int nv = K >> 3;
  // (maximum of magnitudes in packed bf16: exact, NaNs drop out as with fmaxf)
  __nv_bfloat162 amax2 = __floats2bfloat162_rn(0.f, 0.f);
  auto vec_amax = [&](const uint4& v) {
    const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) amax2 = __hmax2(amax2, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w4[j])));
  };
  if constexpr (MODE == 1) {
    norm_row<V>(reinterpret_cast<const uint4*>(x + t * ldx), residual ? reinterpret_cast<uint4*>(residual + t * (long)K) : nullptr,
                reinterpret_cast<const uint4*>(w), row_cache, red, nv, (float)K, eps, gemma ? 1.f : 0.f, [&](int i, const uint4& o) {
                  row_cache[i] = o;
                  vec_amax(o);
                });
  } else if constexpr (MODE == 2) {
    const bool il = interleaved != 0;
#pragma unroll 2
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      const int goff = il ? ((i * 8) >> 7) * 256 + ((i * 8) & 127) : i * 8;
      const int uoff = il ? goff + 128 : K + i * 8;
      const uint4 gt = __ldg(reinterpret_cast<const uint4*>(x + t * ldx + goff));
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(x + t * ldx + uoff));
      uint4 o;
      float2 a, b;
      a = unpack_bf16x2(gt.x); b = unpack_bf16x2(u.x); o.x = pack_bf16x2(act_of(a.x, KIND) * b.x, act_of(a.y, KIND) * b.y);
      a = unpack_bf16x2(gt.y); b = unpack_bf16x2(u.y); o.y = pack_bf16x2(act_of(a.x, KIND) * b.x, act_of(a.y, KIND) * b.y);
      a = unpack_bf16x2(gt.z); b = unpack_bf16x2(u.z); o.z = pack_bf16x2(act_of(a.x, KIND) * b.x, act_of(a.y, KIND) * b.y);
      a = unpack_bf16x2(gt.w); b = unpack_bf16x2(u.w); o.w = pack_bf16x2(act_of(a.x, KIND) * b.x, act_of(a.y, KIND) * b.y);
      row_cache[i] = o;
      vec_amax(o);
    }
  } else {
    const uint4* xr = reinterpret_cast<const uint4*>(x + t * ldx);
#pragma unroll 2
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      const uint4 v = __ldg(xr + i);
      row_cache[i] = v;
      vec_amax(v);
    }
  }
  float amax = fmaxf(__low2float(amax2), __high2float(amax2));
  // block maximum (every thread re-reads only the vectors it wrote, so no barrier is needed for
  // row_cache itself)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) red[warp] = amax;
  __syncthreads();
  float m = (lane < nw) ? red[lane] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  const float sc = fmaxf(m, 1e-12f) / 448.f;
  const float is = 1.f / sc;
  if (threadIdx.x == 0) scales[t] = sc;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const uint4 v = row_cache[i];
    const uint32_t wds[4] = {v.x, v.y, v.z, v.w};
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack_bf16x2(wds[j]);
      const uint32_t two = __nv_cvt_float2_to_fp8x2(make_float2(f.x * is, f.y * is), __NV_SATFINITE, __NV_E4M3);
      if (j < 2) lo |= two << (16 * j); else hi |= two << (16 * (j - 2));
    }
    *reinterpret_cast<uint2*>(out + t * ldo + (long)i * 8) = make_uint2(lo, hi);
  }
}

enum EwKind : int { kEwAdd = 0, kEwRelu = 1, kEwMulScalar = 2, kEwSoftcap = 3, kEwSigmoidMul = 4,
                    kEwMul = 5 };

// Generic bf16 element-wise op over n elements (n % 8 == 0). b may be null.
__global__ void __launch_bounds__(256)
    eltwise_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                   __nv_bfloat16* out, size_t n, int kind, float scalar) {
  const size_t nv = n >> 3;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < nv;
       idx += (size_t)gridDim.x * blockDim.x) {
    uint4 va = reinterpret_cast<const uint4*>(a)[idx];
    uint4 vb = b ? reinterpret_cast<const uint4*>(b)[idx] : make_uint4(0, 0, 0, 0);
    uint32_t* pa = reinterpret_cast<uint32_t*>(&va);
    uint32_t* pb = reinterpret_cast<uint32_t*>(&vb);
    uint4 vo;
    uint32_t* po = reinterpret_cast<uint32_t*>(&vo);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 x = unpack_bf16x2(pa[j]), y = unpack_bf16x2(pb[j]), r;
      switch (kind) {
        case kEwAdd: r.x = x.x + y.x; r.y = x.y + y.y; break;
        case kEwRelu: r.x = fmaxf(x.x, 0.f); r.y = fmaxf(x.y, 0.f); break;
        case kEwMulScalar: r.x = x.x * scalar; r.y = x.y * scalar; break;
        case kEwSoftcap: r.x = scalar * tanhf(x.x / scalar); r.y = scalar * tanhf(x.y / scalar); break;
        case kEwSigmoidMul:  // a * sigmoid(b)
          r.x = x.x / (1.f + __expf(-y.x)); r.y = x.y / (1.f + __expf(-y.y)); break;
        default: r.x = x.x * y.x; r.y = x.y * y.y; break;
      }
      po[j] = pack_bf16x2(r.x, r.y);
    }
    reinterpret_cast<uint4*>(out)[idx] = vo;
  }
}

__global__ void cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ a, float* out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = __bfloat162float(a[i]);
}
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ a, __nv_bfloat16* out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(a[i]);
}

// out[t, :] = table[ids[t], :] * scale; an id outside [0, vocab) writes zeros and flags the
// status word (no allocation, no sync: safe inside CUDA graphs). With vocab sharding
// (vocab_start > 0 or a partial table) rows outside the shard are zero without a flag.
__global__ void __launch_bounds__(128)
    embedding_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                     __nv_bfloat16* out, int H, int64_t vocab_start, int64_t vocab_rows,
                     int64_t vocab_total, float scale, int* status) {
  const int t = blockIdx.x;
  const int64_t id = ids[t];
  const int nv = H >> 3;
  uint4* o = reinterpret_cast<uint4*>(out + (size_t)t * H);
  const int64_t local = id - vocab_start;
  if (id < 0 || id >= vocab_total) {
    if (threadIdx.x == 0 && status) atomicExch(status, (int)kErrBadArg);
  }
  if (local < 0 || local >= vocab_rows || id < 0 || id >= vocab_total) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) o[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)local * H);
  if (scale == 1.f) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) o[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      uint4 v = src[i];
      float2 f;
      f = unpack_bf16x2(v.x); v.x = pack_bf16x2(f.x * scale, f.y * scale);
      f = unpack_bf16x2(v.y); v.y = pack_bf16x2(f.x * scale, f.y * scale);
      f = unpack_bf16x2(v.z); v.z = pack_bf16x2(f.x * scale, f.y * scale);
      f = unpack_bf16x2(v.w); v.w = pack_bf16x2(f.x * scale, f.y * scale);
      o[i] = v;
    }
  }
}

// out[i, :] = x[idx[i], :]  (rows of `bytes_per_row` bytes, multiple of 16)
__global__ void __launch_bounds__(128)
    gather_rows_kernel(const uint8_t* __restrict__ x, const int32_t* __restrict__ idx,
                       uint8_t* out, int row_bytes, int n_src) {
  const int i = blockIdx.x;
  int s = idx[i];
  if (s < 0 || s >= n_src) s = 0;
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)s * row_bytes);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)i * row_bytes);
  for (int j = threadIdx.x; j < (row_bytes >> 4); j += blockDim.x) dst[j] = src[j];
}

static inline int ew_grid(size_t work_items) {
  size_t b = (work_items + 255) / 256;
  size_t cap = (size_t)b200_num_sms() * 16;
  return (int)(b < cap ? (b ? b : 1) : cap);
}

}  // namespace b200

using namespace b200;
typedef __nv_bfloat16 bf16;

extern "C" {

int b200_rmsnorm(const void* x, int ldx, void* residual, const void* w, void* out, int ldo, int T,
                 int H, float eps, int gemma, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((H & 7) || (ldx & 7) || (ldo & 7) || H > 32768) return -1;
  int threads = H / 8 >= 256 ? 256 : ((H / 8 + 31) / 32) * 32;
  if (threads < 32) threads = 32;
  const int v = norm_vectors(H, threads);
  auto kernel = v == 1 ? rmsnorm_kernel<1> : v == 2 ? rmsnorm_kernel<2> : v == 4 ? rmsnorm_kernel<4> : rmsnorm_kernel<0>;
  return launch_pdl(kernel, dim3(T), dim3(threads), v ? 0 : (size_t)H * 2, stream, (const bf16*)x, ldx,
                    (bf16*)residual, (const bf16*)w, (bf16*)out, ldo, H, eps, gemma) == cudaSuccess ? 0 : -2;
}

// x: mode 0 / 1 rows of K values, mode 2 rows of [gate | up] (2K values). out: fp8 [T, K] (row
// stride ldo bytes), scales: fp32 [T]. Launched with the thread count b200_rmsnorm uses for this
// width, so that mode 1 sums in the same order.
int b200_quant_fp8_rowwise(const void* x, long ldx, void* residual, const void* norm_w, float eps, int gemma,
                           int mode, int kind_flags, void* out, long ldo, void* scales, int T, int K,
                           cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((K & 7) || (ldx & 7) || (ldo & 7) || K > 32768 || mode < 0 || mode > 2) return -1;
  if (((uintptr_t)x & 15) || ((uintptr_t)out & 7) || (mode == 1 && !norm_w)) return -1;
  if (mode == 2 && (kind_flags & 0x100) && (K & 127)) return -1;
  // Few rows leave SMs idle and are bound by the latency of a thread's loads: up to 1024 threads a row (32 rows, act
  // 14336: 7.8 -> 4.5 us); beyond two rows an SM the other rows cover it. Mode 1 adds in rmsnorm_kernel's order: 256.
  const int most = mode == 1 || T > 2 * b200_num_sms() ? 256 : 1024;
  int threads = K / 8 >= most ? most : ((K / 8 + 31) / 32) * 32;
  if (threads < 32) threads = 32;
  const int kind = kind_flags & 0xff;
  const int v = norm_vectors(K, threads);
  auto kernel = mode == 0 ? rowquant_fp8_kernel<0, 0>
              : mode == 1 ? (v == 1 ? rowquant_fp8_kernel<1, 0, 1> : v == 2 ? rowquant_fp8_kernel<1, 0, 2> : v == 4 ? rowquant_fp8_kernel<1, 0, 4>
                                                                                                         : rowquant_fp8_kernel<1, 0, 0>)
              : kind == kSilu ? rowquant_fp8_kernel<2, kSilu> : kind == kGeluTanh ? rowquant_fp8_kernel<2, kGeluTanh>
                                                                                  : rowquant_fp8_kernel<2, kGeluErf>;
  static PerDeviceOnce attr_once[9];
  if (attr_once[mode == 0 ? 0 : mode == 1 ? 1 + v : kind == kSilu ? 6 : kind == kGeluTanh ? 7 : 8].first())
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 32768 * 2);
  return launch_pdl(kernel, dim3(T), dim3(threads), (size_t)K * 2, stream, (const bf16*)x, ldx, (bf16*)residual,
                    (const bf16*)norm_w, eps, gemma, (kind_flags >> 8) & 1, (uint8_t*)out, ldo, (float*)scales, K) == cudaSuccess
             ? 0 : -2;
}

int b200_layernorm(const void* x, const void* w, const void* b, void* out, int T, int H, float eps,
                   cudaStream_t stream) {
  if (T <= 0) return 0;
  layernorm_kernel<<<T, 256, 0, stream>>>((const bf16*)x, (const bf16*)w, (const bf16*)b,
                                          (bf16*)out, H, eps);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int b200_act_and_mul(const void* x, int ldx, void* out, int T, int I, int kind,
                     cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((I & 7) || (ldx & 7)) return -1;
  if ((kind & 0x100) && (I & 127)) return -1;      // interleaved layout needs whole blocks
  return launch_pdl(act_and_mul_kernel, dim3(ew_grid((size_t)T * (I / 8))), dim3(256), 0, stream, (const bf16*)x,
                    ldx, (bf16*)out, I, T, kind) == cudaSuccess ? 0 : -2;
}

int b200_eltwise(const void* a, const void* b, void* out, size_t n, int kind, float scalar,
                 cudaStream_t stream) {
  if (n == 0) return 0;
  if (n & 7) return -1;
  eltwise_kernel<<<ew_grid(n / 8), 256, 0, stream>>>((const bf16*)a, (const bf16*)b, (bf16*)out, n,
                                                     kind, scalar);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int b200_cast_bf16_f32(const void* a, void* out, size_t n, cudaStream_t stream) {
  if (n == 0) return 0;
  cast_bf16_to_f32_kernel<<<ew_grid(n), 256, 0, stream>>>((const bf16*)a, (float*)out, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
int b200_cast_f32_bf16(const void* a, void* out, size_t n, cudaStream_t stream) {
  if (n == 0) return 0;
  cast_f32_to_bf16_kernel<<<ew_grid(n), 256, 0, stream>>>((const float*)a, (bf16*)out, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int b200_embedding(const void* ids, const void* table, void* out, int T, int H,
                   int64_t vocab_start, int64_t vocab_rows, int64_t vocab_total, float scale,
                   cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return -1;
  embedding_kernel<<<T, 128, 0, stream>>>((const int64_t*)ids, (const bf16*)table, (bf16*)out, H,
                                          vocab_start, vocab_rows, vocab_total, scale,
                                          device_status_word());
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int b200_gather_rows(const void* x, const void* idx, void* out, int n_out, int n_src,
                     int row_bytes, cudaStream_t stream) {
  if (n_out <= 0) return 0;
  if (row_bytes & 15) return -1;
  gather_rows_kernel<<<n_out, 128, 0, stream>>>((const uint8_t*)x, (const int32_t*)idx,
                                                (uint8_t*)out, row_bytes, n_src);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
