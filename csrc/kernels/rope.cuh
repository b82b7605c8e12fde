// Rotation of a 128-dim head (full NeoX rotation) by one warp, lane l holding dims 4l..4l+3, with the head's RMSNorm in front and
// its place in the paged KV cache: what the preamble kernel of the attention and the QKV product that takes it along share.
#pragma once
#include "sm100.cuh"

namespace b200 {

struct RopeCacheSlot {
  __nv_bfloat16 *k, *v;      // where the token's first k / v head goes, or null
};
__device__ __forceinline__ RopeCacheSlot rope_cache_slot(int64_t slot, __nv_bfloat16* cache, int block_size, int Hkv) {
  if (slot < 0) return {nullptr, nullptr};
  const bool small = (slot >> 31) == 0;               // (64-bit division takes longer than the loads)
  const int64_t blk = small ? (int64_t)((uint32_t)slot / (uint32_t)block_size) : slot / block_size;
  const int64_t off = slot - blk * block_size;
  return {cache + ((blk * 2 + 0) * block_size + off) * (int64_t)Hkv * 128,
          cache + ((blk * 2 + 1) * block_size + off) * (int64_t)Hkv * 128};
}
__device__ __forceinline__ float normed_bf16(float x, float inv, float w) { return __bfloat162float(__float2bfloat16(x * inv * w)); }

// x: the lane's four dims (bf16 values), c / s: cos and sin of dims (l & 15) * 4 .. + 3, nw: norm weight or null.
__device__ __forceinline__ uint2 rope_head(const float (&in)[4], const float4& c4, const float4& s4, const __nv_bfloat16* nw, float eps,
                                           int gemma, int lane) {
  const float c[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
  float x[4] = {in[0], in[1], in[2], in[3]};
  if (nw) {
    float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = rsqrtf(ss / 128.f + eps), g = gemma ? 1.f : 0.f;
    const uint2 wr = *reinterpret_cast<const uint2*>(nw + lane * 4);
    const float2 w0 = unpack_bf16x2(wr.x), w1 = unpack_bf16x2(wr.y);
    const float w[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = normed_bf16(x[k], inv, w[k] + g);   // norm output is bf16
  }
  float y[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float other = __shfl_xor_sync(0xffffffffu, x[k], 16);
    y[k] = lane < 16 ? x[k] * c[k] - other * sn[k] : x[k] * c[k] + other * sn[k];
  }
  return make_uint2(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]));
}

}  // namespace b200
