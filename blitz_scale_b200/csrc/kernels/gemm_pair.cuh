// Register epilogue shared by the kernels whose CTA pairs issue tcgen05.mma.cta_group::2 (gemm_pair.cu, gemm_wide.cu).
#pragma once
#include "ptx.cuh"
#include "gemm_gate.cuh"

namespace blitz {

template <typename T>
__device__ __forceinline__ uint32_t pair_pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pair_pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t pair_pack2<__half>(float a, float b) {
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <typename T>
__device__ __forceinline__ float2 pair_unpack2(uint32_t u);
template <>
__device__ __forceinline__ float2 pair_unpack2<__nv_bfloat16>(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
}
template <>
__device__ __forceinline__ float2 pair_unpack2<__half>(uint32_t u) {
  return __half22float2(*reinterpret_cast<__half2*>(&u));
}
// 32 consecutive output columns of one row -> four 16-byte chunks.  EPI: 0 store, 1 add residual (its 32 values
// come in `res`, read before the accumulator was waited for), 2 silu(g) * u, eight at a time.
template <typename T, int EPI>
__device__ __forceinline__ void pair_convert32(const float (&g)[32], const float (&u)[32], const uint4 (&res)[4],
                                               uint4 (&out4)[4]) {
  uint32_t out[16];
  if (EPI == 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a[8], b[8], y[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        a[i] = g[8 * j + i];
        b[i] = u[8 * j + i];
      }
      silu_mul(a, b, y);
#pragma unroll
      for (int i = 0; i < 4; ++i) out[4 * j + i] = pair_pack2<T>(y[2 * i], y[2 * i + 1]);
    }
  } else if (EPI == 1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t rr[4] = {res[j].x, res[j].y, res[j].z, res[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = pair_unpack2<T>(rr[i]);
        out[j * 4 + i] = pair_pack2<T>(g[j * 8 + 2 * i] + f.x, g[j * 8 + 2 * i + 1] + f.y);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) out[i] = pair_pack2<T>(g[2 * i], g[2 * i + 1]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) out4[j] = make_uint4(out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
}

}  // namespace blitz
