// Epilogues of a product with gate and up columns, shared by the products' kernels:
//
//   2   silu(g) * u
//   7   clamped gated unit with biases:  g <- min(g + b_g, limit),  u <- clamp(u + b_u, -limit, limit),
//       g sigmoid(beta g) (u + 1)
#pragma once
#include "ptx.cuh"
#include "quotient.cuh"
#include "scalar.cuh"

namespace blitz {

constexpr int kEpiClampGlu = 7;
__host__ __device__ constexpr bool epi_gated(int epi) { return epi == 2 || epi == kEpiClampGlu; }
__host__ __device__ constexpr bool epi_f32(int epi) { return epi >= 4 && epi <= 6; }

// N silus of gate values times up values: x / (1 + e^-x) * u, the quotient as IEEE has it (quotient.cuh; tests/native/quotient_check.cpp
// compares the two) without a branch per element: the compiler's division takes one, and leaves its fast path for a quotient of zero.
// Infinities, NaN and denominators beyond 8e37 are divided by the compiler's.
template <int N>
__device__ __forceinline__ void silu_mul(const float (&x)[N], const float (&u)[N], float (&y)[N]) {
  float d[N], most = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) y[i] = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    d[i] = 1.f + __expf(-x[i]);
    const float larger = fmaxf(fabsf(x[i]), d[i]);
    most = larger < 8e37f ? most : INFINITY;
  }
  if (most == 0.f) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      y[i] = refined_quotient(x[i], d[i], ptx::rcp_approx(d[i])) * u[i];
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < N; ++i) {  // (one division's code for all of them; indexed by constants, the arrays stay in registers)
      float a = 0.f, b = 1.f, c = 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        if (j != i) continue;
        a = x[j];
        b = d[j];
        c = u[j];
      }
      const float z = a / b * c;
#pragma unroll
      for (int j = 0; j < N; ++j) y[j] = j == i ? z : y[j];
    }
  }
}

__device__ __forceinline__ float clamp_glu(float g, float u, float limit, float beta) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return __fdividef(g, 1.f + __expf(fminf(-beta * g, 80.f))) * (u + 1.f);
}

// 32 gate and up values of columns n .. n + 31 in place: biases added, then the unit; the results are in g.  bias: the gate
// columns' from `bias` on, the up columns' from `bias + up` on (both 16-byte aligned, up a multiple of 8).
template <typename T>
__device__ __forceinline__ void clamp_glu32(const T* bias, int up, int n, int N, float limit, float beta, const float (&g)[32],
                                            const float (&u)[32], float (&out)[32]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float bg[8] = {}, bu[8] = {};
    if (n + 8 * j < N) {
      ldf8<T>(bias + n + 8 * j, bg);
      ldf8<T>(bias + up + n + 8 * j, bu);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) out[8 * j + i] = clamp_glu(g[8 * j + i] + bg[i], u[8 * j + i] + bu[i], limit, beta);
  }
}

}  // namespace blitz
