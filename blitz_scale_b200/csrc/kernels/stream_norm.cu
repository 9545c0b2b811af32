// Entry of a layer of a model whose residual stream is kept in fp32: whatever is added to the stream before the
// layer (nothing, the token's embedding as the start of the stream, the embedding once more and a step vector at the
// start of a pass of a looped block, the rows that a mixture of experts has left for the token), then the layer's
// RMSNorm, in one kernel: one read and at most one write of the stream.
//
//   x[t] = init ? embed[id[t]] : x[t] (+ embed[id[t]]) (+ step) (+ sum_k add[add_row[t][k]])
//   out[t] = x[src(t)] / sqrt(mean(x^2) + eps) * (w_offset + w)        src(t) = rows ? rows[t] + row_offset : t
//
// A block per token; the row stays in registers between the two passes up to 8192 columns.
//
// Experts' rows in 16 bits (stream_add_norm_kernel): bound by their bytes for prompts, by latency for a decode step.  A thread takes eight
// columns, asks for the row numbers once and then for up to eight rows' pieces and the stream's at the same time, 16 bytes each, so that
// no piece waits for another.  Seven rows a token of 2048 columns: 4096 tokens 41 us, 16 tokens 4.6 (the kernel for everything, a row
// after the other and four columns wide: 60 and 12.4).
#include "launch.cuh"
#include "ptx.cuh"
#include "scalar.cuh"
#include <type_traits>

namespace blitz {

struct StreamNormParams {
  const int32_t* ids;
  const void* embed;
  const void* step;
  const int32_t* rows;
  float* x;
  const void* w;
  void* out;
  const void* add;          // rows of the activation type, or null
  const int32_t* add_row;   // [tokens][n_add]
  int n_add;
  int hidden, vocab, init, add_embed, row_offset;
  float eps, w_offset;
  int* status;
};

constexpr int kSnKeep = 8;  // float4 groups a thread keeps

template <typename T, int VEC, bool ADD>
__global__ void stream_norm_kernel(const StreamNormParams p) {
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  __shared__ float red[33];
  const int t = blockIdx.x;
  const int src = p.rows ? p.rows[t] + p.row_offset : t;
  float* xr = p.x + static_cast<int64_t>(src) * p.hidden;
  const T* step = reinterpret_cast<const T*>(p.step);
  const bool change = p.init || p.add_embed || step != nullptr || ADD;
  const T* er = nullptr;
  if (p.init || p.add_embed) {
    const int id = p.ids[t];
    if (id >= 0 && id < p.vocab) {
      er = reinterpret_cast<const T*>(p.embed) + static_cast<int64_t>(id) * p.hidden;
    } else if (threadIdx.x == 0 && p.status) {
      atomicCAS(p.status, 0, kStatusBadIndex);
    }
  }
  const int n = p.hidden / VEC;
  // one group of VEC columns: VEC == 1 leaves y, z, w zero
  auto load = [&](const float* q) {
    return VEC == 4 ? *reinterpret_cast<const float4*>(q) : make_float4(*q, 0.f, 0.f, 0.f);
  };
  auto add = [&](float4& a, const T* q) {
    const float4 e = VEC == 4 ? ldf4<T>(q) : make_float4(ldf<T>(q), 0.f, 0.f, 0.f);
    a.x += e.x; a.y += e.y; a.z += e.z; a.w += e.w;
  };
  const int32_t* add_row = p.add_row + static_cast<int64_t>(t) * p.n_add;
  auto read = [&](int i) {
    float4 a = p.init ? make_float4(0.f, 0.f, 0.f, 0.f) : load(xr + i * VEC);
    if (er) add(a, er + i * VEC);
    if (step) add(a, step + i * VEC);
    if (ADD)
      for (int k = 0; k < p.n_add; ++k) add(a, reinterpret_cast<const T*>(p.add) + static_cast<int64_t>(add_row[k]) * p.hidden + i * VEC);
    if (change) {
      if (VEC == 4) *reinterpret_cast<float4*>(xr + i * VEC) = a;
      else xr[i] = a.x;
    }
    return a;
  };
  auto square = [](const float4& a) { return a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w; };
  float4 keep[kSnKeep];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < kSnKeep; ++k) {
    const int i = threadIdx.x + k * blockDim.x;
    if (i < n) {
      keep[k] = read(i);
      ss += square(keep[k]);
    }
  }
  for (int i = threadIdx.x + kSnKeep * blockDim.x; i < n; i += blockDim.x) ss += square(read(i));
  if (p.out == nullptr) return;
  ss = block_sum(ss, red);
  const float scale = rsqrtf(ss / static_cast<float>(p.hidden) + p.eps);
  const T* w = reinterpret_cast<const T*>(p.w);
  T* out = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(t) * p.hidden;
  auto write = [&](int i, const float4& v) {
    if (VEC == 4) {
      const float4 g = ldf4<T>(w + i * 4);
      stf4<T>(out + i * 4, make_float4(v.x * scale * (p.w_offset + g.x), v.y * scale * (p.w_offset + g.y),
                                       v.z * scale * (p.w_offset + g.z), v.w * scale * (p.w_offset + g.w)));
    } else {
      stf<T>(out + i, v.x * scale * (p.w_offset + ldf<T>(w + i)));
    }
  };
#pragma unroll
  for (int k = 0; k < kSnKeep; ++k) {
    const int i = threadIdx.x + k * blockDim.x;
    if (i < n) write(i, keep[k]);
  }
  for (int i = threadIdx.x + kSnKeep * blockDim.x; i < n; i += blockDim.x) write(i, load(xr + i * VEC));
}

// Only the rows to add change the stream (16-bit types, whole groups of eight columns, GROUPS of them for each thread).
template <typename T, int GROUPS>
__global__ void __launch_bounds__(512, 2) stream_add_norm_kernel(const StreamNormParams p) {
  ptx::griddep_launch_dependents();
  __shared__ float red[32];
  const int t = blockIdx.x, n = p.hidden / 8;
  float* xr = p.x + static_cast<int64_t>(t) * p.hidden;
  const int32_t* add_row = p.add_row + static_cast<int64_t>(t) * p.n_add;
  ptx::griddep_wait();
  int rows[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) rows[k] = k < p.n_add ? add_row[k] : 0;
  float keep[GROUPS][8];
  float ss = 0.f;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int i = threadIdx.x + g * blockDim.x;
    if (i >= n) continue;
    ldf8<float>(xr + i * 8, keep[g]);
    for (int k0 = 0; k0 < p.n_add; k0 += 8) {
      if (k0 > 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) rows[k] = k0 + k < p.n_add ? add_row[k0 + k] : 0;
      }
      uint4 e[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        e[k] = make_uint4(0, 0, 0, 0);
        if (k0 + k < p.n_add) e[k] = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.add) + static_cast<int64_t>(rows[k]) * p.hidden + i * 8);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k0 + k >= p.n_add) break;
        float f[8];
        unpack8<T>(e[k], f);
#pragma unroll
        for (int c = 0; c < 8; ++c) keep[g][c] += f[c];
      }
    }
    if (p.n_add > 8 && g + 1 < GROUPS) {
#pragma unroll
      for (int k = 0; k < 8; ++k) rows[k] = add_row[k];
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) ss += keep[g][c] * keep[g][c];
  }
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int i = threadIdx.x + g * blockDim.x;
    if (i < n) stf8<float>(xr + i * 8, keep[g]);
  }
  if (p.out == nullptr) return;
  const float scale = rsqrtf(block_sum1(ss, red) / static_cast<float>(p.hidden) + p.eps);
  T* out = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(t) * p.hidden;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int i = threadIdx.x + g * blockDim.x;
    if (i >= n) continue;
    float w[8];
    ldf8<T>(reinterpret_cast<const T*>(p.w) + i * 8, w);
#pragma unroll
    for (int c = 0; c < 8; ++c) w[c] = keep[g][c] * scale * (p.w_offset + w[c]);
    stf8<T>(out + i * 8, w);
  }
}

// Nothing changes the stream (16-bit types, whole groups of eight columns, GROUPS of them for each thread).  Bound by its bytes; the
// kernel for everything keeps eight groups of four columns, 64 registers, so that 256 threads wait for a row and few rows are on an SM.
// us, that kernel / this one: 8192 x 4096 62.0 / 34.7 (5.8 TB/s), 4096 x 2048 20.2 / 9.5, 256 x 4096 5.0 / 3.1.
template <typename T, int GROUPS>
__global__ void __launch_bounds__(512, 3) stream_plain_norm_kernel(const float* __restrict__ x, const T* __restrict__ w, T* __restrict__ out,
                                                                   int hidden, float eps, float w_offset) {
  ptx::griddep_launch_dependents();
  __shared__ float red[32];
  const int n = hidden / 8;
  const float* xr = x + static_cast<int64_t>(blockIdx.x) * hidden;
  T* o = out + static_cast<int64_t>(blockIdx.x) * hidden;
  ptx::griddep_wait();
  float keep[GROUPS][8];
  uint4 weights[GROUPS];
  float ss = 0.f;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int i = threadIdx.x + g * blockDim.x;
    if (i >= n) continue;
    ldf8<float>(xr + i * 8, keep[g]);
    weights[g] = *reinterpret_cast<const uint4*>(w + i * 8);
  }
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    if (threadIdx.x + g * blockDim.x >= n) continue;
#pragma unroll
    for (int c = 0; c < 8; ++c) ss += keep[g][c] * keep[g][c];
  }
  const float scale = rsqrtf(block_sum1(ss, red) / static_cast<float>(hidden) + eps);
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    const int i = threadIdx.x + g * blockDim.x;
    if (i >= n) continue;
    float f[8];
    unpack8<T>(weights[g], f);
#pragma unroll
    for (int c = 0; c < 8; ++c) f[c] = keep[g][c] * scale * (w_offset + f[c]);
    stf8<T>(o + i * 8, f);
  }
}

}  // namespace blitz

extern "C" {
using namespace blitz;

// x [tokens, hidden] fp32; embed / step / w / out in the activation type (dtype 0 fp16, 1 bf16, 2 fp32).  init: the
// stream starts as the tokens' embeddings; add_embed: they are added to it; step: vector added to every token (may be
// null); add: rows [.., hidden] of which token t receives the n_add rows add_row[t] (not together with `rows`); out (may be null): the normalised rows.  rows: read row rows[t] + row_offset of x for output row t.
int blitz_stream_norm(const int32_t* ids, const void* embed, const void* step, const int32_t* rows, int row_offset,
                      float* x, const void* w, void* out, const void* add, const int32_t* add_row, int n_add, int num_tokens, int hidden, int vocab, int init, int add_embed, float eps,
                      float w_offset, int* status, int dtype, cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (hidden <= 0 || x == nullptr || n_add < 0 || (n_add > 0 && (add == nullptr || add_row == nullptr || rows != nullptr))) return -1;
  StreamNormParams p{ids, embed, step, rows, x, w, out, add, add_row, n_add, hidden, vocab, init, add_embed, row_offset, eps, w_offset, status};
  const int n = (hidden & 3) ? hidden : hidden / 4;
  int threads = 32;
  while (threads < n && threads < (n > 1024 ? 512 : 256)) threads <<= 1;
  auto go = [&](auto type, auto vec) {
    using T = decltype(type);
    if constexpr (!std::is_same<T, float>::value) {
      // whole 16-byte pieces of everything, nothing but rows to add, at most two groups of eight columns a thread
      auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
      int wide = 32;
      while (wide < hidden / 8 && wide < 512) wide <<= 1;
      const bool pieces = !init && !add_embed && step == nullptr && (hidden & 7) == 0 && hidden <= 8192 && aligned(x) && aligned(add) && aligned(out) && aligned(w);
      if (pieces && n_add == 0 && rows == nullptr && out != nullptr) {
        return wide * 8 >= hidden
                   ? launch_pdl(stream_plain_norm_kernel<T, 1>, dim3(num_tokens), dim3(wide), 0, stream, (const float*)x, (const T*)w, (T*)out, hidden, eps, w_offset)
                   : launch_pdl(stream_plain_norm_kernel<T, 2>, dim3(num_tokens), dim3(wide), 0, stream, (const float*)x, (const T*)w, (T*)out, hidden, eps, w_offset);
      }
      if (pieces && n_add > 0) {
        return wide * 8 >= hidden ? launch_pdl(stream_add_norm_kernel<T, 1>, dim3(num_tokens), dim3(wide), 0, stream, p)
                                  : launch_pdl(stream_add_norm_kernel<T, 2>, dim3(num_tokens), dim3(wide), 0, stream, p);
      }
    }
    constexpr int V = decltype(vec)::value;
    return n_add > 0 ? launch_pdl(stream_norm_kernel<T, V, true>, dim3(num_tokens), dim3(threads), 0, stream, p)
                     : launch_pdl(stream_norm_kernel<T, V, false>, dim3(num_tokens), dim3(threads), 0, stream, p);
  };
  cudaError_t e = cudaSuccess;
  BLITZ_DISPATCH_DTYPE3(dtype, (e = (hidden & 3) ? go(T{}, std::integral_constant<int, 1>{}) : go(T{}, std::integral_constant<int, 4>{})));
  return (int)e;
}

}  // extern "C"
