// The product kernels behind one entry point: which of them takes a problem is decided here, so that a launch costs the caller one
// call (the decision and its queries took a scripting caller longer than the launch itself).
#include <cuda_runtime.h>
#include <stdint.h>

extern "C" {

int blitz_gemm_decode_supported(int, int, int, int, int);
int blitz_gemm_pair_supported(int, int, int, int, int);
int blitz_gemm_wide_supported(int, int, int, int, int, int);
int blitz_gemm(const void*, int64_t, const void*, int64_t, void*, int64_t, const void*, int, int, int, int, int, int, int, int, int, void*,
               int64_t, unsigned*, int, int*, float, float, int, int, int, cudaStream_t);
int blitz_gemm_decode(const void*, int64_t, const void*, int64_t, void*, int64_t, const void*, int, int, int, int, int, int, int, int, int*,
                      float, float, cudaStream_t);
int blitz_gemm_pair(const void*, int64_t, const void*, int64_t, void*, int64_t, const void*, int, int, int, int, int, int, int, int, int, int,
                    void*, int64_t, unsigned*, int, int*, float, float, cudaStream_t);
int blitz_gemm_wide(const void*, int64_t, const void*, int64_t, void*, int64_t, const void*, int, int, int, int, int, int, int, int*,
                    float, float, int, int, int, cudaStream_t);

// Scratch of one device, as the kernels' own entry points describe it.
struct BlitzGemmScratch {
  void* ws;
  int64_t ws_bytes;
  unsigned* tickets;
  int64_t num_tickets;
  void* pair_ws;
  int64_t pair_bytes;
  unsigned* pair_flags;
  int64_t num_pair_flags;
  int* status;
};

// Which kernel takes a product with "in,out" weights: 0 the tiled one, 1 weight-streaming (its activation tile is read again with every
// weight tile, which the SM's load path cannot keep up with beyond about 128 rows), 2 CTA pairs with K cut into parts, 3 CTA pairs over
// whole tiles.  With at most 74 tiles of 128 x 128 the tiled one cuts K over the SMs, which is faster and sums less in one go.
int blitz_gemm_choice(int M, int N, int K, int epilogue, int groups) {
  if (groups == 1 && M <= 128) return blitz_gemm_decode_supported(M, N, K, 0, epilogue) ? 1 : 0;
  if (groups == 1 && M <= 256) return blitz_gemm_pair_supported(M, N, K, 0, epilogue) ? 2 : 0;
  const int cols = epilogue == 2 || epilogue == 7 ? 64 : 128;
  if (M > 256 && (int64_t)((M + 127) / 128) * ((N + cols - 1) / cols) * groups > 74 && blitz_gemm_wide_supported(M, N, K, 0, epilogue, groups))
    return 3;
  return 0;
}

// Arguments as for blitz_gemm with "in,out" weights.
int blitz_gemm_any(const void* A, int64_t lda, const void* B, int64_t ldb, void* C, int64_t ldc, const void* R, int M, int N, int K,
                   int epilogue, int up_col_off, int dtype, int static_b, const BlitzGemmScratch* s, float alpha, float beta, int groups,
                   int a_step, int c_step, cudaStream_t stream) {
  if (!s) return -1;
  switch (blitz_gemm_choice(M, N, K, epilogue, groups)) {
    case 1:
      return blitz_gemm_decode(A, lda, B, ldb, C, ldc, R, M, N, K, epilogue, up_col_off, dtype, static_b, 0, s->status, alpha, beta, stream);
    case 2:
      return blitz_gemm_pair(A, lda, B, ldb, C, ldc, R, M, N, K, epilogue, up_col_off, dtype, static_b, 0, 0, 0, s->pair_ws, s->pair_bytes,
                             s->pair_flags, (int)s->num_pair_flags, s->status, alpha, beta, stream);
    case 3:
      return blitz_gemm_wide(A, lda, B, ldb, C, ldc, R, M, N, K, epilogue, up_col_off, dtype, static_b, s->status, alpha, beta, groups, a_step,
                             c_step, stream);
    default:
      return blitz_gemm(A, lda, B, ldb, C, ldc, R, M, N, K, 0, epilogue, up_col_off, dtype, 0, 0, s->ws, s->ws_bytes, s->tickets,
                        (int)s->num_tickets, s->status, alpha, beta, groups, a_step, c_step, stream);
  }
}

}  // extern "C"
