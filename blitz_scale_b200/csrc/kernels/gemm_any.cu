// The product kernels behind one entry point: which of them takes a problem is decided here, so that a launch costs the caller one
// call (the decision and its queries took a scripting caller longer than the launch itself).
#include "tmap.cuh"
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <mutex>

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
int blitz_gemm_decode_resident(int);
int blitz_gemm_quad_resident();
int blitz_gemm_quad_supported(int, int, int, int, int);
int blitz_gemm_quad(const void*, int64_t, const void*, int64_t, void*, int64_t, const void*, int, int, int, int, int, int, int*, float, cudaStream_t);
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

// What a device holds at once, as the kernels' own launches ask for it: SMs, clusters of 1 to 8 CTAs of the weight-streaming kernel, and
// clusters of four of gemm_quad.cu.  Asked once per device; without one, the figures are those of a B200.
struct GemmMachine {
  int sms, streams[9], quads;
};
static const GemmMachine& machine() {
  static constexpr GemmMachine kB200{148, {0, 148, 74, 45, 33, 26, 22, 15, 15}, 33};
  static GemmMachine of[64];
  static std::atomic<int> known[64];
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return kB200;
  }
  if (!known[dev].load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> g(mu);
    if (!known[dev].load(std::memory_order_relaxed)) {
      GemmMachine m = kB200;
      m.sms = blitz::device_sm_count();
      for (int i = 1; i <= 8; ++i)
        if (const int n = blitz_gemm_decode_resident(i)) m.streams[i] = n;
      if (const int n = blitz_gemm_quad_resident()) m.quads = n;
      of[dev] = m;
      known[dev].store(1, std::memory_order_release);
    }
  }
  return of[dev];
}

// The same, one at a time: 0 SMs, 1 to 8 clusters of the weight-streaming kernel, 9 clusters of gemm_quad.cu.
int blitz_gemm_resident(int what) {
  const GemmMachine& m = machine();
  return what == 0 ? m.sms : what >= 1 && what <= 8 ? m.streams[what] : what == 9 ? m.quads : -1;
}

// Whether more than 256 rows are better on pairs of CTAs with whole tiles of 256 x 256 (gemm_wide.cu; halves of them where a last round
// of halves fits the 74 pairs) than on 148 CTAs with tiles of 128 x 256 or x 128 and K in parts (gemm_tcgen05.cu).  In a few rounds that
// is a matter of which tiles fill the SMs.  Measured with cold weights, us, pairs / tiles:
//   at most 74 tiles of 128 x 128: K in parts, which also sums less in one go
//   at most 148: one round of tiles.  No half tiles: 300 x 6144 x 4096 25.7 / 19.5, 2048 x 1152 x 8192 45 / 33, with SiLU
//     384 x 2816 x 2048 18.9 / 14.8.  Half tiles: 1024 x 2048 x 2048 12.5 / 11.3, into fp32 15.5 / 13.9; but epilogues that read or
//     compute more hide behind the pairs' two accumulators: residual 512 x 2560 x 1024 8.5 / 9.5, SiLU 1000 x 1024 x 2048 16.9 / 21.2
//     (columns that are not whole slabs of 64 keep the tiles' loads waiting: 6400 x 136 x 2048 12.3 / 15.5)
//   at most 148 tiles of 128 x 256, but more than 74 pairs (rows that fill a little more than one tile of 256): 300 x 10240 x 4096
//     38.7 / 34.6, with SiLU 300 x 5632 x 2048 33.9 / 29.8
//   blocks that fill half of a tile's columns or less: 32 of 1000 x 128 x 512 11.5 / 10.7, but 32 of 4096 x 128 x 512 34.9 / 36.6; a
//     quarter: 32 of 1574 x 64 x 512 15.6 / 12.9, 32 of 2500 21.1 / 23.4
//   one round of whole tiles into fp32, whose epilogue nothing hides: 1290 x 2048 x 1024 17.0 / 15.5, K = 2048 22.2 / 21.5, 4096 32.5 / 33.5
//   all others measured: 0.6 .. 1.0 of the tiles' time, for instance 1574 x 4096 x 4096 46.0 / 55.6, 8192 x 4096 x 14336 615 / 724
static bool pairs_are_better(int M, int N, int K, int epilogue, int groups) {
  const bool gated = epilogue == 2 || epilogue == 7, f32 = epilogue >= 4 && epilogue <= 6;
  const int cols = gated ? 64 : 128;
  auto tiles = [&](int rows, int columns) { return (int64_t)((M + rows - 1) / rows) * ((N + columns - 1) / columns) * groups; };
  const int64_t narrow = tiles(128, cols), pairs = tiles(256, 2 * cols);
  const bool odd = N < 2 * cols && N % 64 != 0;
  const int sms = machine().sms, most = sms / 2;
  if (narrow <= most) return false;
  if (narrow <= sms) return (2 * pairs <= most && (gated || epilogue == 1)) || odd;
  if (tiles(128, 2 * cols) <= sms && pairs > most) return false;
  if (N <= cols && narrow <= (2 * N <= cols ? 512 : 2 * sms)) return false;
  if (f32 && !odd && K <= 2048 && pairs <= most && 2 * pairs > most) return false;
  return true;
}

// Whether K in halves over clusters of four (gemm_quad.cu) takes a product in one round: 33 of its clusters are resident on 148 SMs, and a
// second round costs as much as the first.  More than 256 rows in one round, us, tiles of 128 rows (gemm_tcgen05.cu) / whole or half tiles on CTA
// pairs / these: 300 rows x 2048 columns of K = 256 11.0 / 6.1 / 7.0, 512 13.2 / 7.0 / 7.5, 1024 16.0 / 9.4 / 8.5, 4096 17.9 / 19.6 / 13.0, 14336
// 31.0 / 54.2 / 28.3;  1000 x 1024 of K = 2048 16.8 / 16.6 / 12.5;  3000 x 128 of K = 2048 17.3 / 15.4 / 12.6.  (Two rounds, 300 x 4096 of
// K = 4096: 22.7 / 21.6 / 25.8.)
static bool one_round_of_quads(int M, int N, int K, int epilogue) {
  return (int64_t)((M + 255) / 256) * ((N + 127) / 128) <= machine().quads && blitz_gemm_quad_supported(M, N, K, 0, epilogue);
}

// Of those 129 to 256 rows, the products that are too wide for one round of quads, leave half of the pairs idle in whole tiles, and are deep:
// K cut into parts on CTA pairs (2) pays the exchange of sums through L2, 8 us more than the others, from K = 4608 on, and the more the
// more rows the weight-streaming kernel (1) reads again with every tile.  Each costs a time per K block that grows with the CTAs that
// load at once, and half tiles (3) that of the whole K.  Clusters of an odd number of CTAs do not fill the SMs beside a predecessor's last
// blocks: with nearly as many of them as are resident the last ones start late.  Measured behind a norm with cold weights, us, 1 / 2 / 3:
//   6144 x 8192 with a residual, 136, 192 and 224 rows 33.0 / 34.9 / 39.0, 38.9 / 35.3 / 38.8, 41.6 / 35.7 / 39.4
//   6144 x 14336 48.1 / 48.1 / 60.8 at 160 rows, 52.1 / 48.6 / 61.8 at 224;  8192 x 14336 54.1 / 58.6 / 63.9 at 192, 63.9 / 59.4 / 64.7 at 256
//   5632 x 14336 (44 clusters of three) 46.9 / 46.9 / 60.4 at 136 rows, with a residual 61.4 / 48.4 / 62.4 at 208, 81.8 / 49.5 / 63.2 at 256
// Over 1320 products of 4232 to 9472 columns, K = 5120 to 20480, 130 to 256 rows: 1.003 of the fastest on average, 1.17 at worst (those clusters at 136 rows).
static int deep_few_rows(int M, int tiles, int wide, int kb, bool add, const GemmMachine& m) {
  int p = m.sms / tiles < 8 ? m.sms / tiles : 8;
  while (p > 1 && tiles > m.streams[p]) --p;
  if (p < 1) p = 1;
  const int q = m.sms / 2 / wide;
  float streaming = 0.032f * M + (kb + p - 1) / p * (0.035f + 0.0009f * M + 0.0017f * p * tiles) + (add ? 0.05f * M / p : 0.f);
  if (p > 1 && (p & 1) && 16 * tiles > 15 * m.streams[p]) streaming *= 1.3f;
  const float parts = 10.4f + (kb + q - 1) / q * (0.167f + 0.0027f * q * wide + 0.042f * q);
  const float halves = 2.7f + kb * (0.186f + 0.0022f * wide + 0.0001f * M);
  return parts < halves && parts < streaming ? 2 : streaming <= halves ? 1 : 3;
}

// 129 to 256 rows: the weight-streaming kernel (1), whole or half tiles of 256 x 256 on CTA pairs (3), those with K cut into parts (2), or
// K in halves over clusters of four (4).  The first is as fast as its loads, 128 bytes per row and column of a K block and CTA, with as many parts of
// K as clusters fit, and adds an exchange of the parts' sums; the third takes a quarter of a microsecond per K block of a round of half tiles, 0.4 of
// whole ones; the fourth 0.13 to 0.23 per two K blocks, the more the more columns stream.  Estimates below are in us, without what
// all of them cost.  Measured behind a small kernel with cold weights, us, 1 / 2 / 3 / 4:
//   4096 x 4096 with a residual, 136 and 256 rows 16.1 / 20.8 / 20.4 / 13.8, 21.0 / 22.0 / 21.1 / 14.2;  6144 columns 17.9 / 23.5 / 21.0 / 25.4,
//     25.2 / 24.0 / 21.5 / 26.0
//   4096 columns of K = 14336 32.3 / 40.7 / 59.7 / 32.6, 42.4 / 41.6 / 60.1 / 34.0;  2048 of it 19.0 / 48.1 / 53.1 / 26.7, 27.3 / 47.6 / 54.2 / 28.0
//   1024 columns of K = 4096 10.5 / 19.9 / 18.4 / 11.6, 13.3 / 20.1 / 18.3 / 11.6;  4096 of K = 1024 11.6 / 15.6 / 9.3 / 8.3, 15.2 / 16.3 / 9.6 / 8.8
//   128256 columns of K = 4096, 144 and 256 181 / 214 / 202 / -, 248 / 245 / 212 / -;  8192 of K = 1024 11.4 / 14.5 / 9.7, 15.0 / 15.9 / 10.1
//   6144 columns of K = 8192, 200 and 256 rows 34.5 / 35.6 / 38.8, 40.5 / 35.7 / 39.3
// Gated units need both accumulators' weights at once: fewer stages, and beyond 192 rows room for fewer parts.  144, 192 and 256 rows:
//   14336 x 4096 49.3 / 57.0 / 56.6, 54.3 / 57.5 / 57.7, 66.7 / 58.3 / 58.2;  8192 x 4096 36.0 / 35.9 / 34.8, 38.3 / 36.7 / 35.5, 62.1 / 37.4 / 36.2
//   2816 x 2048 15.7 / 19.1 / 14.3, 17.5 / 19.3 / 14.5, 36.1 / 19.1 / 15.1
// (bench/kernels_bench.py --only choice times all of them at 104 such products: 1.01 of the fastest on average, 1.20 at worst.)
int blitz_gemm_few_rows(int M, int N, int K, int epilogue) {
  const GemmMachine& m = machine();
  const int sms = m.sms, pairs = sms / 2;
  const int tiles = (N + 127) / 128, wide = (N + 255) / 256, kb = (K + 63) / 64;
  if (epilogue == 2 || epilogue == 7) return M <= 192 && tiles > pairs ? 1 : 3;
  const bool quads = one_round_of_quads(M, N, K, epilogue);
  if (!quads && 2 * wide <= pairs && kb > 71) return deep_few_rows(M, tiles, wide, kb, epilogue == 1, m);
  int parts = sms / tiles < 8 ? sms / tiles : 8;
  if (parts > kb) parts = kb;
  while (parts > 1 && tiles > m.streams[parts]) --parts;
  if (parts < 1) parts = 1;
  const bool all = parts > 1 && parts * tiles >= sms * 13 / 16;  // (what nearly all SMs load together is less than what each can)
  const float exchange = parts > 1 ? 0.027f * M + (all ? 2.f : 0.f) : epilogue == 1 ? 0.07f * M : 1.5f;  // (one part: a residual's loads are exposed)
  const float streaming = ((kb + parts - 1) / parts) * ((tiles + sms - 1) / sms) * (0.18f + 0.0011f * M) * (all ? 1.2f : 1.f) + exchange;
  const int rest = wide % pairs;
  const float rounds = 2 * wide <= pairs ? 0.625f : wide / pairs + (rest == 0 ? 0.f : 2 * rest <= pairs ? 0.65f : 1.f);
  const float whole = 0.4f * kb * rounds + 1.5f;
  const float halves = quads ? 3.5f + ((kb + 1) / 2) * (0.13f + 0.0031f * tiles) : 1e30f;
  return halves < whole && halves < streaming ? 4 : streaming <= whole ? 1 : 3;
}

// The kernel that a call with hints starts from, before they are looked at: 0 the tiled one, 1 weight-streaming (128 rows at most), 2 CTA
// pairs with K cut into parts (256 rows at most), 3 CTA pairs over whole tiles.
int blitz_gemm_choice(int M, int N, int K, int epilogue, int groups) {
  if (groups == 1 && M <= 128) return blitz_gemm_decode_supported(M, N, K, 0, epilogue) ? 1 : 0;
  if (groups == 1 && M <= 256) return blitz_gemm_pair_supported(M, N, K, 0, epilogue) ? 2 : 0;
  return M > 256 && pairs_are_better(M, N, K, epilogue, groups) && blitz_gemm_wide_supported(M, N, K, 0, epilogue, groups) ? 3 : 0;
}

// Which kernel runs a product with "in,out" weights that carries no hint: that of blitz_gemm_choice beyond 256 rows and up to 128, the one
// that blitz_gemm_few_rows names in between, or 4, K in halves over clusters of four, which fills a round that the others do not.  (What (2)
// takes the other kernels for few rows take too, and whole tiles take what (4) takes.)
int blitz_gemm_kernel(int M, int N, int K, int epilogue, int groups) {
  const int choice = blitz_gemm_choice(M, N, K, epilogue, groups);
  if (choice == 2) return blitz_gemm_few_rows(M, N, K, epilogue);
  if (groups == 1 && M > 256 && one_round_of_quads(M, N, K, epilogue)) return K > 512 ? 4 : 3;
  return choice;
}

// Arguments as for blitz_gemm with "in,out" weights.
int blitz_gemm_any(const void* A, int64_t lda, const void* B, int64_t ldb, void* C, int64_t ldc, const void* R, int M, int N, int K,
                   int epilogue, int up_col_off, int dtype, int static_b, const BlitzGemmScratch* s, float alpha, float beta, int groups,
                   int a_step, int c_step, cudaStream_t stream) {
  if (!s) return -1;
  switch (blitz_gemm_kernel(M, N, K, epilogue, groups)) {
    case 4:
      return blitz_gemm_quad(A, lda, B, ldb, C, ldc, R, M, N, K, epilogue, dtype, static_b, s->status, alpha, stream);
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
