// Persistent paired-SM tcgen05 GEMM for activation blocks of more than 256 rows (prompts) in the serving layout.
//
//   C[M,N] = A[M,K] * W[K,N]      W "in,out" (N contiguous), 16-bit, fp32 accumulation in TMEM
//
// At these sizes the product is bound by the tensor pipe, and what kept the 128 x 256 tiles of a single CTA (gemm_tcgen05.cu)
// below it is shared memory: per 16-wide K step such a CTA reads 4 KB of A and 8 KB of W and writes as much again per 64, about
// 190 of the 128 bytes per clock an SM has at full rate.  Here the two CTAs of a cluster issue one 256 x 256
// `tcgen05.mma.cta_group::2`: each keeps 128 rows of A and half of the W columns, so an SM reads 8 KB instead of 12 KB per step and
// pulls 32 KB instead of 48 KB per K block out of L2.  Every CTA loads its own halves with plain per-CTA TMA (no cluster multicast).
// A K block of a whole tile takes 300 ns of UMMAs and, beside them, 240 ns of loads once one elected thread issues two loads (three
// from a `lane == 0` branch: 345 ns).  Measured on the products of a Llama-3-8B layer, us (before: gemm_tcgen05.cu, also elected):
//   M = 8192: 6144 x 4096 321 -> 265, 4096 x 4096 222 -> 197, gate and up 1623 -> 1373;  cuBLAS 316 / 227 / 1424 (without SiLU)
//   M = 1574: 75 -> 64, 55 -> 46, 293 -> 257 (before the division in SiLU was exact), 4096 x 14336 188 -> 165;  cuBLAS 55 / 36 / 267 / 118
//
// Tiles are handed out in rounds of one per pair, `group_m` row tiles by all column tiles at a time, so that the pairs working at
// the same moment share rows and columns in L2.  The last, incomplete round is cut into tiles of half the columns where these fit
// one round: they take 0.7 of a whole tile's time (260 against 387 ns per K block) and need no exchange of partial sums.
// Two accumulators (512 TMEM columns): the epilogue of a tile runs beside the next one's main loop.  Eight epilogue warps convert,
// write 128-byte-swizzled 32 x 64 boxes to a staging area and hand them to TMA stores; fp32 outputs are stored directly, whole
// 128-byte lines per thread.
// Block-diagonal products (groups > 1) as in gemm_tcgen05.cu, for K a multiple of 64.
//
// Roles per CTA (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner (+ UMMA issuer in the even CTA), warps 2..9 = epilogue
// (TMEM lane quarter = warp % 4, two warps per quarter).
#include "launch.cuh"
#include "ptx.cuh"
#include "tmap.cuh"
#include "gemm_pair.cuh"
#include <type_traits>

namespace blitz {

constexpr int kWideThreads = 320;
constexpr int kWideEpiWarps = 8;
constexpr int kWideBK = 64;
constexpr int kWideRows = 128;                       // rows of A per CTA; the pair covers 256
constexpr int kWideABytes = kWideRows * kWideBK * 2;
constexpr int kWideStageBytes = 2 * kWideABytes;     // A rows, and up to 128 W columns
constexpr int kWideStages = 6;
constexpr int kWideStagingBytes = 2 * 4 * 4096;      // two boxes of 32 rows x 128 bytes per lane quarter
constexpr int kWideBarrierBytes = (2 * kWideStages + 4) * 8 + 16;
constexpr int kWideSmemBytes = 1024 + kWideStages * kWideStageBytes + kWideStagingBytes + kWideBarrierBytes;
static_assert(kWideSmemBytes <= 227 * 1024, "shared memory of one CTA");

struct WideParams {
  void* C;         // fp32 outputs (the 16-bit ones are stored through tmap_c)
  const void* R;
  float alpha;     // axpy; soft cap; limit of the clamped unit
  float beta;      // clamped unit (R: its biases)
  int64_t ldc;
  int M, N, num_kb;
  int tiles_m, tiles_n, group_m;
  int full;        // tiles of 256 columns; the others come as two halves each
  int items;       // full + 2 * halved tiles
  int up_col_off;  // gated: column of W where the "up" half starts
  int groups, group_tiles, a_step, c_step;  // diagonal blocks: column tiles per block, columns of A and C between two
  int slabs;       // W's columns come in whole slabs of 64: both slabs of a whole tile's half in one load (tmap_b2)
  int static_b;    // W is not written by kernels still running in this stream
  int* status;
};

// One piece of work of a pair.
struct WideItem {
  int m0, n0;      // first row, first output column (within the block)
  int group;
  int width;       // accumulator columns: 256 or 128
  bool any;        // some column exists
};

template <int EPI>
__device__ __forceinline__ WideItem wide_item(const WideParams& p, int i) {
  int tile = i, half = 0;
  WideItem w;
  w.width = 256;
  if (i >= p.full) {
    tile = p.full + ((i - p.full) >> 1);
    half = (i - p.full) & 1;
    w.width = 128;
  }
  const int per = p.group_m * p.tiles_n;
  const int g = tile / per, rem = tile - g * per;
  const int rows = min(p.group_m, p.tiles_m - g * p.group_m);
  int nt = rem / rows;
  w.m0 = (g * p.group_m + rem - nt * rows) * 2 * kWideRows;
  w.group = 0;
  if (p.groups > 1) {
    w.group = nt / p.group_tiles;
    nt -= w.group * p.group_tiles;
  }
  constexpr int kCols = epi_gated(EPI) ? 128 : 256;  // output columns of a whole tile
  w.n0 = nt * kCols + half * (kCols / 2);
  w.any = w.n0 < p.N;
  return w;
}

template <typename T, int EPI>
__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_b2, const __grid_constant__ CUtensorMap tmap_c, const WideParams p) {
  constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  constexpr int S = kWideStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint8_t* staging = smem + S * kWideStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + kWideStagingBytes);
  uint64_t* full_bar = bars;               // [S]  used in the even CTA: bytes of both CTAs
  uint64_t* empty_bar = bars + S;          // [S]  per CTA: stage released by the pair's UMMAs
  uint64_t* tfull_bar = bars + 2 * S;      // [2]  per CTA: accumulator complete
  uint64_t* tempty_bar = bars + 2 * S + 2; // [2]  used in the even CTA: the 16 epilogue warps of the pair drained it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();  // 0 = even CTA (issues the UMMAs), 1 = odd CTA
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&tfull_bar[i], 1);
      ptx::mbar_init(&tempty_bar[i], 2 * kWideEpiWarps);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::tma_prefetch_desc(&tmap_a);
    ptx::tma_prefetch_desc(&tmap_b);
    if (p.slabs) ptx::tma_prefetch_desc(&tmap_b2);
    ptx::tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  // both CTAs have initialised their barriers before either signals the other's
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  ptx::griddep_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs, own halves)
    if (ptx::elect_one()) {
      const uint32_t full0 = ptx::mapa_shared(ptx::smem_u32(full_bar), 0u);  // the even CTA's full barriers
      auto load_b = [&](int stage, const WideItem& w, int kb) {
        uint8_t* sb = smem + stage * kWideStageBytes + kWideABytes;
        const int half = w.width >> 1;
        const int col = epi_gated(EPI) ? (rank == 0 ? 0 : p.up_col_off) + w.n0 : w.n0 + static_cast<int>(rank) * half;
        const int row = (w.group * p.num_kb + kb) * kWideBK;  // (blocks are stacked; with several K is a multiple of 64)
        if (half == 128 && p.slabs) {
          ptx::tma_load_3d_pair(sb, &tmap_b2, full0 + 8u * stage, 0, row, col >> 6);
          return;
        }
        for (int s = 0; s < half / 64; ++s) ptx::tma_load_2d_pair(sb + s * 8192, &tmap_b, full0 + 8u * stage, col + s * 64, row);
      };
      auto load_a = [&](int stage, const WideItem& w, int kb) {
        ptx::tma_load_2d_pair(smem + stage * kWideStageBytes, &tmap_a, full0 + 8u * stage, w.group * p.a_step + kb * kWideBK,
                              w.m0 + static_cast<int>(rank) * kWideRows);
      };
      auto expect = [&](int stage, const WideItem& w) {
        if (rank == 0) ptx::mbar_expect_tx(&full_bar[stage], 2u * (kWideABytes + static_cast<uint32_t>(w.width) * kWideBK));
      };
      // with static weights the first stages' weight tiles are requested before the dependency wait
      int npre = 0;
      if (p.static_b && pair < p.items) {
        const WideItem w = wide_item<EPI>(p, pair);
        if (w.any) {
          npre = min(S, p.num_kb);
          for (int i = 0; i < npre; ++i) {
            expect(i, w);
            load_b(i, w, i);
          }
        }
      }
      ptx::griddep_wait();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const WideItem w = wide_item<EPI>(p, i);
        if (!w.any) continue;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (npre > 0) {
            load_a(stage, w, kb);
            --npre;
          } else {
            if (!ptx::bounded_mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) {
              if (p.status) atomicCAS(p.status, 0, kStatusTimeoutProducer);
              ok = false;
              break;
            }
            expect(stage, w);
            load_a(stage, w, kb);
            load_b(stage, w, kb);
          }
          if (++stage == S) { stage = 0; phase ^= 1u; }
        }
      }
      // drain: the releases of the last stages are remote barrier signals; take them before this CTA may exit (a stage that was
      // never filled answers at once)
      if (ok) {
        for (int i = 0; i < S; ++i) {
          if (!ptx::bounded_mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) break;
          if (++stage == S) { stage = 0; phase ^= 1u; }
        }
      }
    } else {
      ptx::griddep_wait();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ UMMA issuer (even CTA only)
    ptx::griddep_wait();
    if (rank == 0 && ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int buf = 0;
      uint32_t buf_phase = 0;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const WideItem w = wide_item<EPI>(p, i);
        if (!w.any) continue;
        const uint32_t idesc = ptx::make_idesc_f16(kFmt, 0u, 1u, 2 * kWideRows, static_cast<uint32_t>(w.width));
        if (!ptx::bounded_mbar_wait(&tempty_bar[buf], buf_phase ^ 1u, abort_flag)) {
          if (p.status) atomicCAS(p.status, 0, kStatusTimeoutMma);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * 256);
        for (int kb = 0; kb < p.num_kb; ++kb) {
          if (!ptx::bounded_mbar_wait(&full_bar[stage], phase, abort_flag)) {
            if (p.status) atomicCAS(p.status, 0, kStatusTimeoutMma);
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t a_base = ptx::smem_u32(smem + stage * kWideStageBytes);
          const uint32_t b_base = a_base + kWideABytes;
#pragma unroll
          for (int k = 0; k < kWideBK / 16; ++k) {
            // A: K-major, 128-byte rows, 8-row groups 1024 B apart; 16 K elements = 32 B.
            // W: N-major slabs of 64 columns 8192 B apart, 8-K-row groups 1024 B apart; 16 K rows = 2048 B.
            const uint64_t adesc = ptx::make_smem_desc(a_base + k * 32, 16, 1024, ptx::kLayoutSw128);
            const uint64_t bdesc = ptx::make_smem_desc(b_base + k * 2048, 8192, 1024, ptx::kLayoutSw128);
            ptx::umma_f16_ss_pair(d_tmem, adesc, bdesc, idesc, (kb != 0 || k != 0) ? 1u : 0u);
          }
          ptx::umma_commit_pair(&empty_bar[stage], 3);
          if (++stage == S) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        ptx::umma_commit_pair(&tfull_bar[buf], 3);
        buf ^= 1;
        if (buf == 0) buf_phase ^= 1u;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps (256 threads; the two warps of lane quarter q
    // meet on named barrier 3 + q)
    ptx::griddep_wait();
    const int q = warp & 3;
    const int ch = (warp - 2) >> 2;  // which 32-column half of every 64-column slab this warp takes
    const bool issuer = (ch == 0 && lane == 0);  // issues this quarter's TMA stores
    const uint32_t tempty0 = ptx::mapa_shared(ptx::smem_u32(tempty_bar), 0u);
    int buf = 0;
    uint32_t buf_phase = 0;
    int box_no = 0;  // boxes this quarter has handed over
    for (int i = pair; i < p.items; i += pairs) {
      const WideItem w = wide_item<EPI>(p, i);
      if (!w.any) continue;
      const int row0 = w.m0 + static_cast<int>(rank) * kWideRows + q * 32;
      const int row = row0 + lane;
      const bool row_ok = row < p.M;
      const bool quarter_ok = row0 < p.M;  // the same for both warps of a quarter
      const int half = w.width >> 1;
      const int slabs = (epi_gated(EPI) ? half : w.width) >> 6;  // slabs of 64 output columns: 1, 2 or 4
      // the residual of the first slab is requested before the accumulator is complete, the next one's while a slab is converted
      uint4 res[4] = {};
      auto residual = [&](int s, uint4 (&r)[4]) {
        if (EPI != 1 || s >= slabs) return;
        const T* Rp = reinterpret_cast<const T*>(p.R) + static_cast<int64_t>(row) * p.ldc;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = w.n0 + s * 64 + ch * 32 + j * 8;
          r[j] = make_uint4(0, 0, 0, 0);
          if (row_ok && col < p.N) r[j] = *reinterpret_cast<const uint4*>(Rp + col);
        }
      };
      residual(0, res);
      if (!ptx::bounded_mbar_wait(&tfull_bar[buf], buf_phase, abort_flag)) {
        if (p.status && lane == 0) atomicCAS(p.status, 0, kStatusTimeoutEpilogue);
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * 256);
      // (rolled: in a launch of a round or two this code runs once or twice and comes from far away)
#pragma unroll 1
      for (int s = 0; s < slabs; ++s) {
        const int n = w.n0 + s * 64;
        if (!quarter_ok || n >= p.N) continue;
        const int c = s * 64 + ch * 32;  // first of this thread's 32 columns within the tile
        uint32_t v[32];
        float g[32], up[32];
        uint4 next[4] = {};
        residual(s + 1, next);
        ptx::tmem_ld_32x32(taddr + c, v);
        if (epi_gated(EPI)) {
          uint32_t t[32];
          ptx::tmem_ld_32x32(taddr + half + c, t);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 32; ++k) up[k] = __uint_as_float(t[k]);
        } else {
          ptx::tmem_ld_wait();
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) g[k] = __uint_as_float(v[k]);
        if (epi_f32(EPI)) {
          // a thread's 32 columns are a whole 128-byte line
          if (row_ok) {
            float* dst = reinterpret_cast<float*>(p.C) + static_cast<int64_t>(row) * p.ldc + static_cast<int64_t>(w.group) * p.c_step +
                         n + ch * 32;
            float old[4][8];
            const float inv = EPI == 6 ? 1.f / p.alpha : 0.f;
            if (EPI == 5) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (n + ch * 32 + 8 * j < p.N) ptx::ld_global_v8(dst + 8 * j, old[j]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (n + ch * 32 + 8 * j < p.N) {
                float o[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                  o[k] = EPI == 5   ? old[j][k] + p.alpha * g[8 * j + k]
                         : EPI == 6 ? p.alpha * ptx::tanh_ex2(g[8 * j + k] * inv)
                                    : g[8 * j + k];
                ptx::st_global_v8(dst + 8 * j, o);
              }
            }
          }
          continue;
        }
        uint4 o4[4];
        if (EPI == kEpiClampGlu) {
          float y[32];
          clamp_glu32<T>(reinterpret_cast<const T*>(p.R), p.up_col_off, n + ch * 32, p.N, p.alpha, p.beta, g, up, y);
          pair_convert32<T, 0>(y, up, res, o4);
        } else {
          pair_convert32<T, EPI>(g, up, res, o4);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) res[j] = next[j];
        // the quarter's two boxes in turn: the previous contents (two slabs ago) have been read out
        uint8_t* box = staging + ((box_no++ & 1) * 4 + q) * 4096;
        if (issuer) ptx::tma_store_wait_read<1>();
        asm volatile("bar.sync %0, 64;" ::"r"(3 + q) : "memory");
        // 128-byte rows, 16-byte chunks XOR-swizzled by row: the layout the TMA store expects
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(box + lane * 128 + (((ch * 4 + j) ^ (lane & 7)) << 4)) = o4[j];
        ptx::fence_proxy_async_smem();
        asm volatile("bar.sync %0, 64;" ::"r"(3 + q) : "memory");
        if (issuer) {
          ptx::tma_store_2d(&tmap_c, box, w.group * p.c_step + n, row0);
          ptx::tma_store_commit();
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(tempty0 + 8u * buf);
      buf ^= 1;
      if (buf == 0) buf_phase ^= 1u;
    }
    if (issuer) ptx::tma_store_wait<0>();  // the staged boxes have been written out before the CTA may exit
  }

  __syncwarp();
  ptx::tc_fence_before_sync();
  __syncthreads();
  // neither CTA leaves (or frees TMEM) while its partner may still signal its barriers or read its tiles
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

template <typename T, int EPI>
static int wide_launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tb2, const CUtensorMap& tc, const WideParams& p, int pairs,
                       cudaStream_t stream) {
  auto kern = gemm_wide_kernel<T, EPI>;
  static PerDeviceOnce once;
  cudaError_t e = once.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmemBytes); });
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(launch_pdl_cluster(kern, dim3(2 * pairs), dim3(kWideThreads), (size_t)kWideSmemBytes, 2u, stream, ta, tb, tb2, tc, p));
}

template <typename T>
static int wide_dispatch(int epilogue, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tb2, const CUtensorMap& tc, const WideParams& p, int pairs,
                         cudaStream_t stream) {
  switch (epilogue) {
    case 1: return wide_launch<T, 1>(ta, tb, tb2, tc, p, pairs, stream);
    case 2: return wide_launch<T, 2>(ta, tb, tb2, tc, p, pairs, stream);
    case 4: return wide_launch<T, 4>(ta, tb, tb2, tc, p, pairs, stream);
    case 5: return wide_launch<T, 5>(ta, tb, tb2, tc, p, pairs, stream);
    case 6: return wide_launch<T, 6>(ta, tb, tb2, tc, p, pairs, stream);
    case 7: return wide_launch<T, 7>(ta, tb, tb2, tc, p, pairs, stream);
    default: return wide_launch<T, 0>(ta, tb, tb2, tc, p, pairs, stream);
  }
}

}  // namespace blitz

extern "C" {

// Whether blitz_gemm_wide takes this problem: "in,out" weights, whole 16-byte rows, diagonal blocks of whole K blocks.
int blitz_gemm_wide_supported(int M, int N, int K, int b_layout, int epilogue, int groups) {
  return M >= 1 && b_layout == 0 && ((epilogue >= 0 && epilogue <= 2) || (epilogue >= 4 && epilogue <= blitz::kEpiClampGlu)) && (N & 7) == 0 &&
         (K & 7) == 0 && N >= 64 && (groups == 1 || ((epilogue == 0 || epilogue == 4) && K % blitz::kWideBK == 0 && N % 64 == 0));
}

// C = A W with the epilogues, pitches and diagonal blocks of blitz_gemm (N, K: of one block).
// Returns a cudaError_t value, -1 for arguments it cannot take, -2 when the TMA encoder is missing.
int blitz_gemm_wide(const void* A, int64_t lda, const void* W, int64_t ldb, void* C, int64_t ldc, const void* R, int M, int N, int K,
                    int epilogue, int up_col_off, int dtype, int static_b, int* status, float alpha, float beta, int groups,
                    int a_step, int c_step, cudaStream_t stream) {
  using namespace blitz;
  if (groups < 1 || !blitz_gemm_wide_supported(M, N, K, 0, epilogue, groups)) return -1;
  if ((lda & 7) || (ldb & 7) || (ldc & 7) || (epi_gated(epilogue) && (up_col_off & 7))) return -1;
  if (groups > 1 && (((a_step | c_step) & 7) || a_step < 0 || c_step < N)) return -1;
  WideParams p;
  p.C = C;
  p.R = R;
  p.alpha = alpha;
  p.beta = beta;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.num_kb = (K + kWideBK - 1) / kWideBK;
  const int cols = epi_gated(epilogue) ? 128 : 256;
  p.tiles_m = (M + 2 * kWideRows - 1) / (2 * kWideRows);
  p.group_tiles = (N + cols - 1) / cols;
  p.tiles_n = p.group_tiles * groups;
  p.up_col_off = up_col_off;
  p.groups = groups;
  p.a_step = groups > 1 ? a_step : 0;
  p.c_step = groups > 1 ? c_step : 0;
  p.static_b = static_b;
  p.status = status;
  const int pairs_max = device_sm_count() / 2;
  const int tiles = p.tiles_m * p.tiles_n;
  p.group_m = p.tiles_m < 8 ? p.tiles_m : 8;
  const int rest = tiles % pairs_max;
  p.full = 2 * rest <= pairs_max ? tiles - rest : tiles;
  p.items = p.full + 2 * (tiles - p.full);
  const int pairs = p.items < pairs_max ? p.items : pairs_max;

  CUtensorMap ta, tb, tb2, tc;
  if (!get_tmap_2d(&ta, A, (uint64_t)p.a_step * (groups - 1) + K, (uint64_t)M, (uint64_t)lda * 2, kWideBK, kWideRows)) return -2;
  const int w_cols = epi_gated(epilogue) ? up_col_off + N : N;
  if (!get_tmap_2d(&tb, W, (uint64_t)w_cols, (uint64_t)K * groups, (uint64_t)ldb * 2, 64, kWideBK)) return -2;
  p.slabs = w_cols % 64 == 0 && (!epi_gated(epilogue) || up_col_off % 64 == 0);
  tb2 = tb;
  if (p.slabs && !get_tmap_slabs(&tb2, W, (uint64_t)w_cols, (uint64_t)K * groups, (uint64_t)ldb * 2, kWideBK, 2)) return -2;
  if (epi_f32(epilogue)) {
    tc = ta;  // fp32 outputs are stored without TMA; the map is not used
  } else if (!get_tmap_2d(&tc, C, (uint64_t)p.c_step * (groups - 1) + N, (uint64_t)M, (uint64_t)ldc * 2, 64, 32)) {
    return -2;
  }
  return dtype == 1 ? wide_dispatch<__nv_bfloat16>(epilogue, ta, tb, tb2, tc, p, pairs, stream)
                    : wide_dispatch<__half>(epilogue, ta, tb, tb2, tc, p, pairs, stream);
}

}  // extern "C"
