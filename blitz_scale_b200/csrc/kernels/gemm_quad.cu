// Paired-SM tcgen05 GEMM with K in two halves over a cluster of four CTAs, for products of more than 128 rows that are one round of its
// tiles: one tile of 256 x 128 per cluster, at most as many as clusters are resident (the rule is in gemm_any.cu).
//
//   C[M,N] = A[M,K] * W[K,N]      W "in,out" (N contiguous), 16-bit, fp32 accumulation in TMEM
//
// At these sizes a product is a stream of weights (4096 x 14336: 117 MB, 18 us) that every SM has to take part in, beside the activations,
// which every column tile reads again.  Tiles as wide as gemm_wide.cu's leave half of the pairs idle; K cut into parts as in gemm_pair.cu
// sends 98 KB of sums per CTA through L2, which takes 8 us behind the last product.  Here a CTA pair multiplies 256 rows with 128 columns
// (per K block a CTA loads 16 KB of A and 8 KB of W), the two pairs of a cluster take half of K each, and their sums meet in distributed shared memory:
// a CTA hands 64 of its 128 columns, 32 KB, to its counterpart in the other pair and finishes the other 64.  The cluster's four CTAs so share the
// epilogue.  Measured behind a small kernel with cold weights, 256 rows, us (and the best of the other kernels):
// 4096 x 4096 14.2 (20.9), 4096 x 14336 34.0 (41.6).
//
// The parts are added in the order of K.  Epilogues: store, residual add (C may be R), fp32 outputs as in gemm_wide.cu; no gated units.
//
// Roles per CTA (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner (+ UMMA issuer in the pair's even CTA), warps 2..9 = epilogue
// (TMEM lane quarter = warp % 4, two warps per quarter, 32 columns each).
#include "launch.cuh"
#include "ptx.cuh"
#include "tmap.cuh"
#include "gemm_pair.cuh"
#include <type_traits>

namespace blitz {

constexpr int kQuadThreads = 320;
constexpr int kQuadBK = 64;
constexpr int kQuadRows = 128;                       // rows of A per CTA; a pair covers 256
constexpr int kQuadCols = 128;                       // columns of a tile; a CTA loads 64 of them and finishes 64 of them
constexpr int kQuadABytes = kQuadRows * kQuadBK * 2;
constexpr int kQuadStageBytes = kQuadABytes + 64 * kQuadBK * 2;
constexpr int kQuadStages = 8;
constexpr int kQuadStagingBytes = 4 * 4096;          // a box of 32 rows x 128 bytes per lane quarter
constexpr int kQuadZoneBytes = kQuadRows * 64 * 4;   // sums of the other half of K, over the stages
constexpr int kQuadBarrierBytes = (2 * kQuadStages + 1) * 8 + 16;
constexpr int kQuadSmemBytes = 1024 + kQuadStages * kQuadStageBytes + kQuadStagingBytes + kQuadBarrierBytes;
static_assert(kQuadSmemBytes <= 227 * 1024 && kQuadZoneBytes <= kQuadStages * kQuadStageBytes, "shared memory of one CTA");

struct QuadParams {
  void* C;         // fp32 outputs (the 16-bit ones are stored through tmap_c)
  const void* R;
  float alpha;     // axpy; soft cap
  int64_t ldc;
  int M, N, num_kb, half_kb;  // K blocks, and those of the first half
  int tiles_m;
  int static_b;    // W is not written by kernels still running in this stream
  int* status;
};

template <typename T, int EPI>
__global__ void __launch_bounds__(kQuadThreads, 1)
gemm_quad_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_c, const QuadParams p) {
  constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  constexpr uint32_t kIdesc = ptx::make_idesc_f16(kFmt, 0u, 1u, 2 * kQuadRows, kQuadCols);
  constexpr int S = kQuadStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint8_t* staging = smem + S * kQuadStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + kQuadStagingBytes);
  uint64_t* full_bar = bars;           // [S] used in the pair's even CTA: bytes of both CTAs
  uint64_t* empty_bar = bars + S;      // [S] per CTA: stage released by the pair's UMMAs
  uint64_t* tfull_bar = bars + 2 * S;  // per CTA: accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t crank = ptx::cluster_ctarank();
  const uint32_t rank = crank & 1u;                 // in the pair: 0 = even CTA (issues the UMMAs), 1 = odd CTA
  const int part = static_cast<int>(crank >> 1);    // which half of K
  const int tile = static_cast<int>(blockIdx.x >> 2);
  const int m0 = (tile % p.tiles_m) * 2 * kQuadRows + static_cast<int>(rank) * kQuadRows;
  const int n0 = (tile / p.tiles_m) * kQuadCols;
  const int kb_beg = part ? p.half_kb : 0, kb_end = part ? p.num_kb : p.half_kb;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 1);
    }
    ptx::mbar_init(tfull_bar, 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::tma_prefetch_desc(&tmap_a);
    ptx::tma_prefetch_desc(&tmap_b);
    ptx::tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, kQuadCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  // all CTAs have initialised their barriers before any signals another's
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  ptx::griddep_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (every CTA, own halves)
    if (ptx::elect_one()) {
      const uint32_t full0 = ptx::mapa_shared(ptx::smem_u32(full_bar), crank & ~1u);  // the even CTA's full barriers
      auto load_b = [&](int stage, int kb) {
        ptx::tma_load_2d_pair(smem + stage * kQuadStageBytes + kQuadABytes, &tmap_b, full0 + 8u * stage, n0 + static_cast<int>(rank) * 64, kb * kQuadBK);
      };
      auto load_a = [&](int stage, int kb) {
        ptx::tma_load_2d_pair(smem + stage * kQuadStageBytes, &tmap_a, full0 + 8u * stage, kb * kQuadBK, m0);
      };
      auto expect = [&](int stage) {
        if (rank == 0) ptx::mbar_expect_tx(&full_bar[stage], 2u * kQuadStageBytes);
      };
      // with static weights the first stages' weight tiles are requested before the dependency wait
      int npre = p.static_b ? min(S, kb_end - kb_beg) : 0;
      for (int i = 0; i < npre; ++i) {
        expect(i);
        load_b(i, kb_beg + i);
      }
      ptx::griddep_wait();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_beg; kb < kb_end; ++kb) {
        if (npre > 0) {
          load_a(stage, kb);
          --npre;
        } else {
          if (!ptx::bounded_mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) {
            if (p.status) atomicCAS(p.status, 0, kStatusTimeoutProducer);
            ok = false;
            break;
          }
          expect(stage);
          load_a(stage, kb);
          load_b(stage, kb);
        }
        if (++stage == S) { stage = 0; phase ^= 1u; }
      }
      // drain: the releases of the last stages are remote barrier signals; take them before the stages are written by others (a stage
      // that was never filled answers at once)
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
    // ------------------------------------------------------------ UMMA issuer (the pairs' even CTAs)
    ptx::griddep_wait();
    if (rank == 0 && ptx::elect_one()) {
      const uint16_t mask = static_cast<uint16_t>(3u << (crank & ~1u));
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_beg; kb < kb_end; ++kb) {
        if (!ptx::bounded_mbar_wait(&full_bar[stage], phase, abort_flag)) {
          if (p.status) atomicCAS(p.status, 0, kStatusTimeoutMma);
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t a_base = ptx::smem_u32(smem + stage * kQuadStageBytes);
        const uint32_t b_base = a_base + kQuadABytes;
#pragma unroll
        for (int k = 0; k < kQuadBK / 16; ++k) {
          // A: K-major, 128-byte rows, 8-row groups 1024 B apart; 16 K elements = 32 B.
          // W: N-major, one slab of 64 columns per CTA, 8-K-row groups 1024 B apart; 16 K rows = 2048 B.
          const uint64_t adesc = ptx::make_smem_desc(a_base + k * 32, 16, 1024, ptx::kLayoutSw128);
          const uint64_t bdesc = ptx::make_smem_desc(b_base + k * 2048, 8192, 1024, ptx::kLayoutSw128);
          ptx::umma_f16_ss_pair(tmem_base, adesc, bdesc, kIdesc, (kb != kb_beg || k != 0) ? 1u : 0u);
        }
        ptx::umma_commit_pair(&empty_bar[stage], mask);
        if (++stage == S) { stage = 0; phase ^= 1u; }
      }
      if (ok) ptx::umma_commit_pair(tfull_bar, mask);
    }
  } else {
    ptx::griddep_wait();
  }

  __syncwarp();  // lanes of the producer / issuer warps rejoin the elected one before the warp-aligned barriers
  // ------------------------------------------------------------ exchange of the halves, epilogue.  Every thread of the cluster executes
  // the barriers, whatever happened in its role.
  const bool epi = warp >= 2;
  const int q = warp & 3;                   // TMEM lane quarter this warp may read
  const int ch = ((warp - 2) >> 2) & 1;     // which 32 of 64 columns it takes
  const int row_in = q * 32 + lane, row = m0 + row_in;
  const bool row_ok = row < p.M;
  const bool quarter_ok = m0 + q * 32 < p.M;  // the same for both warps of a quarter, and for their counterparts in the other pair
  const int n = n0 + part * 64;             // first column this CTA finishes
  const int col0 = n + ch * 32;             // first of this thread's columns
  const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
  uint4 res[4] = {};
  bool ready = false;
  if (epi) {
    if (EPI == 1) {
      const T* Rp = reinterpret_cast<const T*>(p.R) + static_cast<int64_t>(row) * p.ldc + col0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row_ok && col0 + 8 * j < p.N) res[j] = *reinterpret_cast<const uint4*>(Rp + 8 * j);
    }
    ready = ptx::bounded_mbar_wait(tfull_bar, 0, abort_flag);
    if (!ready) *abort_flag = 1;
    if (!ready && p.status && lane == 0) atomicCAS(p.status, 0, kStatusTimeoutEpilogue);
    ptx::tc_fence_after_sync();
  }
  // barrier 1: both pairs have finished their UMMAs, so nobody's stages are read or written any more
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  ready = epi && *abort_flag == 0;  // (the same for all of the CTA's warps, which meet again below)
  const uint32_t zone = ptx::smem_u32(smem) + static_cast<uint32_t>(ch * 8 * kQuadRows + row_in) * 16u;  // [column / 4][row][4]
  if (ready && quarter_ok) {
    const uint32_t dst = ptx::mapa_shared(zone, crank ^ 2u);
    uint32_t v[32];
    ptx::tmem_ld_32x32(taddr + (1 - part) * 64 + ch * 32, v);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) ptx::st_shared_cluster_v4(dst + j * (kQuadRows * 16), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
  // barrier 2: the other half's sums are in place
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  if (ready && quarter_ok && n < p.N) {
    uint32_t v[32];
    float g[32];
    ptx::tmem_ld_32x32(taddr + part * 64 + ch * 32, v);
    ptx::tmem_ld_wait();
    const float4* other = reinterpret_cast<const float4*>(smem + (static_cast<size_t>(ch) * 8 * kQuadRows + row_in) * 16);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 f = other[j * kQuadRows];
      g[4 * j] = __uint_as_float(v[4 * j]) + f.x;
      g[4 * j + 1] = __uint_as_float(v[4 * j + 1]) + f.y;
      g[4 * j + 2] = __uint_as_float(v[4 * j + 2]) + f.z;
      g[4 * j + 3] = __uint_as_float(v[4 * j + 3]) + f.w;
    }
    if (epi_f32(EPI)) {
      // a thread's 32 columns are a whole 128-byte line
      if (row_ok) {
        float* dst = reinterpret_cast<float*>(p.C) + static_cast<int64_t>(row) * p.ldc + col0;
        const float inv = EPI == 6 ? 1.f / p.alpha : 0.f;
        float old[4][8] = {};
        if (EPI == 5) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col0 + 8 * j < p.N) ptx::ld_global_v8(dst + 8 * j, old[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (col0 + 8 * j < p.N) {
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
    } else {
      uint4 o4[4];
      pair_convert32<T, EPI>(g, g, res, o4);
      // 128-byte rows, 16-byte chunks XOR-swizzled by row: the layout the TMA store expects
      uint8_t* box = staging + q * 4096;
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(box + lane * 128 + (((ch * 4 + j) ^ (lane & 7)) << 4)) = o4[j];
      ptx::fence_proxy_async_smem();
      asm volatile("bar.sync %0, 64;" ::"r"(3 + q) : "memory");
      if (ch == 0 && lane == 0) {
        ptx::tma_store_2d(&tmap_c, box, n, m0 + q * 32);
        ptx::tma_store_commit();
        ptx::tma_store_wait<0>();  // the box has been written out before the CTA may exit
      }
    }
  }

  __syncwarp();
  ptx::tc_fence_before_sync();
  __syncthreads();
  // neither CTA of a pair leaves (or frees TMEM) while its partner reads its accumulator
  ptx::cluster_arrive_release();
  ptx::cluster_wait_acquire();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, kQuadCols);
  }
}

template <typename T, int EPI>
static int quad_launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const QuadParams& p, int tiles, cudaStream_t stream) {
  auto kern = gemm_quad_kernel<T, EPI>;
  static PerDeviceOnce once;
  cudaError_t e = once.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kQuadSmemBytes); });
  if (e != cudaSuccess) return static_cast<int>(e);
  return static_cast<int>(launch_pdl_cluster(kern, dim3(4 * tiles), dim3(kQuadThreads), (size_t)kQuadSmemBytes, 4u, stream, ta, tb, tc, p));
}

template <typename T>
static int quad_dispatch(int epilogue, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const QuadParams& p, int tiles,
                         cudaStream_t stream) {
  switch (epilogue) {
    case 1: return quad_launch<T, 1>(ta, tb, tc, p, tiles, stream);
    case 4: return quad_launch<T, 4>(ta, tb, tc, p, tiles, stream);
    case 5: return quad_launch<T, 5>(ta, tb, tc, p, tiles, stream);
    case 6: return quad_launch<T, 6>(ta, tb, tc, p, tiles, stream);
    default: return quad_launch<T, 0>(ta, tb, tc, p, tiles, stream);
  }
}

}  // namespace blitz

extern "C" {

// Whether blitz_gemm_quad takes this problem: "in,out" weights, whole 16-byte rows, two K blocks, no gated unit.
int blitz_gemm_quad_supported(int M, int N, int K, int b_layout, int epilogue) {
  return M >= 1 && b_layout == 0 && (epilogue == 0 || epilogue == 1 || (epilogue >= 4 && epilogue <= 6)) && (N & 7) == 0 && (K & 7) == 0 && N >= 64 &&
         K > blitz::kQuadBK;
}

// How many of this kernel's clusters the current device holds at once (0: no device to ask).
int blitz_gemm_quad_resident() {
  using namespace blitz;
  auto kern = gemm_quad_kernel<__nv_bfloat16, 0>;  // (threads and shared memory are the same for all of them)
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kQuadSmemBytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return max_active_clusters(kern, dim3(kQuadThreads), kQuadSmemBytes, 4u);
}

// C = A W with the epilogues and pitches of blitz_gemm.
// Returns a cudaError_t value, -1 for arguments it cannot take, -2 when the TMA encoder is missing.
int blitz_gemm_quad(const void* A, int64_t lda, const void* W, int64_t ldb, void* C, int64_t ldc, const void* R, int M, int N, int K,
                    int epilogue, int dtype, int static_b, int* status, float alpha, cudaStream_t stream) {
  using namespace blitz;
  if (!blitz_gemm_quad_supported(M, N, K, 0, epilogue) || (lda & 7) || (ldb & 7) || (ldc & 7)) return -1;
  QuadParams p;
  p.C = C;
  p.R = R;
  p.alpha = alpha;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.num_kb = (K + kQuadBK - 1) / kQuadBK;
  p.half_kb = (p.num_kb + 1) / 2;
  p.tiles_m = (M + 2 * kQuadRows - 1) / (2 * kQuadRows);
  p.static_b = static_b;
  p.status = status;
  const int tiles = p.tiles_m * ((N + kQuadCols - 1) / kQuadCols);
  CUtensorMap ta, tb, tc;
  if (!get_tmap_2d(&ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, kQuadBK, kQuadRows)) return -2;
  if (!get_tmap_2d(&tb, W, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, kQuadBK)) return -2;
  if (epi_f32(epilogue)) {
    tc = ta;  // fp32 outputs are stored without TMA; the map is not used
  } else if (!get_tmap_2d(&tc, C, (uint64_t)N, (uint64_t)M, (uint64_t)ldc * 2, 64, 32)) {
    return -2;
  }
  return dtype == 1 ? quad_dispatch<__nv_bfloat16>(epilogue, ta, tb, tc, p, tiles, stream) : quad_dispatch<__half>(epilogue, ta, tb, tc, p, tiles, stream);
}

}  // extern "C"
