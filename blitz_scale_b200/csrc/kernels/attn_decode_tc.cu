// Paged-KV decode attention, tensor-core version (the serving path).
//
// Decode attention is a stream over the K and V pages of every sequence; with
// GQA the 4-8 query heads that share a KV head turn the per-token work into a
// small matrix product, so the FLOPs go to mma.sync (m16n8k16, query heads
// padded to 16 rows) and the instruction stream per token drops ~10x against a
// CUDA-core dot product; the kernel is then bound by HBM as it should be.
// tcgen05 is not used here on purpose: its minimum M of 64 rows would waste
// 94 % of each instruction on padding for one query token per sequence.
//
// Data movement: a producer warp walks the page table and issues TMA
// (cp.async.bulk.tensor.3d, plain per-CTA loads) boxes of [tokens x 64 dims]
// straight from the paged layout [page][K|V][token][kv_head][head_dim] into
// 128-byte-swizzled shared memory, six stages of 64 tokens (192 KB in flight
// per SM for head_dim 128).  The four consumer warps of a half each own 16 of the 64 tokens
// of a stage: S = Q K^T via ldmatrix + mma, online softmax in registers
// (exp2, fp32), O += P V via ldmatrix.trans + mma.  Warps merge their partial
// (m, l, O) through shared memory; with num_splits > 1 each item writes an fp32
// partial and a merge kernel combines the splits (flash-decoding).
//
// The kernel is persistent: one CTA per SM walks its pieces of work and the TMA pipeline runs across their
// boundaries, so it never drains between sequences.  It is launched with programmatic dependent launch: shared
// memory is cleared and the barriers are set up while the previous kernel is
// still running; the first load waits for it.
//
// A CTA is two independent halves, each with a producer warp, a ring of three stages and four consumer warps: a chunk's chain of
// waits, products, maxima and exponentials takes a group of warps about twice as long as memory takes to deliver it (one group with
// six stages: 0.87 us a chunk even out of L2, against 0.72 at the full HBM rate), and what follows a piece's last chunk (merge over
// the warps, division, store) runs beside the other half's chunks.  Measured, 32 query and 8 KV heads of 128, 256 x 513 tokens,
// whole sequences: 111 us with one group, 98 us so (5.5 TB/s).
//
// Pieces.  num_splits >= 1: (sequence, KV head, split) items in a grid-stride loop over the halves.  num_splits = 0: the
// chunks of all sequences laid end to end are cut into equal contiguous ranges, as many as there are halves per KV head, and every half takes one head of one range, so that neither a long sequence nor a small batch leaves SMs idle; the halves that
// stream the heads of the same tokens do so at the same time (a token's heads are neighbours in memory).  A range's first and last
// sequence may be incomplete: such pieces go to scratch as fp32 partials, and whichever half finishes an item's last piece combines them (in the order of the ranges, so that the
// result does not depend on who that is).  Every half computes the ranges itself from the page table (a scan over the batch in
// shared memory), so the launch does not depend on the lengths and replays from a CUDA graph.  Measured: 61 sequences of 170 .. 3500
// tokens (67 k in all) 57 us, 82 us as whole sequences and 104 us as those before the halves.  An incomplete piece costs about 4 us
// (fence, ticket, merge), all of them about 7 us a launch: which division serves a batch is measured at decode_parts (runtime/engine.py).
//
// Models that ask for it get a sliding window with kept first tokens (only the 64-token chunks that hold a visible key
// are fetched: a sequence costs at most window + kept tokens whatever its length), soft-capped scores
// (cap * tanh(s / cap)) and a per-head sink, a term e^sink in the softmax denominator, which the merge adds once.
//
// The cache must hold finite values in every slot of an allocated page (the
// pool is zero-filled at creation): masked positions get probability 0, and
// 0 x NaN would still poison the accumulator.
//
// Keys and values may differ in size, and either may be smaller than the tile it is computed in (64 or 128 columns, a
// multiple of 8): TMA fills the columns behind a head's end with zeros.  A gate (one number per head and row, through a
// sigmoid) multiplies a head's output as it is stored.  More than 8 query heads per KV head run as several groups that
// read the same keys and values (the second one from L2).
//
// A bias by distance per head, bias[h][min(i - j, bias_len - 1)], is added to the scaled scores; only chunks with a distance
// inside the table look it up (four entries a lane, requested before the wait for the chunk).
//
// The window may be a chunk counted from position 0 (`chunked`: the keys of the position's own chunk are visible), and weights may
// be sigmoids of the scores instead of a softmax (`sigmoid`): then nothing refers to a maximum or is normalised, and warps and
// splits just add up.
//
// Replaces src/kernel/attention_decode.cu:13-40 and the host-side plan of
// src/kernel/flashinfer_types.cu:52-80.
#include "launch.cuh"
#include "ptx.cuh"
#include "tmap.cuh"
#include "common.cuh"
#include "mma.cuh"
#include "scalar.cuh"

namespace blitz {

constexpr int kTcThreads = 2 * 128 + 2 * 32;  // four consumer warps per half, then a producer warp per half
constexpr int kTcMaxShared = 256;     // sequences, and heads of each, whose chunks can be dealt out (num_splits = 0)
constexpr int kTcMaxSharedHeads = 128;
constexpr int kTcChunk = 64;
constexpr int kTcHalves = 2;
constexpr int kTcStages = 3;          // of a half
constexpr int kTcSlabBytes = kTcChunk * 128;

struct DecodeTcParams {
  const void* q;
  int64_t q_stride;
  const int32_t* indices;
  const int32_t* indptr;
  const int32_t* last_page_len;
  void* out;
  int64_t out_stride;
  float* part_o;
  float* part_lse;
  int batch, q_heads, kv_heads, group, page_size, max_pages, num_splits, box_tokens;
  int kv_div;               // kv_heads counts groups of at most 8 query heads: kv_div of them share a KV head
  int dim, vdim, page_rows; // page n's token `off` is row n * page_rows + off of both pools
  int v_rows;               // > 0: one tensor (and one map) for keys and values, which lie this many rows behind their keys
  const void* gate;         // [batch][gate_stride], a column per query head, or null
  int64_t gate_stride;
  int tail_box_tokens;  // box height of the second tensor map, used for the last (partly filled) chunk of a sequence
  float scale_log2;
  int chunked, sigmoid;         // see the top of the file
  int window, keep_first;       // 0: every key; else a token sees the last `window` positions and the first `keep_first`
  float cap_scale, cap_log2;    // soft cap (cap_log2 > 0): score in log2 units = cap_log2 * tanh(q.k * cap_scale)
  const void* sink;             // [q_heads] in the activation type, or null
  const void* bias;             // [q_heads][bias_len] in the activation type, or null
  int bias_len;
  int static_table;             // indices, indptr and last_page_len are not written by kernels still running in this stream
  unsigned* tickets;            // num_splits = 0: [batch][kv_heads] pieces finished, zero between launches
  int* status;
};

template <int HD, int VD = HD>
struct TcCfg {
  static constexpr int kSlabs = HD / 64, kValueSlabs = VD / 64;
  static constexpr int kStageBytes = (kSlabs + kValueSlabs) * kTcSlabBytes;
  static constexpr int kMergeFloats = 4 * 8 * VD + 2 * 4 * 8;  // of one half
  static constexpr int kSmemBytes = kTcHalves * (kTcStages * kStageBytes + kMergeFloats * 4) + (kTcMaxShared + 1) * 4 + 1024 + 124;
};

template <typename T>
__device__ __forceinline__ float head_gate(const T* z) { return 1.f / (1.f + expf(-to_f<T>(*z))); }

// A piece of work: chunks c_beg .. c_end of the visible chunks of (sequence b, KV head h).
struct DecItem {
  int b, h, kv_head, pg_beg, seq_len, c_beg, c_end;
  int part;              // where its partial result goes (in units of a group of heads); -1: it is the whole item
  int lo, first;         // visible keys: [0, first) and [lo, seq_len)
  int n_first, c_window; // chunks of the kept tokens; first chunk of the window behind them
  // the n-th visible chunk
  __device__ __forceinline__ int chunk(int n) const { return n < n_first ? n : c_window + n - n_first; }
};
// Lengths and visible chunks of a sequence; returns the number of the latter.
__device__ __forceinline__ int dec_sequence(const DecodeTcParams& p, int b, DecItem& it) {
  it.b = b;
  it.pg_beg = p.indptr[b];
  const int npages = p.indptr[b + 1] - it.pg_beg;
  it.seq_len = npages > 0 ? (npages - 1) * p.page_size + p.last_page_len[b] : 0;
  it.lo = p.window > 0 ? (p.chunked ? max(0, it.seq_len - 1) / p.window * p.window : max(0, it.seq_len - p.window)) : 0;
  it.first = min(p.keep_first, it.lo);
  it.n_first = (it.first + kTcChunk - 1) / kTcChunk;
  it.c_window = max(it.lo / kTcChunk, it.n_first);
  return it.n_first + max(0, (it.seq_len + kTcChunk - 1) / kTcChunk - it.c_window);
}
// The pieces of a half, one after the other.
struct DecWalk {
  int x, end;        // items of a grid-stride loop, or chunks of a range
  int self, halves;  // which half of how many
  int b, h;          // (of a range) sequence that chunk x belongs to, head
  bool first;        // nothing has been taken from the range yet
};
// Ranges: how many, where one begins, which one a chunk is in.  (No range is empty.  A few hundred ranges of fewer than seven million
// chunks stay within 32 bits: a 64-bit division takes about a fifth of a microsecond, and several follow one another here.)
__device__ __forceinline__ unsigned dec_ranges(const DecodeTcParams& p, unsigned chunks, unsigned halves) { return min(chunks, halves / static_cast<unsigned>(p.kv_heads)); }
__device__ __forceinline__ int dec_range_begin(unsigned r, unsigned chunks, unsigned ranges) { return static_cast<int>(chunks * r / ranges); }
__device__ __forceinline__ int dec_range_of(unsigned x, unsigned chunks, unsigned ranges) { return static_cast<int>(((x + 1) * ranges + chunks - 1) / chunks) - 1; }
__device__ __forceinline__ DecWalk dec_walk(const DecodeTcParams& p, const int* before, int half) {
  DecWalk w;
  w.halves = kTcHalves * static_cast<int>(gridDim.x);
  w.self = w.x = half * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);  // (little work: one half of every SM)
  w.end = p.batch * p.kv_heads * p.num_splits;
  w.b = w.h = 0;
  w.first = true;
  if (p.num_splits == 0) {
    const int chunks = before[p.batch], ranges = dec_ranges(p, chunks, w.halves), r = static_cast<unsigned>(w.self) / static_cast<unsigned>(p.kv_heads);
    w.h = w.self - r * p.kv_heads;
    w.x = r < ranges ? dec_range_begin(r, chunks, ranges) : 0;
    w.end = r < ranges ? dec_range_begin(r + 1, chunks, ranges) : 0;
    int lo = 0, hi = p.batch - 1;  // the last sequence that starts at or before x (empty ones in front of it are passed over)
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (before[mid] <= w.x) lo = mid;
      else hi = mid - 1;
    }
    w.b = lo;
  }
  return w;
}
__device__ __forceinline__ bool dec_next(const DecodeTcParams& p, const int* before, DecWalk& w, DecItem& it) {
  if (w.x >= w.end) return false;
  if (p.num_splits > 0) {
    const int item = w.x, split = item % p.num_splits;
    it.h = (item / p.num_splits) % p.kv_heads;
    const int n = dec_sequence(p, item / (p.num_splits * p.kv_heads), it), cps = (n + p.num_splits - 1) / p.num_splits;
    it.c_beg = min(n, split * cps);
    it.c_end = min(n, (split + 1) * cps);
    it.part = p.num_splits == 1 ? -1 : split;
    w.x += w.halves;
  } else {
    while (before[w.b + 1] <= w.x) ++w.b;
    const int n = dec_sequence(p, w.b, it);
    it.h = w.h;
    it.c_beg = w.x - before[w.b];
    it.c_end = min(n, it.c_beg + w.end - w.x);
    it.part = it.c_end - it.c_beg == n ? -1 : w.self * 2 + (w.first ? 0 : 1);
    w.x += it.c_end - it.c_beg;
    w.first = false;
  }
  it.kv_head = p.kv_div == 1 ? it.h : it.h / p.kv_div;
  return true;
}
// Combines the pieces of head h of a sequence whose first chunk is number `start`, in ranges c0 .. c1, for query head gg of its group;
// the calling warp has seen that all of them are in memory.
template <typename T>
__device__ __forceinline__ void dec_merge(const DecodeTcParams& p, int b, int h, int gg, int start, int c0, int c1, int chunks, int ranges) {
  const int lane = threadIdx.x & 31, head = h * p.group + gg;
  // a range's first piece is in its half's first place: lane i looks up that of the i-th of 32 ranges
  auto place = [&](int c) { return ((c * p.kv_heads + h) * 2 + (dec_range_begin(c, chunks, ranges) >= start ? 0 : 1)) * p.group + gg; };
  const int first = c0 + lane <= c1 ? place(c0 + lane) : 0;
  const float first_lse = c0 + lane <= c1 ? __ldcg(p.part_lse + first) : -INFINITY;
  const float snk = p.sink ? to_f<T>(reinterpret_cast<const T*>(p.sink)[head]) * 1.4426950408889634f : -INFINITY;
  float M = fmaxf(snk, first_lse);
  for (int c = c0 + 32 + lane; c <= c1; c += 32) M = fmaxf(M, __ldcg(p.part_lse + place(c)));
#pragma unroll
  for (int d = 16; d; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, sum = 0.f;
  if (M > -INFINITY) {
    for (int c = c0; c <= c1; c += 32) {
      const int here = min(32, c1 - c + 1), at = c == c0 ? first : lane < here ? place(c + lane) : 0;
      const float w0 = lane < here ? exp2f((c == c0 ? first_lse : __ldcg(p.part_lse + at)) - M) : 0.f;
#pragma unroll 8
      for (int i = 0; i < here; ++i) {
        const float w = __shfl_sync(0xffffffffu, w0, i);
        const float* o = p.part_o + static_cast<int64_t>(__shfl_sync(0xffffffffu, at, i)) * p.vdim;
        sum += w;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (lane + 32 * k < p.vdim) acc[k] += w * __ldcg(o + lane + 32 * k);
      }
    }
    if (p.sink) sum += exp2f(snk - M);
  }
  if (p.sigmoid) sum = 1.f;  // (every piece's reference is zero: the weights are ones)
  const float g = p.gate ? 1.f / (1.f + expf(-to_f<T>(reinterpret_cast<const T*>(p.gate)[b * p.gate_stride + head]))) : 1.f;
  T* out = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(b) * p.out_stride + static_cast<int64_t>(head) * p.vdim;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (lane + 32 * k < p.vdim) stf(out + lane + 32 * k, sum > 0.f ? acc[k] / sum * g : 0.f);
}

// PLAIN: heads as large as the tiles, one tensor for keys and values, no gate, at most 8 query heads per KV head.
template <typename T, int HD, int VD = HD, bool PLAIN = true>
__global__ void __launch_bounds__(kTcThreads, 1)
attn_decode_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_k_tail,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_v_tail,
                      const DecodeTcParams p) {
  using Cfg = TcCfg<HD, VD>;
  constexpr int SL = Cfg::kSlabs, SV = Cfg::kValueSlabs;
  const int dim = PLAIN ? HD : p.dim, vdim = PLAIN ? VD : p.vdim;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = ptx::smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  float* mrg = reinterpret_cast<float*>(smem + kTcHalves * kTcStages * Cfg::kStageBytes);  // per half: [4][8][VD], [4][8], [4][8]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(mrg + kTcHalves * Cfg::kMergeFloats);   // [half][stage]
  uint64_t* empty_bar = full_bar + kTcHalves * kTcStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty_bar + kTcHalves * kTcStages);
  volatile int* last_piece = abort_flag + 1;                              // [half]
  int* before = const_cast<int*>(last_piece) + kTcHalves;  // num_splits = 0: [batch + 1] chunks (of one head) of the sequences before each

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.group;

  // zero the stages once: rows a short last chunk never fills must stay finite
  for (int i = threadIdx.x; i < kTcHalves * kTcStages * Cfg::kStageBytes / 16; i += kTcThreads)
    reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
  if (threadIdx.x == 0) {
    for (int i = 0; i < kTcHalves * kTcStages; ++i) {
      ptx::mbar_init(&full_bar[i], 1);
      ptx::mbar_init(&empty_bar[i], 4);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::tma_prefetch_desc(&tmap_k);
    ptx::tma_prefetch_desc(&tmap_v);
    ptx::tma_prefetch_desc(&tmap_k_tail);
    ptx::tma_prefetch_desc(&tmap_v_tail);
  }
  ptx::fence_proxy_async_smem();
  __syncthreads();
  // programmatic dependent launch: the set-up above may overlap the previous kernel; q and the KV pages
  // are its outputs, so wait before the first load
  ptx::griddep_launch_dependents();
  if (!p.static_table) ptx::griddep_wait();
  if (p.num_splits == 0) {
    DecItem seq;
    if (threadIdx.x < p.batch) before[threadIdx.x + 1] = dec_sequence(p, threadIdx.x, seq);
    __syncthreads();
    if (warp == 0) {
      int n[kTcMaxShared / 32], sum = 0;
#pragma unroll
      for (int i = 0; i < kTcMaxShared / 32; ++i) {
        const int b = lane * (kTcMaxShared / 32) + i;
        n[i] = b < p.batch ? before[b + 1] : 0;
        sum += n[i];
      }
      int total = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, total, d);
        if (lane >= d) total += up;
      }
      int run = total - sum;
      if (lane == 0) before[0] = 0;
#pragma unroll
      for (int i = 0; i < kTcMaxShared / 32; ++i) {
        const int b = lane * (kTcMaxShared / 32) + i;
        run += n[i];
        if (b < p.batch) before[b + 1] = run;
      }
    }
    __syncthreads();
  }

  const int half = warp < 8 ? warp >> 2 : warp - 8;
  smem += half * kTcStages * Cfg::kStageBytes;
  full_bar += half * kTcStages;
  empty_bar += half * kTcStages;
  if (warp >= 8) {
    // ------------------------------------------------------------ producer (a whole warp; one lane issues)
    // A TMA box can only be issued once its page id is known, and a page id read from global memory right before
    // the issue costs one memory latency per chunk, which by itself is more than HBM's time for the chunk.  So the
    // warp reads page ids 32 at a time (one coalesced load, lane l keeps entry l of the window), hands them out by
    // shuffle, and requests the next item's page-table window and lengths while the current item streams.
    const int ps = p.page_size;
    auto load_window = [&](const DecItem& it, int first_page) -> int {
      const int npages = p.indptr[it.b + 1] - it.pg_beg;
      return (first_page + lane < npages) ? p.indices[it.pg_beg + first_page + lane] : 0;
    };
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    DecWalk walk = dec_walk(p, before, half);
    DecItem it{}, nit{};
    bool more = dec_next(p, before, walk, it);
    int win_base = more ? (it.chunk(it.c_beg) * kTcChunk) / ps : 0;
    int win = more ? load_window(it, win_base) : 0;
    ptx::griddep_wait();
    while (more && ok) {
      // next piece's metadata and first window: in flight while this one streams
      more = dec_next(p, before, walk, nit);
      const int nwin_base = more ? (nit.chunk(nit.c_beg) * kTcChunk) / ps : 0;
      const int nwin = more ? load_window(nit, nwin_base) : 0;
      for (int c = it.c_beg; c < it.c_end && ok; ++c) {
        const int tok0 = it.chunk(c) * kTcChunk;
        const int ntok = min(kTcChunk, it.seq_len - tok0);
        // a full chunk comes in boxes of box_tokens rows; the last chunk of a sequence only as far as it is
        // filled, in the smaller boxes of the second map (a 64-token page with 18 live tokens costs 32 rows)
        const bool tail = ntok < kTcChunk;
        const int bt = tail ? p.tail_box_tokens : p.box_tokens;
        const CUtensorMap* tk = tail ? &tmap_k_tail : &tmap_k;
        const CUtensorMap* tv = PLAIN || p.v_rows > 0 ? tk : tail ? &tmap_v_tail : &tmap_v;
        const uint32_t box_bytes = static_cast<uint32_t>(bt) * 128u;
        const int pieces = (ntok + bt - 1) / bt;
        const int last_page = (tok0 + ntok - 1) / ps;
        if (last_page >= win_base + 32) {  // sequences of more than 32 pages: move the window
          win_base = tok0 / ps;
          win = load_window(it, win_base);
        }
        // every lane waits, so that the warp stays converged
        ok = __all_sync(0xffffffffu, ptx::bounded_mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag));
        if (!ok) {
          if (p.status && lane == 0) atomicCAS(p.status, 0, kStatusTimeoutProducer);
          break;
        }
        if (ptx::elect_one()) ptx::mbar_expect_tx(&full_bar[stage], static_cast<uint32_t>(pieces) * (SL + SV) * box_bytes);
        uint8_t* sb = smem + stage * Cfg::kStageBytes;
        for (int i = 0; i < pieces; ++i) {
          const int t = tok0 + i * bt;
          int page = __shfl_sync(0xffffffffu, win, (t / ps - win_base) & 31);
          if (page < 0 || page >= p.max_pages) {
            if (p.status && lane == 0) atomicCAS(p.status, 0, kStatusBadIndex);
            page = 0;
          }
          if (ptx::elect_one()) {
            const int z = page * (PLAIN ? 2 * ps : p.page_rows) + (t % ps), h = PLAIN ? it.h : it.kv_head;
#pragma unroll
            for (int s = 0; s < (SL > SV ? SL : SV); ++s) {
              if (s < SL) ptx::tma_load_3d(sb + s * kTcSlabBytes + i * box_bytes, tk, &full_bar[stage], s * 64, h, z);
              if (s < SV) ptx::tma_load_3d(sb + (SL + s) * kTcSlabBytes + i * box_bytes, tv, &full_bar[stage], s * 64, h, z + (PLAIN ? ps : p.v_rows));
            }
          }
        }
        if (++stage == kTcStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      it = nit;
      win_base = nwin_base;
      win = nwin;
    }
  } else {
    // ------------------------------------------------------------ consumers (128 threads per half, named barrier 1 + half)
    const int wg = warp & 3, tid = threadIdx.x & 127;
    float* mrg_o = mrg + half * Cfg::kMergeFloats;
    float* mrg_m = mrg_o + 4 * 8 * VD;
    float* mrg_l = mrg_m + 32;
    auto meet = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); };
    const int g = lane >> 2, t4 = lane & 3;
    const int tokw = wg * 16;
    const int mi = lane >> 3, mr = lane & 7;  // ldmatrix: matrix index and row within it
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;  // after a timeout this warp stops waiting but keeps meeting the others at the barriers
    // The consumers stop consuming between two items (merge, then the next item's lengths and query rows), and a
    // pause longer than the pipeline can absorb empties the memory pipe, which then costs a full latency to refill.
    // So the next item's descriptor and Q fragments are requested while the current item is being processed.
    auto load_q = [&](const DecItem& d, uint32_t (&a0)[HD / 16], uint32_t (&a2)[HD / 16]) {
      // Q as A fragments (rows >= G and columns >= dim are zero padding; rows 8..15 are never populated since G <= 8)
      const int cols = g < G ? dim : 0;
      const T* qrow = reinterpret_cast<const T*>(p.q) + static_cast<int64_t>(d.b) * p.q_stride +
                      static_cast<int64_t>(d.h * G + g) * dim;
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        a0[ks] = ks * 16 < cols ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * t4) : 0u;
        a2[ks] = ks * 16 + 8 < cols ? *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * t4 + 8) : 0u;
      }
    };
    DecWalk walk = dec_walk(p, before, half);
    DecItem it{}, nit{};
    bool more = dec_next(p, before, walk, it);
    ptx::griddep_wait();
    if (p.num_splits == 0 && half == 0)  // sequences without a visible key are in nobody's range: their output is zero
      for (int b = blockIdx.x; b < p.batch; b += gridDim.x)
        if (before[b] == before[b + 1])
          for (int e = tid; e < p.q_heads * vdim; e += 128) stf(reinterpret_cast<T*>(p.out) + static_cast<int64_t>(b) * p.out_stride + e, 0.f);
    uint32_t qa0[HD / 16], qa2[HD / 16];
    if (more) load_q(it, qa0, qa2);
    while (more) {
      uint32_t nqa0[HD / 16], nqa2[HD / 16];
      more = dec_next(p, before, walk, nit);
      if (more) load_q(nit, nqa0, nqa2);
      float o[VD / 8][4];
#pragma unroll
      for (int i = 0; i < VD / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
      float m = -INFINITY, l = 0.f;
      const T* bias_row = nullptr;
      float far_bias = 0.f;
      if (!PLAIN && p.bias != nullptr && g < G) {
        bias_row = reinterpret_cast<const T*>(p.bias) + static_cast<int64_t>(it.h * G + g) * p.bias_len;
        far_bias = to_f<T>(bias_row[p.bias_len - 1]) * 1.4426950408889634f;
      }
      for (int c = it.c_beg; c < it.c_end; ++c) {
        float bias[4] = {far_bias, far_bias, far_bias, far_bias};  // of the lane's four keys, in log2 units
        if (!PLAIN && bias_row != nullptr) {
          const int d0 = it.seq_len - 1 - (it.chunk(c) * kTcChunk + tokw + 2 * t4);  // distance of the first of them
          if (it.seq_len - 1 - (it.chunk(c) * kTcChunk + tokw + 15) < p.bias_len - 1) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              bias[k] = to_f<T>(bias_row[min(max(d0 - (k & 1) - (k >> 1) * 8, 0), p.bias_len - 1)]) * 1.4426950408889634f;
          }
        }
        if (ok && !ptx::bounded_mbar_wait(&full_bar[stage], phase, abort_flag)) {
          if (p.status && lane == 0) atomicCAS(p.status, 0, kStatusTimeoutEpilogue);
          ok = false;
        }
        const int tok0 = it.chunk(c) * kTcChunk;
        const int nvalid = min(kTcChunk, it.seq_len - tok0);
        // visible keys of this warp's 16: below `kept` or from `from` on (both relative to the chunk)
        const int kept = it.first - tok0, from = it.lo - tok0;
        if (ok && tokw < nvalid && (tokw < kept || (tokw + 16 > from && nvalid > from))) {
          const uint32_t kbase = ptx::smem_u32(smem + stage * Cfg::kStageBytes);
          const uint32_t vbase = kbase + SL * kTcSlabBytes;
          float s_lo[4] = {0.f, 0.f, 0.f, 0.f}, s_hi[4] = {0.f, 0.f, 0.f, 0.f};
          {
            const int tok = tokw + (mi >> 1) * 8 + mr;
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
              const int ch = ks * 2 + (mi & 1);
              const uint32_t addr = kbase + (ch >> 3) * kTcSlabBytes + tok * 128 + (((ch & 7) ^ (tok & 7)) << 4);
              uint32_t b0, b1, b2, b3;
              ldmatrix_x4(addr, b0, b1, b2, b3);
              mma16816<T>(s_lo, qa0[ks], 0u, qa2[ks], 0u, b0, b1);
              mma16816<T>(s_hi, qa0[ks], 0u, qa2[ks], 0u, b2, b3);
            }
          }
          const int col = tokw + 2 * t4;
          auto visible = [&](int k) { return k < nvalid && (k >= from || k < kept); };
          const bool v0 = visible(col), v1 = visible(col + 1), v2 = visible(col + 8), v3 = visible(col + 9);
          auto score = [&](float x) {  // log2 units
            return p.cap_log2 > 0.f ? p.cap_log2 * ptx::tanh_ex2(x * p.cap_scale) : x * p.scale_log2;
          };
#pragma unroll
          for (int k = 0; k < 2; ++k) {  // rows 8..15 of the fragments are padding
            s_lo[k] = score(s_lo[k]) + (PLAIN ? 0.f : bias[k]);
            s_hi[k] = score(s_hi[k]) + (PLAIN ? 0.f : bias[2 + k]);
          }
          const bool plain_sum = !PLAIN && p.sigmoid;
          float mx = plain_sum ? 0.f : -INFINITY;
          if (!plain_sum) {
            if (v0) mx = fmaxf(mx, s_lo[0]);
            if (v1) mx = fmaxf(mx, s_lo[1]);
            if (v2) mx = fmaxf(mx, s_hi[0]);
            if (v3) mx = fmaxf(mx, s_hi[1]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          }
          const float m_new = fmaxf(m, mx);
          const float alpha = exp2f(m - m_new);  // m = -inf -> 0
          auto weight = [&](float x) { return plain_sum ? __fdividef(1.f, 1.f + exp2f(fminf(-x, 120.f))) : exp2f(x - m_new); };
          const float p0 = v0 ? weight(s_lo[0]) : 0.f;
          const float p1 = v1 ? weight(s_lo[1]) : 0.f;
          const float p2 = v2 ? weight(s_hi[0]) : 0.f;
          const float p3 = v3 ? weight(s_hi[1]) : 0.f;
          l = l * alpha + (p0 + p1 + p2 + p3);
          m = m_new;
          const uint32_t pa0 = pk2<T>(p0, p1), pa2 = pk2<T>(p2, p3);
#pragma unroll
          for (int i = 0; i < VD / 8; ++i) {
            o[i][0] *= alpha;
            o[i][1] *= alpha;
          }
          {
            const int tok = tokw + (mi & 1) * 8 + mr;
#pragma unroll
            for (int np = 0; np < VD / 16; ++np) {
              const int ch = np * 2 + (mi >> 1);
              const uint32_t addr = vbase + (ch >> 3) * kTcSlabBytes + tok * 128 + (((ch & 7) ^ (tok & 7)) << 4);
              uint32_t b0, b1, b2, b3;
              ldmatrix_x4_trans(addr, b0, b1, b2, b3);
              mma16816<T>(o[2 * np], pa0, 0u, pa2, 0u, b0, b1);
              mma16816<T>(o[2 * np + 1], pa0, 0u, pa2, 0u, b2, b3);
            }
          }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&empty_bar[stage]);
        if (++stage == kTcStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      // per-warp partials -> shared memory (rows < 8 only), then the 4 warps combine them
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      if (t4 == 0) {
        mrg_m[wg * 8 + g] = m;
        mrg_l[wg * 8 + g] = l;
      }
#pragma unroll
      for (int i = 0; i < VD / 8; ++i) {
        float2 v = make_float2(o[i][0], o[i][1]);
        *reinterpret_cast<float2*>(&mrg_o[(wg * 8 + g) * VD + i * 8 + 2 * t4]) = v;
      }
      meet();
      for (int e = tid; e < G * VD; e += 128) {
        const int gg = e / VD, d = e % VD;
        if (!PLAIN && d >= vdim) continue;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w) M = fmaxf(M, mrg_m[w * 8 + gg]);
        const int head = it.h * G + gg;
        const bool with_sink = p.sink != nullptr && it.part < 0;  // else the merge kernel adds it
        const float sink = with_sink ? to_f<T>(reinterpret_cast<const T*>(p.sink)[head]) * 1.4426950408889634f : -INFINITY;
        M = fmaxf(M, sink);
        float L = 0.f, O = 0.f;
        if (M > -INFINITY) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const float sc = exp2f(mrg_m[w * 8 + gg] - M);
            L += mrg_l[w * 8 + gg] * sc;
            O += mrg_o[(w * 8 + gg) * VD + d] * sc;
          }
        }
        if (with_sink) L += exp2f(sink - M);
        if (!PLAIN && p.sigmoid) L = 1.f;
        float val = L > 0.f ? O / L : 0.f;
        if (it.part < 0) {
          if (!PLAIN && p.gate != nullptr) val *= head_gate(reinterpret_cast<const T*>(p.gate) + it.b * p.gate_stride + head);
          T* op = reinterpret_cast<T*>(p.out) + static_cast<int64_t>(it.b) * p.out_stride +
                  static_cast<int64_t>(head) * vdim;
          if (std::is_same<T, __nv_bfloat16>::value)
            reinterpret_cast<__nv_bfloat16*>(op)[d] = __float2bfloat16(val);
          else
            reinterpret_cast<__half*>(op)[d] = __float2half(val);
        } else {
          const int64_t base = p.num_splits > 0 ? (static_cast<int64_t>(it.b) * p.q_heads + head) * p.num_splits + it.part
                                                : static_cast<int64_t>(it.part) * G + gg;
          p.part_o[base * vdim + d] = val;
          if (d == 0) p.part_lse[base] = L > 0.f ? M + log2f(L) : -INFINITY;
        }
      }
      if (p.num_splits == 0 && it.part >= 0) {  // an incomplete piece: whoever comes last to its item combines them all
        __threadfence();
        meet();
        const int chunks = before[p.batch], ranges = dec_ranges(p, chunks, walk.halves), start = before[it.b];
        const int c0 = dec_range_of(start, chunks, ranges), c1 = dec_range_of(before[it.b + 1] - 1, chunks, ranges);
        if (tid == 0) {
          unsigned* ticket = p.tickets + it.b * p.kv_heads + it.h;
          const bool last = atomicAdd(ticket, 1u) == static_cast<unsigned>(c1 - c0);
          if (last) *ticket = 0;  // ready for the next launch
          last_piece[half] = last;
        }
        meet();
        if (last_piece[half]) {
          __threadfence();
          for (int gg = wg; gg < G; gg += 4) dec_merge<T>(p, it.b, it.h, gg, start, c0, c1, chunks, ranges);
        }
      }
      meet();  // the merge area is reused by the next piece
      it = nit;
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        qa0[ks] = nqa0[ks];
        qa2[ks] = nqa2[ks];
      }
    }
  }
}

// Combine split partials: out = sum_s w_s o_s / (sum_s w_s + e^sink), w_s = 2^(lse_s - max lse).  A lane looks after the weight of
// every 32nd split, so that the loads of the partials do not wait for one another's weights (16 splits: 6.8 us behind the attention
// with a serial loop, 3.6 us so).  EARLY, at most eight splits: their partials are on their way while the weights are (8 splits: 4.2 -> 2.6 us;
// with more the values held back lengthen the loop, 16 splits of one row of 32 heads: 1 us, 40: 4 us).
template <typename T, bool EARLY>
__global__ void attn_merge_tc_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse,
                                     T* __restrict__ out, int64_t out_stride, int q_heads, int hd, int num_splits,
                                     const T* __restrict__ sink, const T* __restrict__ gate, int64_t gate_stride, int sum_only) {
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();
  const int b = blockIdx.x, head = blockIdx.y, lane = threadIdx.x & 31;
  const int64_t base = (static_cast<int64_t>(b) * q_heads + head) * num_splits;
  const float snk = sink ? to_f<T>(sink[head]) * 1.4426950408889634f : -INFINITY;
  const int d = threadIdx.x;  // (a block has a thread per column)
  constexpr int kEarly = 8;
  float early[kEarly], first = -INFINITY;
  float M = snk;
  if constexpr (EARLY) {
#pragma unroll
    for (int i = 0; i < kEarly; ++i) early[i] = i < num_splits && d < hd ? part_o[(base + i) * hd + d] : 0.f;
    if (lane < num_splits) first = part_lse[base + lane];
    M = fmaxf(M, first);
  } else {
    for (int s = lane; s < num_splits; s += 32) M = fmaxf(M, part_lse[base + s]);
  }
#pragma unroll
  for (int d = 16; d; d >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, d));
  const float g = gate ? head_gate(gate + b * gate_stride + head) : 1.f;
  float acc = 0.f, wsum = 0.f;
  if (M > -INFINITY) {
    if constexpr (EARLY) {
      const float mine = lane < num_splits ? exp2f(first - M) : 0.f;
#pragma unroll
      for (int i = 0; i < kEarly; ++i) {
        if (i >= num_splits) break;
        const float w = __shfl_sync(0xffffffffu, mine, i);
        wsum += w;
        if (d < hd) acc += w * early[i];
      }
    } else {
      for (int s0 = 0; s0 < num_splits; s0 += 32) {
        const float mine = s0 + lane < num_splits ? exp2f(part_lse[base + s0 + lane] - M) : 0.f;
        const int here = min(32, num_splits - s0);
#pragma unroll 8
        for (int i = 0; i < here; ++i) {
          const float w = __shfl_sync(0xffffffffu, mine, i);
          wsum += w;
          if (d < hd) acc += w * part_o[(base + s0 + i) * hd + d];
        }
      }
    }
    if (sink) wsum += exp2f(snk - M);
  }
  if (sum_only) wsum = 1.f;  // (every split's reference is zero: the weights are ones)
  if (d < hd) stf(out + static_cast<int64_t>(b) * out_stride + static_cast<int64_t>(head) * hd + d, wsum > 0.f ? acc / wsum * g : 0.f);
}

template <typename T, int HD, int VD, bool PLAIN>
static int launch_tc(const CUtensorMap (&tm)[4], const DecodeTcParams& p, int batch, cudaStream_t stream) {
  using Cfg = TcCfg<HD, VD>;
  auto kern = attn_decode_tc_kernel<T, HD, VD, PLAIN>;
  static PerDeviceOnce once;
  cudaError_t e = once.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes); });
  if (e != cudaSuccess) return (int)e;
  const int items = batch * p.kv_heads * p.num_splits;  // (few: one per SM)
  const int sms = device_sm_count();
  return (int)launch_pdl(kern, dim3(p.num_splits == 0 || items > sms ? sms : items), dim3(kTcThreads), Cfg::kSmemBytes, stream, tm[0],
                         tm[1], tm[2], tm[3], p);
}

template <typename T>
static int launch_tc(const CUtensorMap (&tm)[4], const DecodeTcParams& p, int batch, cudaStream_t stream) {
  const bool plain = p.dim == p.vdim && (p.dim == 64 || p.dim == 128) && p.v_rows > 0 && p.gate == nullptr && p.bias == nullptr && p.kv_div == 1 && !p.sigmoid;
  if (plain) return p.dim == 64 ? launch_tc<T, 64, 64, true>(tm, p, batch, stream) : launch_tc<T, 128, 128, true>(tm, p, batch, stream);
  if (p.dim > 64)
    return p.vdim > 64 ? launch_tc<T, 128, 128, false>(tm, p, batch, stream) : launch_tc<T, 128, 64, false>(tm, p, batch, stream);
  return p.vdim > 64 ? launch_tc<T, 64, 128, false>(tm, p, batch, stream) : launch_tc<T, 64, 64, false>(tm, p, batch, stream);
}

}  // namespace blitz

extern "C" {
using namespace blitz;

// Bytes of scratch: part_o and part_lse in fp32; num_splits = 0: the same for any batch it takes, and before them a ticket per
// sequence and head, which have to be zero before the first call (the kernel leaves them zero).
constexpr int64_t kTcTickets = (int64_t)kTcMaxShared * kTcMaxSharedHeads;
int64_t blitz_attn_decode_workspace_bytes(int batch, int q_heads, int head_dim, int num_splits) {
  if (num_splits == 0)
    return ((int64_t)device_sm_count() * kTcHalves * 2 * 8 * (head_dim + 1) + kTcTickets) * (int64_t)sizeof(float);
  if (num_splits < 0 || num_splits == 1) return 0;
  return (int64_t)batch * q_heads * num_splits * (head_dim + 1) * (int64_t)sizeof(float);
}

// k_pool, v_pool: [max_pages][page_rows][kv_heads][dim or vdim], a page's tokens in its first page_size rows (one tensor for
// keys and values: page_rows = 2 page_size, v_pool at the first value plane).  workspace: scratch of
// blitz_attn_decode_workspace_bytes() bytes for value heads of vdim (may be null when num_splits == 1).  num_splits: 0 = equal
// shares of all chunks (whole items beyond 256 sequences or 128 heads), n = every (sequence, KV head) in n parts.
// page_size must be a power of two >= 8 (pages smaller than 64 tokens are fetched as several boxes per stage).  dim and
// vdim: multiples of 8 up to 128.  window (0 = none) / keep_first, softcap (0 = none), sink and gate (null = none) as
// described at the top of the file.  bias: [q_heads][bias_len] in the activation type, or null.  static_table != 0 promises that
// indices, indptr and last_page_len are not written by kernels still running in this stream: they are read before those finish.
int blitz_attn_decode(const void* q, int64_t q_stride, const void* k_pool, const void* v_pool, const int32_t* indices,
                      const int32_t* indptr, const int32_t* last_page_len, void* out, int64_t out_stride,
                      void* workspace, int batch, int q_heads, int kv_heads, int dim, int vdim, int page_size, int page_rows,
                      int max_pages, int num_splits, float sm_scale, int window, int keep_first, int chunked, int sigmoid, float softcap,
                      const void* sink, const void* bias, int bias_len, const void* gate, int64_t gate_stride, int static_table, int* status, int dtype,
                      cudaStream_t stream) {
  if (batch <= 0) return 0;
  if (window < 0 || keep_first < 0 || softcap < 0.f || (bias != nullptr && bias_len < 1)) return -1;
  if ((chunked && (window < 1 || keep_first)) || (sigmoid && (sink || softcap > 0.f))) return -1;
  if (num_splits < 0 || kv_heads < 1 || (q_heads % kv_heads) != 0 || (q_stride & 1)) return -1;
  if (dim < 8 || dim > 128 || (dim & 7) || vdim < 8 || vdim > 128 || (vdim & 7)) return -1;
  if (page_size < 8 || (page_size & (page_size - 1)) != 0 || page_rows < page_size) return -1;
  if (num_splits != 1 && workspace == nullptr) return -1;
  const int group = q_heads / kv_heads;
  int div = (group + 7) / 8;
  while (group % div) ++div;
  if (num_splits == 0 && (batch > kTcMaxShared || kv_heads * div > kTcMaxSharedHeads)) num_splits = 1;
  const int bt = page_size < kTcChunk ? page_size : kTcChunk;
  const int bt_tail = bt < 16 ? bt : 16;
  const bool one = dim == vdim && page_rows == 2 * page_size &&
                   v_pool == reinterpret_cast<const char*>(k_pool) + (int64_t)page_size * kv_heads * dim * 2;
  if (one) v_pool = k_pool;
  // rows of a pool: those of the last page end with its tokens
  const uint64_t rows = one ? (uint64_t)max_pages * page_rows : (uint64_t)(max_pages - 1) * page_rows + page_size;
  CUtensorMap tm[4];
  for (int i = 0; i < 4; ++i) {
    const uint64_t d = i < 2 ? dim : vdim;
    if (!get_tmap_3d(&tm[i], i < 2 ? k_pool : v_pool, d, (uint64_t)kv_heads, rows, d * 2, d * 2 * kv_heads, 64, 1,
                     (uint32_t)(i & 1 ? bt_tail : bt)))
      return -2;
  }
  DecodeTcParams p;
  p.q = q; p.q_stride = q_stride; p.indices = indices; p.indptr = indptr; p.last_page_len = last_page_len;
  p.out = out; p.out_stride = out_stride;
  p.tickets = num_splits == 0 ? reinterpret_cast<unsigned*>(workspace) : nullptr;
  p.part_o = reinterpret_cast<float*>(workspace) + (num_splits == 0 ? kTcTickets : 0);
  const int64_t parts = num_splits == 0 ? (int64_t)device_sm_count() * kTcHalves * 2 * (group / div) : (int64_t)batch * q_heads * num_splits;
  p.part_lse = workspace ? p.part_o + parts * vdim : nullptr;
  p.batch = batch; p.q_heads = q_heads; p.kv_heads = kv_heads * div; p.kv_div = div; p.group = group / div;
  p.page_size = page_size; p.max_pages = max_pages; p.dim = dim; p.vdim = vdim; p.page_rows = page_rows; p.v_rows = one ? page_size : 0;
  p.num_splits = num_splits; p.box_tokens = bt; p.tail_box_tokens = bt_tail;
  p.scale_log2 = sm_scale * 1.4426950408889634f; p.status = status;
  p.chunked = chunked; p.sigmoid = sigmoid; p.static_table = static_table;
  p.window = window; p.keep_first = keep_first; p.sink = sink; p.bias = bias; p.bias_len = bias_len; p.gate = gate; p.gate_stride = gate_stride;
  p.cap_scale = softcap > 0.f ? sm_scale / softcap : 0.f; p.cap_log2 = softcap * 1.4426950408889634f;
  int rc = dtype == 1 ? launch_tc<__nv_bfloat16>(tm, p, batch, stream) : launch_tc<__half>(tm, p, batch, stream);
  if (rc != 0) return rc;
  if (num_splits > 1) {
    auto merge = [&](auto type) {
      using T = decltype(type);
      return (int)launch_pdl(p.num_splits <= 8 ? attn_merge_tc_kernel<T, true> : attn_merge_tc_kernel<T, false>, dim3(batch, q_heads), dim3(vdim > 64 ? 128 : 64), 0, stream, p.part_o, p.part_lse,
                             (T*)out, out_stride, q_heads, vdim, num_splits, (const T*)sink, (const T*)gate, gate_stride, sigmoid);
    };
    rc = dtype == 1 ? merge(__nv_bfloat16{}) : merge(__half{});
  }
  return rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// Allocation-free variant (declared and documented in attn_decode_noalloc.h).  The split-KV partials go to
// an array that is part of the library image instead of a caller-provided workspace.
#include "attn_decode_noalloc.h"

namespace blitz {

// Device global memory, present on every GPU that loads the library.  In host code this name is only a
// handle for the runtime: its device address is looked up once per device below and that address, not the
// name, is what the kernels receive.
static __device__ __align__(256) unsigned char g_noalloc_scratch[BLITZ_ATTN_NOALLOC_SCRATCH_BYTES];

constexpr int kNoallocMaxDevices = kMaxDevicesPerProcess;
// Device address of the scratch on each device: written once under the set-up lock and published with release
// order, so a host thread that sees a non-null value also sees a fully set-up device.
static std::atomic<void*> g_noalloc_ptr[kNoallocMaxDevices];
static PerDeviceOnce g_noalloc_once;

// Per-device set-up with that device current: resolve the scratch address, raise the shared-memory limits.
static cudaError_t noalloc_setup(int dev) {
  void* ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  if (ptr == nullptr) return cudaErrorInvalidSymbol;
  e = cudaFuncSetAttribute(attn_decode_tc_kernel<__nv_bfloat16, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<128>::kSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(attn_decode_tc_kernel<__nv_bfloat16, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<64>::kSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(attn_decode_tc_kernel<__half, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<128>::kSmemBytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(attn_decode_tc_kernel<__half, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<64>::kSmemBytes);
  if (e != cudaSuccess) return e;
  g_noalloc_ptr[dev].store(ptr, std::memory_order_release);
  return cudaSuccess;
}

// Tensor map of one KV layer built on the stack (the cached builder keeps a host-side table; this path keeps nothing).
static bool noalloc_tmap(CUtensorMap* out, const void* kv_layer, int head_dim, int kv_heads, int max_pages, int page_size,
                         int box_tokens) {
  PFN_encodeTiled enc = get_encode_fn();
  if (!enc || (reinterpret_cast<uintptr_t>(kv_layer) & 15) != 0) return false;
  cuuint64_t dims[3] = {(cuuint64_t)head_dim, (cuuint64_t)kv_heads, (cuuint64_t)max_pages * 2 * page_size};
  cuuint64_t strides[2] = {(cuuint64_t)head_dim * 2, (cuuint64_t)kv_heads * head_dim * 2};
  cuuint32_t box[3] = {64, 1, (cuuint32_t)box_tokens};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(kv_layer), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T, int HD>
static int noalloc_launch(const CUtensorMap (&tm)[4], const DecodeTcParams& p, int sms, cudaStream_t stream) {
  const int items = p.batch * p.kv_heads * p.num_splits;
  attn_decode_tc_kernel<T, HD><<<items < sms ? items : sms, kTcThreads, TcCfg<HD>::kSmemBytes, stream>>>(tm[0], tm[1], tm[2], tm[3], p);
  return (int)cudaGetLastError();
}

}  // namespace blitz

extern "C" int blitz_attn_decode_noalloc(const void* q, int64_t q_stride, const void* kv_layer, const int32_t* indices,
                                         const int32_t* indptr, const int32_t* last_page_len, void* out,
                                         int64_t out_stride, int batch, int q_heads, int kv_heads, int head_dim,
                                         int page_size, int max_pages, int num_splits, float sm_scale, int* status,
                                         int dtype, cudaStream_t stream) {
  using namespace blitz;
  if (batch <= 0) return 0;
  if (num_splits < 1 || kv_heads <= 0 || (q_heads % kv_heads) != 0 || (q_stride & 1) || (out_stride & 1)) return -1;
  const int G = q_heads / kv_heads;
  if (G > 8 || (head_dim != 64 && head_dim != 128)) return -1;
  if (page_size < 8 || (page_size & (page_size - 1)) != 0) return -1;
  const int64_t need = num_splits > 1 ? (int64_t)batch * q_heads * num_splits * (head_dim + 1) * (int64_t)sizeof(float) : 0;
  if (need > (int64_t)BLITZ_ATTN_NOALLOC_SCRATCH_BYTES) return BLITZ_ATTN_NOALLOC_TOO_LARGE;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kNoallocMaxDevices) return -1;
  e = g_noalloc_once.run([&] { return noalloc_setup(dev); });
  if (e != cudaSuccess) return (int)e;
  void* const scratch = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) return (int)cudaErrorInvalidSymbol;
  const int bt = page_size < kTcChunk ? page_size : kTcChunk;
  const int bt_tail = bt < 16 ? bt : 16;
  CUtensorMap tm[4];
  for (int i = 0; i < 4; ++i)
    if (!noalloc_tmap(&tm[i], kv_layer, head_dim, kv_heads, max_pages, page_size, i & 1 ? bt_tail : bt)) return -2;
  DecodeTcParams p;
  p.q = q; p.q_stride = q_stride; p.indices = indices; p.indptr = indptr; p.last_page_len = last_page_len;
  p.out = out; p.out_stride = out_stride;
  p.part_o = reinterpret_cast<float*>(scratch);
  p.part_lse = p.part_o + (int64_t)batch * q_heads * num_splits * head_dim;
  p.batch = batch; p.q_heads = q_heads; p.kv_heads = kv_heads; p.group = G; p.page_size = page_size;
  p.max_pages = max_pages; p.num_splits = num_splits; p.box_tokens = bt; p.tail_box_tokens = bt_tail;
  p.scale_log2 = sm_scale * 1.4426950408889634f; p.status = status; p.tickets = nullptr;
  p.kv_div = 1; p.dim = p.vdim = head_dim; p.page_rows = 2 * page_size; p.v_rows = page_size; p.gate = nullptr; p.gate_stride = 0;
  p.chunked = p.sigmoid = p.static_table = 0;
  p.window = 0; p.keep_first = 0; p.sink = nullptr; p.bias = nullptr; p.bias_len = 0; p.cap_scale = p.cap_log2 = 0.f;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  int rc;
  if (dtype == 1)
    rc = head_dim == 128 ? noalloc_launch<__nv_bfloat16, 128>(tm, p, sms, stream)
                         : noalloc_launch<__nv_bfloat16, 64>(tm, p, sms, stream);
  else
    rc = head_dim == 128 ? noalloc_launch<__half, 128>(tm, p, sms, stream)
                         : noalloc_launch<__half, 64>(tm, p, sms, stream);
  if (rc != 0 || num_splits == 1) return rc;
  dim3 grid(batch, q_heads);
  if (dtype == 1)
    attn_merge_tc_kernel<__nv_bfloat16, false><<<grid, head_dim, 0, stream>>>(p.part_o, p.part_lse, (__nv_bfloat16*)out, out_stride,
                                                                       q_heads, head_dim, num_splits, nullptr, nullptr, 0, 0);
  else
    attn_merge_tc_kernel<__half, false><<<grid, head_dim, 0, stream>>>(p.part_o, p.part_lse, (__half*)out, out_stride, q_heads,
                                                                head_dim, num_splits, nullptr, nullptr, 0, 0);
  return (int)cudaGetLastError();
}
