// Shared declarations of the MoBA forward kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernel_setup.cuh"
#include "moba_b200.h"

namespace moba {

constexpr int kMeanLanes = 32;           // row accumulators of a chunk mean
constexpr int kMaxTopk = 64;             // parallel.py:436

// Launch-time view of a problem, passed to kernels by value.
struct Params {
  int64_t T;                             // tokens of k / v (and of cu_seqlens)
  int64_t Tq;                            // query tokens: the window [win_lo, win_lo + Tq) of the packed tokens
  int win_lo;                            // q, out, selected and the partials are indexed by token - win_lo
  int B, Hq, Hkv, G, D;
  int max_seqlen, C, topk;
  int mc, slots, hist, NP;               // NP = partial results per row
  int64_t rows, lists;
  int fp16;                              // element type of q, k, v, out: 0 bf16, 1 fp16
  int64_t sel_rs;                        // elements between two ranks of `selected` (heads of the full tensor * Tq)
  int64_t sq_t, sq_h, sk_t, sk_h, sv_t, sv_h, so_t, so_h;
};

__host__ inline int cdiv_i(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Token tiles of `tile` tokens per sequence that the gating and scatter grids enumerate: those
// of max_seqlen when every token is a query; with a query window only as many as Tq tokens can
// overlap (one more than they fill), counted from window_tile0 of the sequence, so that a
// decode step on a long prefix does not walk over the tiles of the whole prefix.
__host__ __device__ inline int window_tiles(const Params& p, int tile) {
  const int64_t all = ((int64_t)p.max_seqlen + tile - 1) / tile;
  if (p.Tq == p.T) return (int)all;
  const int64_t w = (p.Tq + tile - 1) / tile + 1;
  return (int)(w < all ? w : all);
}
// First tile of the sequence starting at packed token s0 that can hold a token of the window.
__device__ __forceinline__ int window_tile0(const Params& p, int s0, int tile) {
  return (p.Tq == p.T || p.win_lo <= s0) ? 0 : (p.win_lo - s0) / tile;
}

__device__ __forceinline__ float bf16_lo(uint32_t x) { return __uint_as_float(x << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t x) { return __uint_as_float(x & 0xffff0000u); }

// 16-bit element helpers; kHalf selects fp16, otherwise bf16.  Tensors are passed as
// __nv_bfloat16* whatever their element type: only these helpers interpret the bits.
template <bool kHalf>
__device__ __forceinline__ float2 unpack2(uint32_t x) {
  if (kHalf) return __half22float2(*reinterpret_cast<const __half2*>(&x));
  return make_float2(bf16_lo(x), bf16_hi(x));
}
template <bool kHalf>
__device__ __forceinline__ uint32_t pack2_16(float lo, float hi) {       // round to nearest even
  if (kHalf) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <bool kHalf>
__device__ __forceinline__ void unpack8(const uint4 x, float (&f)[8]) {
  const float2 a = unpack2<kHalf>(x.x), b = unpack2<kHalf>(x.y), c = unpack2<kHalf>(x.z), d = unpack2<kHalf>(x.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}

// Partial results of the dense stage (one per row and attended chunk; the reference keeps them
// in the input dtype, attention.py:727).  The normalised O row is stored as fp16 scaled by a
// power of two chosen per row, so that its largest magnitude lands in [2^13, 2^14): 11
// significant bits on every element whatever the range of V, no overflow.  partial_lse holds
// two floats per entry: the natural-log LSE (-inf: the entry contributes nothing) and 1 / scale.
struct PartialScale { float scale, inv; };
__device__ __forceinline__ PartialScale partial_scale(float amax) {
  // floor(log2 amax) from the exponent field: -127 for zero and subnormals, 128 for inf / NaN
  int s = 13 - ((int)((__float_as_uint(amax) >> 23) & 0xFF) - 127);
  s = s < -100 ? -100 : (s > 100 ? 100 : s);
  PartialScale r;
  r.scale = __uint_as_float((uint32_t)(127 + s) << 23);
  r.inv = __uint_as_float((uint32_t)(127 - s) << 23);
  return r;
}
__device__ __forceinline__ uint32_t pack2_half(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Chunk slot geometry (routing.py:565-579).
struct Slot {
  int start, end;        // token range [start, end)
  bool historical;       // may be selected by later queries
};
__device__ __forceinline__ Slot slot_of(const int32_t* __restrict__ cu, int b, int j, int C) {
  const int s0 = cu[b], s1 = cu[b + 1];
  Slot s;
  const long long st = (long long)s0 + (long long)j * C;
  s.start = st < s1 ? (int)st : s1;
  const long long en = (long long)s.start + C;
  s.end = en < s1 ? (int)en : s1;
  s.historical = s.end < s1;
  return s;
}

// Work item of the dense stage.
struct Item {
  int valid;             // 0: nothing to do
  int causal;            // 1: own chunk, rows are consecutive tokens of one head
  int nrows;             // rows in this item (<= tile rows)
  int row_start;         // routed: first index into row_list; own: first row inside the query window
  int tok0;              // own: first query token
  int head;              // own: query head
  int kv_head;
  int kv_tok0;           // first key token
  int kv_len;            // keys to visit
};

// Slots that can hold tokens of the query window: [lo, lo + n).  All slots when every token
// is a query; otherwise from the slot of the window's first token to that of its last one
// (packed tokens rise with the slot index), so that a short window - a decode step is one
// token - does not enumerate the own-chunk tiles of the whole batch.
struct SlotRange { int lo, n; };
__device__ __forceinline__ SlotRange own_slot_range(const Params& p, const int32_t* __restrict__ cu) {
  SlotRange sr;
  sr.lo = 0;
  sr.n = (int)p.slots;
  if (p.Tq == p.T) return sr;
  int at[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int tok = e == 0 ? p.win_lo : p.win_lo + (int)p.Tq - 1;
    int l = 0, r = p.B;                       // last sequence with cu[b] <= tok
    while (r - l > 1) {
      const int mid = (l + r) >> 1;
      if (__ldg(cu + mid) <= tok) l = mid; else r = mid;
    }
    at[e] = l * p.mc + (tok - __ldg(cu + l)) / p.C;
  }
  sr.lo = at[0];
  sr.n = at[1] - at[0] + 1;
  return sr;
}

// Decode work item `i`.  Routed items come first (list-major, tiles of
// `tile_rows` rows), own-chunk items follow with the longest tiles first, over the
// slots [own.lo, own.lo + own.n) (own.n < 0: all slots).
// `list_hint` >= 0: the list of a routed item, found by the caller (the last l with
// tile_prefix[l] <= i); otherwise it is searched for in tile_prefix.
__device__ __forceinline__ Item decode_item(const Params& p, int i, int n_routed, int tile_rows,
                                            const int32_t* __restrict__ cu,
                                            const int32_t* __restrict__ list_counts,
                                            const int32_t* __restrict__ list_offsets,
                                            const int32_t* __restrict__ tile_prefix, int list_hint = -1,
                                            SlotRange own = SlotRange{0, -1}) {
  Item it;
  it.valid = 0;
  if (i < n_routed) {
    int l = list_hint;
    if (l < 0) {
      int lo = 0, hi = (int)p.lists;         // last l with tile_prefix[l] <= i
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (tile_prefix[mid] <= i) lo = mid; else hi = mid;
      }
      l = lo;
    }
    const int tile = i - tile_prefix[l];
    const int slot = l / p.Hkv;
    const int b = slot / p.mc, j = slot - b * p.mc;
    it.valid = 1;
    it.causal = 0;
    it.row_start = list_offsets[l] + tile * tile_rows;
    const int left = list_counts[l] - tile * tile_rows;
    it.nrows = left < tile_rows ? left : tile_rows;
    it.kv_head = l - slot * p.Hkv;
    it.kv_tok0 = cu[b] + j * p.C;
    it.kv_len = p.C;
    it.tok0 = 0;
    it.head = 0;
    return it;
  }
  const int tiles_per_chunk = (p.C + tile_rows - 1) / tile_rows;
  const int per_tile = (own.n < 0 ? (int)p.slots : own.n) * p.Hq;
  int idx = i - n_routed;
  const int ti = tiles_per_chunk - 1 - idx / per_tile;
  idx -= (idx / per_tile) * per_tile;
  const int slot = own.lo + idx / p.Hq;
  const int h = idx - (slot - own.lo) * p.Hq;
  const int b = slot / p.mc, j = slot - b * p.mc;
  const Slot s = slot_of(cu, b, j, p.C);
  const int tok0 = s.start + ti * tile_rows;
  if (ti < 0) return it;
  // the tile keeps its place in the chunk; of its rows, those inside the query window
  // [first, nrows) are computed (a window may start and end anywhere)
  const int win_hi = p.win_lo + (int)p.Tq;
  const int tok_end = s.end < win_hi ? s.end : win_hi;
  const int first = p.win_lo > tok0 ? p.win_lo - tok0 : 0;
  const int nrows = tok_end - tok0 < tile_rows ? tok_end - tok0 : tile_rows;
  if (first >= nrows) return it;
  it.valid = 1;
  it.causal = 1;
  it.tok0 = tok0;
  it.nrows = nrows;
  it.head = h;
  it.kv_head = h / p.G;
  it.kv_tok0 = s.start;
  it.kv_len = tok0 + nrows - s.start;
  it.row_start = first;
  return it;
}

__host__ __device__ inline int own_item_count(int slots, int Hq, int C, int tile_rows) {
  return slots * Hq * ((C + tile_rows - 1) / tile_rows);
}

// ---- programmatic dependent launch -------------------------------------------
// The kernels of a call follow one another on one stream and each is often only a few microseconds
// long.  Launched with launch_pdl a kernel may become resident while the one before it drains: it
// sets up (barriers, tensor memory, descriptors), then pdl_wait() holds it until the grid before it has
// completed and its writes are visible.  Every kernel so launched calls pdl_wait() in all of its threads before its
// first access to global memory, and pdl_trigger() behind it (the merge: not always), so that at most the next
// kernel of the stream is resident early.  Both are no-ops in a kernel launched the ordinary way.
// Measured (B200, events around back-to-back calls), together with the clear of the counters moved into the
// chunk-mean kernel and the prefix sums into the tail of the gating kernel (seven stream operations
// become five): one decode token on a 131072-token prefix 224 -> 194 us, 700 tokens behind 50021 245 -> 237 us.
//
// A kernel that is resident early is placed where the one before it has left room, not evenly, and runs with the
// split of L1 and shared memory that it finds.  A few microseconds of launch are not worth that where it runs long:
//   - the merge triggers nothing in a call that averages more than kTriggerMeanBytes of K: what follows it is
//     likely a call of the same kind, whose chunk means are few long CTAs (268 MB of K in chunks of 4096, head_dim 64, 700
//     new tokens, back to back: 375 us with the trigger, 339 without, 369 with no kernel chained; one decode token
//     behind 20011, appended back to back: 37.9 with it, 38.6 without);
//   - the merge itself is not chained from kChainedMergeBytes of partial rows on (131072 tokens x 16, head_dim 64,
//     chunk 64, 2.1 GB: 6.83 -> 6.62 ms; 32768 x 32/8, chunk 1024, 1.1 GB 3.98 -> 3.85; 32768 x 32/8, head_dim 128,
//     chunk 128, 2.1 GB 2.27 -> 2.22; 13311 x 16, 0.22 GB 332 -> 329 us; a decode step's 16 KB: 161 -> 163);
//   - the gating kernel is not chained behind the means of more (slot, kv head) pairs than have a CTA resident at a time with
//     one CTA a pair (130859 tokens, chunk 128, 16 heads, 700 new tokens: 434 -> 413 us; few chunks: 1 to 3 us slower).  At head
//     dim 256 a pair has four CTAs, and chaining is the better way up to there too: 96 pairs 81.2 -> 78.0 us, 384 186 -> 184, 648
//     84.9 -> 81.2, 1024 449 -> 445.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
constexpr int64_t kTriggerMeanBytes = 8 << 20;
constexpr int64_t kChainedMergeBytes = 64 << 20;
constexpr int64_t kChainedMeanPairs = 148 * 8;
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(bool chained, void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                                  const Args&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, const Args&... args) {
  return launch_chained(true, kernel, grid, threads, smem, st, args...);
}

// Exclusive prefix sums over the lists, by one block of kThreads threads, kPer lists a thread and
// round: offsets of the lists in row_list, of their tiles in the item order; cursors are cleared.
struct ListScan {
  const int32_t* counts;
  int32_t* offsets;
  int32_t* tile_prefix;
  int32_t* cursors;
  int64_t lists;
  int32_t tile_rows;
};
// `scratch`: 2 * kThreads / 32 ints of shared memory.
template <int kThreads, int kPer>
__device__ __forceinline__ void scan_lists(const ListScan& a, int* scratch) {
  constexpr int kWarps = kThreads / 32;
  int* warp_rows = scratch;
  int* warp_tiles = scratch + kWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int carry_rows = 0, carry_tiles = 0;
  for (int64_t base = 0; base < a.lists; base += kThreads * kPer) {
    const int64_t l0 = base + (int64_t)threadIdx.x * kPer;
    int n[kPer], rows = 0, tiles = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      n[u] = l0 + u < a.lists ? __ldcg(a.counts + l0 + u) : 0;
      rows += n[u];
      tiles += (n[u] + a.tile_rows - 1) / a.tile_rows;
    }
    int xr = rows, xt = tiles;                                  // inclusive over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int yr = __shfl_up_sync(0xffffffffu, xr, o);
      const int yt = __shfl_up_sync(0xffffffffu, xt, o);
      if (lane >= o) { xr += yr; xt += yt; }
    }
    if (lane == 31) { warp_rows[warp] = xr; warp_tiles[warp] = xt; }
    __syncthreads();
    int pre_r = carry_rows + xr - rows, pre_t = carry_tiles + xt - tiles;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) { pre_r += warp_rows[w]; pre_t += warp_tiles[w]; }
      carry_rows += warp_rows[w];
      carry_tiles += warp_tiles[w];
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (l0 + u < a.lists) { a.offsets[l0 + u] = pre_r; a.tile_prefix[l0 + u] = pre_t; a.cursors[l0 + u] = 0; }
      pre_r += n[u];
      pre_t += (n[u] + a.tile_rows - 1) / a.tile_rows;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { a.offsets[a.lists] = carry_rows; a.tile_prefix[a.lists] = carry_tiles; }
}

// ---- launchers implemented in the kernel files -----------------------------
cudaError_t launch_chunk_metadata(const Params& p, const int32_t* cu, int32_t* cu_chunk,
                                  int32_t* chunk_end, int8_t* valid, cudaStream_t st);
// K and V rows of the query window into the caches (strides of `p`), and cu_seqlens = {0, T}
cudaError_t launch_append_rows(const Params& p, const __nv_bfloat16* k_new, const __nv_bfloat16* v_new, int64_t kn_t,
                               int64_t kn_h, int64_t vn_t, int64_t vn_h, __nv_bfloat16* k, __nv_bfloat16* v,
                               int32_t* cu, cudaStream_t st);
cudaError_t launch_chunk_means(const Params& p, const __nv_bfloat16* k, const int32_t* cu,
                               __nv_bfloat16* means, cudaStream_t st);
cudaError_t launch_chunk_means_range(const Params& p, int slot_begin, int slot_end, const __nv_bfloat16* k,
                                     const int32_t* cu, __nv_bfloat16* means, cudaStream_t st,
                                     int32_t* zero = nullptr, int64_t zero_words = 0);
// Up to this many lists the gating kernel's last CTA computes the prefix sums over them, which saves a launch; the
// kernel that does it otherwise takes more lists at a time and leaves the gating CTAs without the ticket.  Whole
// call, fused / apart: 4 lists 30.3 / 31.2 us, 20 48.1 / 48.8, 128 48.1 / 48.1, 256 107.9 / 105.2 and 198.5 / 189.6,
// 392 180 / 175, 2048 278.7 / 273.6, 30000 2792 / 2775 (gating alone 90 us longer, scatter 60 shorter).  Calls of few
// rows are as long as the host takes to issue them, and there a launch counts for more: one decode token, 160
// lists, 35.0 / 35.0 us with the host ahead, 38.9 / 40.4 through an append; 256 lists 121.5 / 120.4 with the host ahead.
inline bool gate_scans_lists(const Params& p) { return p.lists <= (p.rows <= 4096 ? 256 : 128); }
// with `scan`, the last CTA to finish also computes the prefix sums over the lists (`ticket`: a counter at zero)
cudaError_t launch_gate_topk(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* means,
                             const int32_t* cu, int32_t* selected, int32_t* list_counts,
                             cudaStream_t st, const ListScan* scan = nullptr, int32_t* ticket = nullptr, bool chained = true);
// The same with optional statistics (int32[4], added to: [0] rows whose near-ties were ranked
// again in the contract order, [1] largest |estimate - contract score| / eps seen there in
// units of 2^-16, [2] rows where that ratio exceeded 1, [3] rows ranked over all candidates)
// and flags (1: rank every row over all candidates, 2: rank the kept candidates of every row again).
cudaError_t launch_gate_topk_stats(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* means,
                                   const int32_t* cu, int32_t* selected, int32_t* list_counts, int32_t* stats,
                                   int flags, cudaStream_t st, const ListScan* scan = nullptr,
                                   int32_t* ticket = nullptr, bool chained = true);
// false when the shared memory the gating kernel needs for `p` exceeds what an SM offers
bool gate_topk_fits(const Params& p);
cudaError_t launch_compact(const Params& p, const int32_t* cu, const int32_t* selected,
                           const int32_t* list_counts, int32_t* list_offsets, int32_t* tile_prefix,
                           int32_t* cursors, int32_t* row_list, float2* partial_lse, int tile_rows,
                           cudaStream_t st);
// the second half of launch_compact, behind prefix sums computed elsewhere
cudaError_t launch_scatter(const Params& p, const int32_t* cu, const int32_t* selected, const int32_t* list_offsets,
                           int32_t* cursors, int32_t* row_list, float2* partial_lse, cudaStream_t st);
cudaError_t launch_merge(const Params& p, const __half* partial_out, const float2* partial_lse,
                         const int32_t* status, __nv_bfloat16* out, float* lse_out, cudaStream_t st, bool trigger = false);

constexpr int kMmaTileRows = 128;        // rows per work item, mma.sync kernel
constexpr int kTc5TileRows = 256;        // rows per work item, tcgen05 kernel (two 128-row MMA tiles)
constexpr int kTileRowsWide = 128;       // rows per work item, tcgen05 kernel at head_dim 256 (one tile)
// Row tiles of a list are 128 rows for chunks of at most this many keys (and at head dim 256), 256 otherwise.
#ifndef MOBA_SMALL_CHUNK
#define MOBA_SMALL_CHUNK 256
#endif
constexpr int kSmallChunk = MOBA_SMALL_CHUNK;
__host__ __device__ inline bool tc5_small_tiles(int head_dim, int chunk) { return head_dim <= 128 && chunk <= kSmallChunk; }
// Chunks of at most this many keys run the tcgen05 kernel for short items (one 128-row tile per item, two CTAs per
// SM; where the lists are cut into 256 rows it takes a half at a time), and so do query windows whose rows of
// one kv head fit one tile (decode steps): a second row tile would be empty.  Measured against the 256-row kernel,
// whole call: chunk 512, 32768 tokens x 32/8 heads, top-k 8 3.61 -> 3.27 ms (head_dim 64 2.85 -> 2.42), 2 x 4096 x 16
// 340 -> 308 us, 19456 x 32 983 -> 888 us; small launches gain too (700 to 20000 tokens, 1 to 16 heads, chunks 300 and
// 512: dense stage 0.69 to 1.00 of the other's).  Windows: 1 to 128 rows per kv head, 9000 to 131072 tokens, 1 to 16 kv
// heads, chunks 1024 to 4096: 0.49 to 1.03 of the other's dense stage, with no more CTAs than items (window_ctas).
// Up to 1024 keys the halves of a 256-row tile still read K and V twice as often for less than the second CTA per SM
// gives, whole call: 700 tokens behind 50021, 32/8 heads 197 -> 183 us, 64 behind them 120 -> 93, 1500 behind 20000
// at head_dim 64 153 -> 148; 12001 x 16/2 753 -> 713; 5000 + 3000 x 8/1 164 -> 156; 32768 x 16 at 64 1977 -> 1805, 20000 x 16/4 at
// 96 1323 -> 1222.  Long calls are another matter: back to back they run at the power limit, where the tensor work counts and
// the tiles read twice cost more than the second CTA gives.  By partial rows, calls back to back for a second, chunk 1024:
//   head_dim 128  1.9 M (19456 x 32) 1018 -> 998 us, 2.1 M (16384 x 16) 1112 -> 1116, 3.1 M (32768 x 32, top-k 3) 2203 -> 2236, 3.8 M
//                 (20000 x 32, chunk 900) 2467 -> 2538, 4.2 M (16384 x 32/8) 2183 -> 2244, 8.4 M (32768 x 32/8) 4.63 -> 4.72 ms
//   head_dim 96   4.2 M (32768 x 16) 2362 -> 2335, 8.4 M (65536 x 32/8, top-k 4) 5.10 -> 5.20 ms, 16.8 M 9.85 -> 9.97
//   head_dim 64   16.8 M (65536 x 32) 8.31 -> 7.99 ms
// With fewer key tiles an item longer calls gain: head_dim 128, 3.8 M, chunk 640 (30000 x 16/2) 1848 -> 1768 us, 4.2 M, chunk 768
// (16384 x 32/4) 1962 -> 1963; head_dim 96, 16.8 M, chunk 700 8.63 -> 8.61 ms.  At 2048 and 4096 keys all but a few lose
// (20000 x 8/4 759 -> 826).
constexpr int kShortChunk = 512, kShortChunkMid = 768, kShortChunkFew = 1024;
constexpr int64_t kShortFewRows = (int64_t)2 << 20, kShortMidRows = (int64_t)4 << 20;
static_assert(kSmallChunk <= kShortChunk, "lists cut into 128 rows run the kernel of one-tile items");
inline bool tc5_short_items(const Params& p) {
  if (p.D > 128) return false;
  if (p.Tq * p.G <= kTileRowsWide) return true;
  // (own-chunk items are counted in int32; a slot table that large stays with the 256-row kernel)
  const bool mid = p.C <= kShortChunkMid;
  const int64_t most = p.D == 64 || (mid && p.D == 96) ? INT64_MAX : mid || p.D == 96 ? kShortMidRows : kShortFewRows;
  const bool few = p.C <= kShortChunkFew && p.rows * p.NP <= most;
  return (p.C <= kShortChunk || few) && (int64_t)p.slots * p.Hq * ((p.C + 127) / 128) < ((int64_t)1 << 30);
}

// Chunks of 96 to 128 keys, one key tile an item, run a kernel that keeps several items of an SM in flight, where the lists are a few tiles
// long: a list or an own-chunk tile of its own costs the warp that describes them and new K and V, and half-filled tiles (chunks of
// 64 keys have half of their items that way) cost it as much as full ones.  Dense stage, kernel for short items over this one,
// 20000 tokens x 16 heads, top-k 2 / 4 / 8, by kv heads:
//   head dim 128  chunk 128  1: 1.21 / 1.14 / 1.09   4: 1.18 / 1.12 / 1.06   16: 0.83 / 1.01 / 1.07
//                 chunk 96   1: 1.03 / 1.13 / 1.13   4: 1.05 / 1.09 / 1.12   16: 0.72 / 0.99 / 1.05
//                 chunk 64   1: 0.73 / 0.85 / 0.99   4: 0.68 / 0.85 / 0.97   16: 0.55 / 0.70 / 0.90
//   head dim 64   chunk 128  1: 1.19 / 1.17 / 1.22   4: 1.23 / 1.19 / 1.23   16: 1.02 / 1.22 / 1.27
//                 chunk 96   1: 1.13 / 1.15 / 1.19   4: 1.15 / 1.17 / 1.21   16: 0.92 / 1.10 / 1.18
//                 chunk 64   1: 0.91 / 1.01 / 1.09   4: 0.90 / 1.01 / 1.10   16: 0.75 / 0.91 / 1.05
//   head dim 96   chunk 128  1: 1.18 / 1.13 /  -     4:  -   /  -   / 1.04   16:  -   / 0.99 / 1.04;   chunk 96  4, top-k 8: 1.08
// So: three tiles a list (ranks x chunk x heads of a group, in a long sequence whose tokens are all queries), and chunks of 64 to 95 keys
// at head dim 64 with seven ranks.
// A window of queries, or short sequences, have the lists of their whole prefix and few rows on each: what counts there is the rows that a
// list has on average (one_tile_rows), and a call of at most kOneTileFewItems items, where an SM has one or none, takes this
// kernel whatever they are.  Dense stage, this kernel against the one for short items (us), with the average:
//   18 rows   1000 tokens behind 50000, 16/16 heads, chunk 128, top-k 8   264 / 104
//   19        1254 behind 24248, 8/8, chunk 128, top-k 4                   77 / 36
//   221       50 sequences, 20476 tokens, 16/16, chunk 96, top-k 8        217 / 170
//   275       42 sequences, 6125 tokens, 32/8, chunk 96, top-k 3           88 / 63
//   358       3000 tokens, 16/16, chunk 128, top-k 4                     36.9 / 38.9
//   433       45 sequences, 35790 tokens, 16/16, chunk 96, top-k 12       421 / 439
//   497       9 sequences, 5068 tokens, 32/16, chunk 128, top-k 4        66.6 / 71.7
//   300 tokens, 16/4 heads, chunk 128, top-k 8 (46 items)                14.4 / 16.4
// By rows x keys of a list (chunks of 96 keys want a third more rows), over 380 calls of 130 to 60000 tokens, one sequence, batches and
// windows: lines of 256 to 448 rows of 128 keys choose within 0.3 % of the faster call on average, without one it was 3.5 %
// (at worst 1.85 x); at head dim 64 of 160 to 256, where 192 keeps the last entry of the table's last row here.
// Windows of at most 128 rows per kv head (few items, whose own-chunk ones cover the heads of a group) stay with the kernel for short items,
// and so does a q of more than 64 GB (row offsets are 32 bits there, in 16-byte pieces).
constexpr int kOneTileFewItems = 64;
// Rows of a list on average, as far as the host can tell: sequences taken to be of one length, a window to lie at the end of its prefix.
inline double one_tile_rows(const Params& p) {
  const double group_chunk = (double)p.G * p.C, hist = p.hist;
  if (p.Tq < p.T) {
    int64_t prefix = p.max_seqlen > p.Tq ? p.max_seqlen : p.Tq;
    if (prefix > p.T) prefix = p.T;
    return group_chunk * hist * (double)p.Tq / (double)prefix;
  }
  const double chunks = (double)p.T / ((double)p.B * p.C);   // of a sequence: the first is nobody's list, its tokens select nothing
  if (chunks <= 1) return 0;
  const double ranks = chunks >= hist + 1 ? hist * (chunks - (hist + 1) / 2) : chunks * (chunks - 1) / 2;
  return group_chunk * ranks / (chunks > 2 ? chunks - 1 : 1);
}
inline bool tc5_one_tile(const Params& p) {
  const bool keys = p.C >= 96 || (p.D == 64 && p.C >= 64 && p.hist >= 7);
  if (!tc5_short_items(p) || p.C > 128 || !keys || (int64_t)p.hist * p.C * p.G < 3 * kTileRowsWide || p.Tq * p.G <= kTileRowsWide ||
      (p.Tq - 1) * p.sq_t + (p.Hq - 1) * p.sq_h >= ((int64_t)1 << 35))
    return false;
  const int64_t items = (p.T * p.Hkv + p.rows) / p.C;
  return items <= kOneTileFewItems || one_tile_rows(p) * p.C >= (p.D == 64 ? 192 : 288) * 128.0;
}
// Windows of at most this many rows per kv head (decode steps) run a kernel that has keys, not rows, as the lanes of tensor memory
// (figures and the reason for eight there; chunks of any length: the shortest make no difference).
constexpr int kFewRows = 8;
inline bool tc5_few_rows(const Params& p) {
  return (p.D == 96 || p.D == 128) && p.Tq * p.G <= kFewRows;
}

// The kernel of the tcgen05 dense stage that runs a problem (MOBA_KERNEL_* of moba_b200.h).
inline int tc5_kernel(const Params& p) {
  if (p.D == 256) return p.C <= kSmallChunk ? MOBA_KERNEL_WIDE_SHORT : MOBA_KERNEL_WIDE;
  if (tc5_one_tile(p)) return MOBA_KERNEL_ONE_TILE;
  if (tc5_few_rows(p)) return MOBA_KERNEL_FEW_ROWS;
  return tc5_short_items(p) ? MOBA_KERNEL_SHORT : MOBA_KERNEL_ROWS_256;
}

cudaError_t launch_attend_mma(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                              const __nv_bfloat16* v, const int32_t* cu, const int32_t* list_counts,
                              const int32_t* list_offsets, const int32_t* tile_prefix,
                              const int32_t* row_list, __half* partial_out, float2* partial_lse,
                              int32_t* work_counter, cudaStream_t st);
cudaError_t launch_attend_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                              const __nv_bfloat16* v, const int32_t* cu, const int32_t* list_counts,
                              const int32_t* list_offsets, const int32_t* tile_prefix,
                              const int32_t* row_list, __half* partial_out, float2* partial_lse,
                              int32_t* work_counter, int32_t* status, cudaStream_t st);
cudaError_t launch_attend_one_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                  const int32_t* cu, const int32_t* list_counts, const int32_t* list_offsets,
                                  const int32_t* tile_prefix, const int32_t* row_list, __half* partial_out,
                                  float2* partial_lse, int32_t* work_counter, int32_t* status, int sms, cudaStream_t st);
cudaError_t launch_attend_few_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                  const int32_t* cu, const int32_t* list_counts, const int32_t* list_offsets,
                                  const int32_t* tile_prefix, const int32_t* row_list, __half* partial_out,
                                  float2* partial_lse, int32_t* work_counter, int32_t* status, int sms, cudaStream_t st);

cudaError_t launch_bounded_wait_probe(int32_t* status, unsigned long long limit_ns, cudaStream_t st);

// ---- backward (training path), attend_bwd.cu ---------------------------------
cudaError_t launch_count_lists(const Params& p, const int32_t* selected, int32_t* list_counts, cudaStream_t st);
cudaError_t launch_bwd_delta(const Params& p, const __nv_bfloat16* out, const __nv_bfloat16* dout, int64_t do_t,
                             int64_t do_h, const float* lse, float* delta, float* lse2, cudaStream_t st);
cudaError_t launch_bwd_dq(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                          const __nv_bfloat16* dout, int64_t do_t, int64_t do_h, const int32_t* cu,
                          const int32_t* list_counts, const int32_t* list_offsets, const int32_t* tile_prefix,
                          const int32_t* row_list, const float* lse2, const float* delta, float* partial_dq,
                          int32_t* work_counter, cudaStream_t st);
cudaError_t launch_bwd_dq_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                              const __nv_bfloat16* v, const __nv_bfloat16* dout, const int32_t* cu,
                              const int32_t* list_counts, const int32_t* list_offsets, const int32_t* tile_prefix,
                              const int32_t* row_list, const float* lse2, const float* delta, float* partial_dq,
                              int32_t* work_counter, int32_t* status, cudaStream_t st);
// Chunks of at most this many keys run the dq kernel of one-tile items.
constexpr int kDqShortChunk = 128;
inline bool bwd_dq_short_items(const Params& p) {
  return p.D <= 128 && p.C <= kDqShortChunk;
}
cudaError_t launch_bwd_dkdv_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                                const __nv_bfloat16* v, const __nv_bfloat16* dout, const int32_t* cu,
                                const int32_t* list_counts, const int32_t* list_offsets, const int32_t* row_list,
                                const float* lse2, const float* delta, __nv_bfloat16* dk, __nv_bfloat16* dv,
                                __nv_bfloat16* packed, int32_t* work_counter, int32_t* status, cudaStream_t st);
// 16-bit elements of the `packed` scratch of launch_bwd_dkdv_tc5 (Q and dO rows of the routed lists)
inline int64_t bwd_packed_elems(const Params& p) { return 2 * ((int64_t)p.hist * p.rows + 64) * p.D; }
cudaError_t launch_bwd_sum_dq(const Params& p, const float* partial_dq, const int32_t* selected, const int32_t* status,
                              __nv_bfloat16* dq, int64_t dq_t, int64_t dq_h, cudaStream_t st);
cudaError_t launch_bwd_dkdv(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                            const __nv_bfloat16* dout, int64_t do_t, int64_t do_h, const int32_t* cu,
                            const int32_t* list_counts, const int32_t* list_offsets, const int32_t* row_list,
                            const float* lse2, const float* delta, __nv_bfloat16* dk, int64_t dk_t, int64_t dk_h,
                            __nv_bfloat16* dv, int64_t dv_t, int64_t dv_h, int32_t* work_counter, cudaStream_t st);

}  // namespace moba
