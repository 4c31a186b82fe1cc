// Work items of one 128-row tile: the description of an item and the walk through the queue of items,
// shared by the kernels whose roles run through a flat stream of items (the forward's kernels for
// one-tile and short items and for head dim 256, and the dq kernel for short chunks).
#pragma once

#include "common.cuh"
#include "fast_div.cuh"
#include "sm100_ptx.cuh"

namespace moba {
namespace {

constexpr int kShortPrefix = 2048;         // ints of tile_prefix kept in shared memory
constexpr int kShortSlots = 4;             // item descriptions in flight

// tile_prefix is kept in shared memory sampled every 2^shift entries (shift 0: whole), so that
// finding the list of a routed item costs a round or two of global loads (find_list).
__host__ __device__ inline int prefix_shift(int64_t lists, int cache_entries) {
  int shift = 0;
  while ((lists >> shift) + 2 > cache_entries) ++shift;
  return shift;
}
template <typename CtrlT>
__device__ __forceinline__ void fill_prefix_cache(CtrlT& c, const int32_t* __restrict__ tile_prefix, int64_t lists,
                                                  int nthreads) {
  const int shift = prefix_shift(lists, CtrlT::kPrefix);
  const int n = (int)(lists >> shift) + 1;                   // samples 0, 2^shift, ..., the last one <= lists
  for (int i = threadIdx.x; i < n; i += nthreads) c.prefix_cache[i] = tile_prefix[(int64_t)i << shift];
}
// last k in [0, n) with at(k) <= i, at rising and at(0) <= i: 32 places a round, one for each lane of the (whole) warp
template <typename F>
__device__ __forceinline__ int search_warp(int n, int i, F&& at) {
  const int lane = threadIdx.x & 31;
  int lo = 0;
  while (n > 1) {
    const int step = (n + 31) >> 5, k = lane * step;
    const int m = __popc(__ballot_sync(0xffffffffu, k < n && at(lo + k) <= i)) - 1;
    lo += m * step;
    n = min(step, n - m * step);
  }
  return lo;
}
// last l in [0, lists) with tile_prefix[l] <= i (i is a routed item: tile_prefix[lists] > i); executed by a whole warp.
// (Halving took eleven dependent reads where this takes two or three: with several items of an SM in flight the warp that
// describes them was what the others waited for.)
template <typename CtrlT>
__device__ __forceinline__ int find_list(const CtrlT& c, const int32_t* __restrict__ tile_prefix, int64_t lists, int i) {
  const int shift = prefix_shift(lists, CtrlT::kPrefix);
  const int l = search_warp((int)(lists >> shift) + 1, i, [&](int k) { return c.prefix_cache[k]; }) << shift;
  // tile_prefix[l + 2^shift] > i, or the lists end before
  return l + search_warp(min(1 << shift, (int)lists - l), i, [&](int k) { return __ldg(tile_prefix + l + k); });
}

// Where the items come from.
struct ItemQueue {
  const int32_t* cu;
  const int32_t* list_counts;
  const int32_t* list_offsets;
  const int32_t* tile_prefix;
  const int32_t* row_list;
  int32_t* work_counter;
  int32_t batch;                           // items a CTA draws at a time
  int32_t grouped;                         // own-chunk items cover the heads of a group (short windows)
  int32_t tile_shift;                      // 1: the tiles of tile_prefix are 256 rows, two items each
  FastDiv by_np, by_hq, by_hkv, by_mc, by_g;
};
inline ItemQueue item_queue(const Params& p, const int32_t* cu, const int32_t* list_counts, const int32_t* list_offsets,
                            const int32_t* tile_prefix, const int32_t* row_list, int32_t* work_counter, int batch, bool grouped,
                            int tile_shift) {
  return ItemQueue{cu, list_counts, list_offsets, tile_prefix, row_list, work_counter, batch, grouped, tile_shift,
                   fast_div(p.NP), fast_div(p.Hq), fast_div(p.Hkv), fast_div(p.mc), fast_div(p.G)};
}
// A CTA draws several items at a time, so that row tiles of one list follow one another on it (K and V
// stay in place), but at most an eighth of its share of the launch, for the balance.
inline int short_batch(const Params& p, int ctas, bool grouped) {
  const int64_t items = p.hist * p.rows / kTileRowsWide + (grouped ? 0 : p.rows / kTileRowsWide);
  const int64_t share = items / (ctas * 8);
  return share < 1 ? 1 : share > 8 ? 8 : (int)share;
}

// CTAs for a window of at most 128 rows per kv head: no more than it can have items, one per list its rows can be
// on and one per kv head and chunk it touches.  With two CTAs per SM waiting for work, few items gathered in pairs on
// some SMs while others had none.  Dense stage, chunk 4096, top-k 8, against the 256-row kernel with one CTA per SM:
//   20011 tokens, 16/4 heads, 32 new   74 us there, 86 with all CTAs, 70 with this many
//   131072, 16/4, 32 new               84           98                76
//   131072, 8/8, 1 new                 78           83                74
//   131072, 32/8, 1 new               144           86                86   (more items than SMs)
inline int window_ctas(const Params& p, int ctas) {
  const int64_t routed = p.hist * p.rows < p.lists ? p.hist * p.rows : p.lists;
  int64_t chunks = p.Tq / p.C + p.B + 1;                     // every sequence may add a part of a chunk
  if (chunks > p.Tq) chunks = p.Tq;
  const int64_t items = routed + chunks * p.Hkv;
  return items < ctas ? (int)items : ctas;
}

struct ShortItem {
  int32_t done;                            // 1: the queue is empty
  int32_t new_kv;                          // 0: K and V of the item before are those of this one (one tile)
  int32_t nrows, causal;
  int32_t kv_len;
  int32_t tok_rel;                         // own chunk: first query token minus first key token
  int32_t group;                           // own chunk: rows per token (1, or the heads of the group)
  int32_t tile0;                           // 128-key tiles of the CTA before this item
  int32_t tok0, head;                      // first key token, kv head
};

// Walks the items a CTA draws; executed by the whole describing warp.
struct ShortQueue {
  int cur, end;                            // items of the current draw left: [cur, end)
  int ahead, drawn, dealt;                 // short_pick<true>, see short_start: the draw behind it (lane 0), draws so far, of them without the counter
  int list, list_first, list_end;          // list of the last routed item and the items it covers
  int list_off, list_count, kv_tok0, kv_head;
};
template <typename CtrlT>
__device__ __forceinline__ int short_draw(const ItemQueue& a, const CtrlT& c) {
  return (threadIdx.x & 31) != 0 ? 0 : c.abort ? 0x3fffffff : atomicAdd(a.work_counter, 1);
}
// A draw that is asked for before the one in hand is used up.  A CTA that describes its items far ahead would draw several before
// others have started, so the first draws of every CTA are dealt out instead: CTA b has draws b, b + CTAs, ... .  Nine is what a CTA can
// draw before its first item is done (eight descriptions of one-tile items ahead, and the draw ahead).  Dense stage (us) with 0 / 1 / 2 / 9 dealt:
//   one decode step on 131072 tokens, 8/1 heads, top-k 12 (32 items at most)   86.0 / 51.2 / 51.2 / 51.2
//   32/8 and 16/16 heads, and behind 20479 and 65536 tokens                  all the same (63.5, 49.2, 16.4, 30.7)
//   one-tile items: 2 x 4096 x 16 119.8 / 117.8 / 118.8 / 115.7, 32768 x 32/8 1020 / 1014 / 1022 / 1022, 13311 x 16/4 at head dim 64
//   112 / 112 / 111 / 112: what is dealt in advance costs no balance there (the runs of one side differ by 3 %)
constexpr int kDealt = 9;
template <typename CtrlT>
__device__ __forceinline__ int short_draw_ahead(const ItemQueue& a, const CtrlT& c, ShortQueue& w) {
  const int d = w.drawn++;
  if (d < w.dealt) return d * (int)gridDim.x + (int)blockIdx.x;
  return w.dealt * (int)gridDim.x + short_draw(a, c);
}
template <typename CtrlT>
__device__ __forceinline__ void short_start(const ItemQueue& a, const CtrlT& c, ShortQueue& w) {
  w.cur = w.end = 0;
  w.list = -1;
  w.list_first = w.list_end = 0;
  w.list_off = w.list_count = w.kv_tok0 = w.kv_head = 0;
  const int big = max(c.n_items - 2 * (int)gridDim.x, 0) / a.batch, draws = big + c.n_items - big * a.batch;
  w.drawn = 0;
  w.dealt = min((draws + (int)gridDim.x - 1) / (int)gridDim.x, kDealt);
  w.ahead = short_draw_ahead(a, c, w);
}

// The next item: its description in `it`, its first key token and kv head, and where its rows are: from row_list[rows_at]
// on, or (own chunk) query tokens of the window from rows_at on, heads from `head` on.
// kDrawAhead: the draw behind the one in hand is under way (short_start), so that its latency is not waited for.
template <bool kDrawAhead, typename CtrlT>
__device__ __forceinline__ void short_pick(const Params& p, const ItemQueue& a, CtrlT& c, ShortQueue& w, ShortItem& it,
                                           int& kv_tok0, int& kv_head, int& rows_at, int& head) {
  const int n_routed = c.n_routed, n_items = c.n_items;
  it.done = 1;
  it.nrows = 0;
  it.causal = 0;
  it.kv_len = 0;
  it.tok_rel = 0;
  it.group = 1;
  kv_tok0 = 0;
  kv_head = 0;
  rows_at = 0;
  head = 0;
  for (;;) {
    if (w.cur >= w.end) {
      const int mine = kDrawAhead ? w.ahead : short_draw(a, c);
      if (kDrawAhead) w.ahead = short_draw_ahead(a, c, w);
      const int idx = __shfl_sync(0xffffffffu, mine, 0);
      // Draws of `batch` items, and of single ones for the last two of every CTA: with a whole batch drawn last, some
      // CTAs worked three items longer than others.  Against batches to the end: dense stage of 2 x 4096 tokens x 16
      // heads 127.3 -> 125.9 us, at head dim 256 290 -> 281; 8191 x 16/4 122.5 -> 118.
      const int big = max(n_items - 2 * (int)gridDim.x, 0) / a.batch;
      w.cur = idx < big ? idx * a.batch : big * a.batch + (idx - big);
      w.end = idx < big ? w.cur + a.batch : w.cur + 1;
      if (w.cur >= n_items) return;
    }
    const int idx = w.cur++;
    if (idx < n_routed) {
      const int cut = idx >> a.tile_shift;                    // tile of tile_prefix
      if (cut < w.list_first || cut >= w.list_end) {
        const int l = find_list(c, a.tile_prefix, p.lists, cut);
        const int slot = l / a.by_hkv;
        const int b = slot / a.by_mc, j = slot - b * p.mc;
        w.list = l;
        w.list_first = __ldg(a.tile_prefix + l);
        w.list_end = __ldg(a.tile_prefix + l + 1);
        w.list_off = __ldg(a.list_offsets + l);
        w.list_count = __ldg(a.list_counts + l);
        w.kv_tok0 = __ldg(a.cu + b) + j * p.C;
        w.kv_head = l - slot * p.Hkv;
      }
      const int tile = idx - (w.list_first << a.tile_shift);
      if (tile * kTileRowsWide >= w.list_count) continue;     // the second half of a 256-row tile may be empty
      it.nrows = min(w.list_count - tile * kTileRowsWide, kTileRowsWide);
      it.kv_len = p.C;
      kv_tok0 = w.kv_tok0;
      kv_head = w.kv_head;
      rows_at = w.list_off + tile * kTileRowsWide;
      break;
    }
    // own chunk: rows are (token, head) pairs, `group` heads per token
    const int g = a.grouped ? p.G : 1;
    const int units = a.grouped ? p.Hkv : p.Hq;
    // grouped: a slot's part of the window is one item
    const int tiles_per_chunk = a.grouped ? 1 : (p.C + kTileRowsWide - 1) / kTileRowsWide;
    const int per_tile = c.own.n * units;
    int i = idx - n_routed;
    int ti = 0;
    if (tiles_per_chunk > 1) {
      const int x = i / per_tile;
      ti = tiles_per_chunk - 1 - x;                           // longest tiles first
      i -= x * per_tile;
    }
    const int unit = i / (a.grouped ? a.by_hkv : a.by_hq), slot = c.own.lo + unit;
    head = (i - unit * units) * g;
    const int b = slot / a.by_mc, j = slot - b * p.mc;
    const Slot s = slot_of(a.cu, b, j, p.C);
    const int tile0 = s.start + ti * kTileRowsWide;
    const int lo = max(tile0, p.win_lo);
    const int hi = min(a.grouped ? s.end : min(tile0 + kTileRowsWide, s.end), p.win_lo + (int)p.Tq);
    if (lo >= hi) continue;
    it.nrows = (hi - lo) * g;
    it.causal = 1;
    it.group = g;
    it.tok_rel = lo - s.start;
    it.kv_len = hi - s.start;
    kv_tok0 = s.start;
    kv_head = head / a.by_g;
    rows_at = lo - p.win_lo;
    break;
  }
  it.done = 0;
}

// Element offset in q of the row of an entry id (t * Hq + h) * NP + rank.
__device__ __forceinline__ int64_t entry_qoff(const Params& p, const ItemQueue& a, int entry) {
  const int row = entry / a.by_np, t = row / a.by_hq;
  return (int64_t)t * p.sq_t + (int64_t)(row - t * p.Hq) * p.sq_h;
}

// The next item with its rows: those of this lane (4 * lane ... + 3) in `ent` (-1: none, behind the last row), their
// element offsets in q in `qoff`.
template <typename CtrlT>
__device__ __forceinline__ void short_next(const Params& p, const ItemQueue& a, CtrlT& c, ShortQueue& w, ShortItem& it,
                                           int& kv_tok0, int& kv_head, int (&ent)[4], int64_t (&qoff)[4]) {
  const int lane = threadIdx.x & 31;
  int rows_at, head;
  short_pick<false>(p, a, c, w, it, kv_tok0, kv_head, rows_at, head);
#pragma unroll
  for (int u = 0; u < 4; ++u) { ent[u] = -1; qoff[u] = 0; }
  if (it.done) return;
  if (!it.causal) {
    const int32_t* rows = a.row_list + rows_at + 4 * lane;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (4 * lane + u < it.nrows) ent[u] = __ldg(rows + u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (ent[u] >= 0) qoff[u] = entry_qoff(p, a, ent[u]);
    return;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int r = 4 * lane + u;
    if (r < it.nrows) {
      const int x = it.group == 1 ? r : r / a.by_g;           // (a group is the heads of a kv head)
      const int t = rows_at + x, h = head + r - x * it.group;
      ent[u] = (int32_t)(((int64_t)t * p.Hq + h) * p.NP);
      qoff[u] = (int64_t)t * p.sq_t + (int64_t)h * p.sq_h;
    }
  }
}

// Rows [0, nrows) of an item into a 128-byte-swizzled tile of [128][64] blocks, by kWarps warps (this one is number
// `part`): pieces [piece0, piece0 + kPieces) of 16 bytes of each row, whole rows per instruction.  off(r):
// element offset of row r from `base`.
template <int kPieces, int kWarps, typename F>
__device__ __forceinline__ void copy_rows_async(uint32_t tile, const __nv_bfloat16* base, int piece0, int part, int nrows,
                                                F&& off) {
  constexpr int kRowsPerInstr = 32 / kPieces;
  const int lane = threadIdx.x & 31;
  const int ch = lane % kPieces, r0 = lane / kPieces;
  const uint32_t dst = tile + (uint32_t)((ch >> 3) * (128 * 128));
  const __nv_bfloat16* src = base + (piece0 + ch) * 8;
  constexpr int kStride = kWarps * kRowsPerInstr, kBatch = 8;
  if (r0 < kRowsPerInstr) {                                    // 12 pieces (head dim 96): 24 of the 32 lanes copy
    // The offsets of a batch are read before its first copy: a copy is a barrier to the compiler, and with a shared-memory
    // read in front of every one of them it took 130 cycles a copy, the longest link of the chain of a one-tile item.
    // 2 x 4096 tokens x 16 heads, chunk 128: dense stage 133 -> 128 us, at head dim 256 314 -> 291; dq of 8191 tokens x
    // 16/4 heads 254 -> 238.
#pragma unroll 1
    for (int r = r0 + part * kRowsPerInstr; r < nrows; r += kBatch * kStride) {
      int64_t o[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) o[u] = r + u * kStride < nrows ? off(r + u * kStride) : 0;
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int x = r + u * kStride;
        if (x < nrows) ptx::cp_async_16(dst + (uint32_t)(x * 128 + (((ch & 7) ^ (x & 7)) << 4)), src + o[u]);
      }
    }
  }
}

// One warp describes the items of the CTA ahead of everybody else: item m goes into slot m % kSlots of the
// control block once the slot's item before has been let go by its readers (slot_free: every reader either arrives on it
// or is ordered before one that does, which each kernel argues at its mbar_init), and the
// end of the queue is published `kEnds` times (once per group of threads that takes the items in turn).
// False when a wait gave up.  kRowIndex: row indices t * Hq + h are kept too.
template <int kSlots, int kEnds, bool kReuse, bool kRowIndex, typename CtrlT>
__device__ __forceinline__ bool describe_items(const Params& p, const ItemQueue& iq, CtrlT& c) {
  const int lane = threadIdx.x & 31;
  ShortQueue w;
  w.cur = w.end = 0;
  w.list = -1;
  w.list_first = w.list_end = 0;
  w.list_off = w.list_count = w.kv_tok0 = w.kv_head = 0;
  ShortItem it;
  int ent[4], tok0, head, last_tok0 = -1, last_head = -1, ends = 0;
  int64_t qoff[4];
  uint32_t tiles = 0;
  for (int n = 0; ends < kEnds; ++n) {
    if (ends == 0) short_next(p, iq, c, w, it, tok0, head, ent, qoff);
    it.new_kv = !(kReuse && tok0 == last_tok0 && head == last_head);
    it.tok0 = tok0;
    it.head = head;
    it.tile0 = (int32_t)tiles;
    tiles += (uint32_t)(it.kv_len + 127) >> 7;
    last_tok0 = tok0;
    last_head = head;
    ends += it.done;
    const int slot = n % kSlots;
    if (n >= kSlots &&
        !__all_sync(0xffffffffu, ptx::mbar_wait(ptx::smem_u32(&c.slot_free[slot]), ((n / kSlots) - 1) & 1)))
      return false;
    *reinterpret_cast<int4*>(&c.entry[slot][4 * lane]) = make_int4(ent[0], ent[1], ent[2], ent[3]);
    *reinterpret_cast<longlong2*>(&c.qoff[slot][4 * lane]) = make_longlong2(qoff[0], qoff[1]);
    *reinterpret_cast<longlong2*>(&c.qoff[slot][4 * lane + 2]) = make_longlong2(qoff[2], qoff[3]);
    if constexpr (kRowIndex) {
      int row[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) row[u] = ent[u] >= 0 ? ent[u] / iq.by_np : 0;
      *reinterpret_cast<int4*>(&c.grow[slot][4 * lane]) = make_int4(row[0], row[1], row[2], row[3]);
    }
    if (lane == 0) c.item[slot] = it;
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&c.item_full[slot]));
  }
  return true;
}

__device__ __forceinline__ void store32(void* ptr, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(ptr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

}  // namespace
}  // namespace moba
