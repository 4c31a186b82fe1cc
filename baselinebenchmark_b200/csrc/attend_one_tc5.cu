// Dense stage for chunks of 96 to 128 keys (64 and up at head dim 64 with seven ranks; tc5_one_tile says which calls): every work item is one 128-row tile of queries
// against one tile of keys, and one CTA per SM keeps three or four of them in flight.
//
// The work of such an item is small (1024 cycles of MMA at head dim 128, about as many of exponentials), its chain is
// long: Q rows, Q.K^T, S, softmax, P.V, O, rows.  attend_tc5_short_kernel runs two such chains per SM, in two CTAs that have one
// place for each operand; an item took 7000 cycles of a CTA.  Here all of an SM's tensor memory and shared memory serve one
// stream of items:
//   tensor memory  places of 128 columns (four at head dim 64, else three).  S takes a place, P its columns 0-63 once S has
//                  been read, and O dims 0-63 its columns 64-127; dims 64 and up go to the columns behind the places, of which there
//                  are two sets at head dim 128 (P.V waits for the rows of the item before last), one per place at 96.
//                  So Q.K^T of later items runs while the softmax of an item is under way
//   shared memory  Q in as many stages as there are places, K and V in two: the next list's K and V arrive behind the items of this one
//   warps 0-15   four softmax warpgroups, which take the items in turn: one thread per row, softmax and epilogue
//   warp 16      describes the items, in runs of consecutive tiles of a list (the rows are resolved by those who need them)
//   warps 17, 19 issue Q.K^T and P.V; 17 owns the tensor memory
//   warps 18, 24 K and V tiles (TMA), one of each per list or run of own-chunk items on the same keys
//   warps 20-23  Q rows (cp.async): two warps per item, in turn
// Bits: the operations and their order are those of the other tcgen05 kernels; rows come out the same.
//
// What bounds it: instructions.  An item takes 1550 issue slots of every scheduler and about 3100 cycles (2 x 4096 tokens x 16
// heads, ncu: slots 49 % busy, tensor pipe 32 %), since at most three of four softmax warps of a scheduler have a place to work
// on.  Dense stage, against attend_tc5_short_kernel (us): 2 x 4096 x 16 heads 124 -> 113, 13311 tokens x 16/4 at head dim 64 144 -> 119,
// 32768 x 32/8 1085 -> 976-997.  What each part gave there (first figure, from 136 with one warp for all MMAs): the MMAs in two warps
// 122, copies of three instructions 115, a third Q tile 111 to 113; runs in place of single descriptions 124 -> 119 on the second.
// Not kept: two threads a row (half of its scores and dims each; correct, but 88 registers spill: 214), all exponentials on the
// special-function unit (no difference at head dim 128, 122 -> 130 at 64).
#include "attend_rows.cuh"
#include "common.cuh"
#include "short_items.cuh"
#include "sm100_ptx.cuh"

namespace moba {

bool make_kv_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int Hkv, int64_t st,
                 int64_t sh, int box_rows);

namespace {

constexpr int kOneThreads = 800;
constexpr int kDescWarp = 16, kQkWarp = 17, kKWarp = 18, kPvWarp = 19, kCopyWarp = 20, kVWarp = 24;
constexpr int kOneRuns = 8;                // descriptions in flight
constexpr int kOneReaders = 24;            // warps that read them: all but the one that writes them
constexpr int kOneGroups = 4;              // softmax warpgroups

template <int D>
struct OneShape {
  static constexpr int kTile = (D + 63) / 64 * kHalfBytes;   // bytes of a Q, K or V tile
  static constexpr int kPlaces = D == 64 ? 4 : 3;            // of S, P and half of O in tensor memory
  static constexpr int kQ = D == 64 ? 4 : 3;                 // Q tiles
  static constexpr int kPrefix = D == 64 ? kShortPrefix : 448;   // ints of tile_prefix kept in shared memory
};

// A run: the tiles of one list that a draw covers, or one own-chunk tile; its items are tiles of 128 rows, the last one of what is left.
struct alignas(16) OneRun {
  int32_t flags;                           // kDone: the queue is empty; kFresh: K and V are not those of the run before; kCausal: own chunk
  int32_t rows, rows_at, qhead;            // see short_pick
  int32_t tok0, head;                      // first key token, kv head
  int32_t kv_len, tok_rel;
};
enum { kDone = 1, kFresh = 2, kCausal = 4 };

template <int kInts>
struct OneCtrl {
  static constexpr int kPrefix = kInts;
  uint64_t q_full[4], q_free[4];
  uint64_t k_full[2], k_free[2], v_full[2], v_free[2];
  uint64_t s_full[kOneGroups], o_full[kOneGroups];           // [softmax warpgroup]: each waits for phases of its own, in turn
  uint64_t p_full[4], o_free[4];                             // [place]
  uint64_t run_full[kOneRuns], run_free[kOneRuns];
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;
  SlotRange own;
  OneRun run[kOneRuns];
  int32_t prefix_cache[kInts];
};
// (The array is declared with the alignment of a swizzled block, and the kernel says so in the status if it should not have it.  Aligning the
// address in the kernel makes every base a register: 20 to 60 bytes spill, 113.7 -> 126 us on 2 x 4096 x 16 heads, 112 -> 139 on 13311 x 16/4 at 64.)
template <int D> constexpr size_t one_smem_bytes() {
  return (size_t)(OneShape<D>::kQ + 4) * OneShape<D>::kTile + sizeof(OneCtrl<OneShape<D>::kPrefix>);
}
static_assert(one_smem_bytes<128>() <= 232448, "shared memory of one CTA");

template <bool kHalf, int D>
__global__ void __launch_bounds__(kOneThreads, 1)
attend_tc5_one_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const ShortArgs sa) {
  using Shape = OneShape<D>;
  constexpr int kTile = Shape::kTile, kPlaces = Shape::kPlaces, kQ = Shape::kQ;
  constexpr uint32_t kTileDesc = kTile >> 4, kHi = 128 * kPlaces;             // first column behind the places
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t sQ = smem_u32(smem);
  const uint32_t sK = sQ + kQ * kTile;
  const uint32_t sV = sK + 2 * kTile;
  using Ctrl = OneCtrl<Shape::kPrefix>;
  Ctrl& c = *reinterpret_cast<Ctrl*>(smem + (kQ + 4) * kTile);
  const KernelArgs& a = sa.a;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (sQ & 1023) {
    pdl_wait();
    if (threadIdx.x == 0) atomicExch(a.status, ST_PRODUCER);
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&c.q_full[i]), 64);                   // the copies of two warps' lanes
      mbar_init(smem_u32(&c.q_free[i]), 1);
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.p_full[i]), kTileM);
      mbar_init(smem_u32(&c.o_full[i]), 1);
      mbar_init(smem_u32(&c.o_free[i]), kTileM);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.k_full[i]), 1);
      mbar_init(smem_u32(&c.k_free[i]), 1);
      mbar_init(smem_u32(&c.v_full[i]), 1);
      mbar_init(smem_u32(&c.v_free[i]), 1);
    }
    for (int i = 0; i < kOneRuns; ++i) {
      mbar_init(smem_u32(&c.run_full[i]), 1);
      mbar_init(smem_u32(&c.run_free[i]), kOneReaders);
    }
    c.abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == kQkWarp) {
    tmem_alloc(smem_u32(&c.tmem_slot), 512);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + own_item_count(c.own.n, p.Hq, p.C, kTileM);
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kOneThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  bool ok = true;                          // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  // The description of run r, for every warp but the one that writes them; false at the end (or when a wait gave up).
  int run = 0;
  OneRun d;
  auto next_run = [&]() {
    const int slot = run % kOneRuns;
    if (!wait(&c.run_full[slot], (run / kOneRuns) & 1)) return false;
    d = c.run[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&c.run_free[slot]));
    ++run;
    return (__shfl_sync(0xffffffffu, d.flags, 0) & kDone) == 0;
  };
  if (warp == kDescWarp) {
    // ---- descriptions
    ShortQueue w;
    short_start(sa.iq, c, w);
    int last_tok0 = -1, last_head = -1;
    for (bool done = false; !done; ++run) {
      ShortItem it;
      OneRun o;
      short_pick<true>(p, sa.iq, c, w, it, o.tok0, o.head, o.rows_at, o.qhead);
      done = it.done;
      o.rows = it.nrows;
      if (!done && !it.causal) {                               // the other tiles of the draw on this list
        const int tile = w.cur - w.list_first, more = min(w.end, w.list_end) - w.cur;
        if (more > 0) {
          o.rows += min(more * kTileM, w.list_count - tile * kTileM);
          w.cur += more;
        }
      }
      o.kv_len = it.kv_len;
      o.tok_rel = it.tok_rel;
      o.flags = (done ? kDone : 0) | (o.tok0 != last_tok0 || o.head != last_head ? kFresh : 0) | (it.causal ? kCausal : 0);
      last_tok0 = o.tok0;
      last_head = o.head;
      const int slot = run % kOneRuns;
      if (run >= kOneRuns && !wait(&c.run_free[slot], (run / kOneRuns - 1) & 1)) break;
      if (lane == 0) {
        c.run[slot] = o;
        mbar_arrive(smem_u32(&c.run_full[slot]));
      }
      __syncwarp();
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == kKWarp || warp == kVWarp) {
    // ---- K tiles, V tiles
    const bool is_v = warp == kVWarp;
    const CUtensorMap* m = is_v ? &tmap_v : &tmap_k;
    uint64_t* full = is_v ? c.v_full : c.k_full;
    uint64_t* free_ = is_v ? c.v_free : c.k_free;
    const uint32_t dst0 = is_v ? sV : sK;
    int at = 0;                            // tiles requested
    while (next_run()) {
      if (!(d.flags & kFresh)) continue;
      const int st = at & 1;
      if (at >= 2 && !wait(&free_[st], (at / 2 - 1) & 1)) break;
      ++at;
      if (lane == 0) {
        const uint32_t bar = smem_u32(&full[st]), dst = dst0 + st * kTile;
        mbar_expect_tx(bar, kTile);
        tma_load_3d(dst, m, bar, 0, d.head, d.tok0);
        if (D > 64) tma_load_3d(dst + kHalfBytes, m, bar, 64, d.head, d.tok0);
      }
      __syncwarp();
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp >= kCopyWarp) {
    // ---- Q rows: two warps the even items, two the odd ones; rows half * 64 ... + 63 each.  A warp of this kernel issues an
    // instruction every 14 cycles, so what counts is their number: three a copy (the row's offset from the lane that holds it, the
    // address, the copy), with the swizzled places in shared memory kept in registers and rows behind the item's last copied from
    // row 0 instead of left out.
    constexpr int kPieces = D / 8, kRows = 32 / kPieces;       // 16-byte pieces of a row, rows per instruction
    constexpr int kSwz = 8 / kRows;                            // instructions after which the swizzle repeats
    const int half = warp & 1, odd = ((warp - kCopyWarp) >> 1) & 1;
    const int ch = lane % kPieces, r0 = lane / kPieces;
    const bool copies = r0 < kRows;                            // 12 pieces (head dim 96): 24 of the 32 lanes copy
    uint32_t dst[kSwz];
#pragma unroll
    for (int i = 0; i < kSwz; ++i) {
      const int r = half * 64 + i * kRows + r0;
      dst[i] = sQ + (uint32_t)((ch >> 3) * kHalfBytes + r * 128 + (((ch & 7) ^ (r & 7)) << 4));
    }
    const uint4* src = reinterpret_cast<const uint4*>(a.q) + ch;
    int n = 0;
    while (ok && next_run()) {
      for (int t = 0; t < d.rows; t += kTileM, ++n) {
        if ((n & 1) != odd) continue;
        uint32_t off[2] = {0, 0};          // of rows half * 64 + lane and 32 behind it, in pieces
        const int r = t + half * 64 + lane;
        if (d.flags & kCausal) {
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (r + u * 32 < d.rows) off[u] = (uint32_t)(((int64_t)(d.rows_at + r + u * 32) * p.sq_t + (int64_t)d.qhead * p.sq_h) >> 3);
        } else {
          int e[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) e[u] = r + u * 32 < d.rows ? __ldg(a.row_list + d.rows_at + r + u * 32) : 0;
#pragma unroll
          for (int u = 0; u < 2; ++u) off[u] = (uint32_t)(entry_qoff(p, sa.iq, e[u]) >> 3);
        }
        const int st = n % kQ;
        if (n >= kQ && !wait(&c.q_free[st], (n / kQ - 1) & 1)) break;
        const uint32_t stage = (uint32_t)st * kTile;
        // eight copies at a time: their offsets first (a copy is a barrier to the compiler)
        constexpr int kCopies = (32 + kRows - 1) / kRows;      // of 32 rows
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
          for (int i0 = 0; i0 < kCopies; i0 += 8) {
            uint32_t o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = __shfl_sync(0xffffffffu, off[u], ((i0 + i) * kRows + r0) & 31);
            if (copies) {
#pragma unroll
              for (int i = 0; i < 8; ++i)
                cp_async_16(dst[(i0 + i) % kSwz] + stage + (uint32_t)((u * 32 + (i0 + i) / kSwz * 8) * 128), src + o[i]);
            }
          }
        }
        cp_async_mbar_arrive(smem_u32(&c.q_full[st]));
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == kQkWarp || warp == kPvWarp) {
    // ---- MMA issuers: Q.K^T of the items in one warp, P.V in another (each of the waits in front of an MMA takes some hundred
    // cycles of a warp that shares its scheduler).  The whole warp runs this code, one elected lane issues; what decides its
    // way is made the same in all lanes for the compiler too, so that operands stay in uniform registers.
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    static_assert(kQ == kPlaces, "one counter for both");
    int taken = 0, n = 0, place = 0, par = 0;   // K / V tiles, items, n mod kPlaces, (n / kPlaces) mod 2
    if (warp == kQkWarp) {
      while (ok && next_run()) {
        const int rows = __shfl_sync(0xffffffffu, d.rows, 0);
        if (__shfl_sync(0xffffffffu, d.flags, 0) & kFresh) {
          if (taken > 0) tc_commit_el(el, smem_u32(&c.k_free[(taken - 1) & 1]));      // behind the Q.K^T of the items before
          if (!wait(&c.k_full[taken & 1], (taken >> 1) & 1)) break;
          ++taken;
        }
        const uint32_t k = dk + (uint32_t)((taken - 1) & 1) * kTileDesc;
#pragma unroll 1
        for (int t = 0; t < rows; t += kTileM) {
          if (!wait(&c.q_full[place], par)) break;
          fence_proxy_async_smem();                           // rows written by cp.async, read by the tensor core
          if (n >= kPlaces && !wait(&c.o_free[place], par ^ 1)) break;
          tc_fence_after();
          const uint32_t q = dq + (uint32_t)place * kTileDesc;
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t koff = (uint32_t)((ks >> 2) * (kHalfBytes >> 4) + (ks & 3) * 2);
            mma_ss_el<kDescHi>(el, tm + place * 128, q + koff, k + koff, kIdescQK<kHalf>, ks > 0);
          }
          tc_commit_el(el, smem_u32(&c.s_full[n % kOneGroups]));
          tc_commit_el(el, smem_u32(&c.q_free[place]));
          ++n;
          if (++place == kPlaces) { place = 0; par ^= 1; }
        }
      }
    } else {
      while (ok && next_run()) {
        const int rows = __shfl_sync(0xffffffffu, d.rows, 0);
        if (__shfl_sync(0xffffffffu, d.flags, 0) & kFresh) {
          if (taken > 0) tc_commit_el(el, smem_u32(&c.v_free[(taken - 1) & 1]));
          if (!wait(&c.v_full[taken & 1], (taken >> 1) & 1)) break;
          ++taken;
        }
        const uint32_t v = dv + (uint32_t)((taken - 1) & 1) * kTileDesc;
#pragma unroll 1
        for (int t = 0; t < rows; t += kTileM) {
          // head dim 128: the columns of dims 64 and up were last those of item m - 2
          if (D == 128 && n >= 2 && !wait(&c.o_free[place == 2 ? 0 : place + 1], place == 2 ? par : par ^ 1)) break;
          if (!wait(&c.p_full[place], par)) break;
          tc_fence_after();
          const uint32_t pt = tm + place * 128;
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ts_el<kDescHi>(el, pt + 64, pt + ks * 8, v + ks * (2048 >> 4), kIdescPV<kHalf, 64>, ks > 0);
          if (D > 64) {
            const uint32_t hi = tm + kHi + (uint32_t)(D == 128 ? (n & 1) * 64 : place * 32);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)
              mma_ts_el<kDescHi>(el, hi, pt + ks * 8, v + (kHalfBytes >> 4) + ks * (2048 >> 4),
                                 kIdescPV<kHalf, D == 128 ? 64 : 32>, ks > 0);
          }
          tc_commit_el(el, smem_u32(&c.o_full[n % kOneGroups]));
          ++n;
          if (++place == kPlaces) { place = 0; par ^= 1; }
        }
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else {
    // ---- softmax + epilogue, one thread per row; warpgroup x takes items x, x + 4, ...
    const int x = warp >> 2;
    const int row0 = (warp & 3) * 32, row = row0 + lane;
    const uint32_t tl = tmem + ((uint32_t)row0 << 16);
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    int n = 0;
    while (ok && next_run()) {
      const bool causal = (d.flags & kCausal) != 0;
      for (int t = 0; t < d.rows; t += kTileM, ++n) {
        if (n % kOneGroups != x) continue;
        const int place = n % kPlaces;
        const uint32_t par = (n / kOneGroups) & 1;
        const bool active = t + row0 < d.rows;   // warps without rows only keep the barriers going
        int32_t e = -1;
        if (t + row < d.rows)
          e = causal ? (int32_t)(((int64_t)(d.rows_at + row) * p.Hq + d.qhead) * p.NP) : __ldg(a.row_list + d.rows_at + t + row);
        const int lim = causal ? min(d.kv_len, d.tok_rel + row + 1) : d.kv_len;  // keys < lim are visible
        const uint32_t tS = tl + place * 128;
        float m_ref = -INFINITY, l = 0.f;
        if (!wait(&c.s_full[x], par)) break;
        if (active) {
          tc_fence_after();
          const bool masked = kBN > d.kv_len || (causal && kBN - 1 > d.tok_rel);
          if (masked) softmax_row_rolled<true, kHalf, D>(tS, 0, 0, 0, lim, sl2, m_ref, l, [] {});
          else softmax_row_rolled<false, kHalf, D>(tS, 0, 0, 0, lim, sl2, m_ref, l, [] {});
          tc_fence_before();
        }
        mbar_arrive(smem_u32(&c.p_full[place]));
        if (!wait(&c.o_full[x], par)) break;
        if (active) {
          tc_fence_after();
          const uint32_t tO = tS + 64, tHi = tl + kHi + (uint32_t)(D == 128 ? (n & 1) * 64 : place * 32);
          // the row's largest magnitude decides the power of two its fp16 copy is scaled by
          const float amax = amax_row_rolled<D>(tO, tHi);
          const float inv = 1.f / l;
          const PartialScale ps = partial_scale(amax * inv);
          store_row_rolled<D>(tO, tHi, a.partial_out + (int64_t)(e >= 0 ? e : 0) * D, inv * ps.scale, e >= 0,
                              a.wide_store != 0, [&] {
                                tc_fence_before();
                                mbar_arrive(smem_u32(&c.o_free[place]));   // the place may be overwritten
                              });
          if (e >= 0) a.partial_lse[e] = make_float2((m_ref + log2f(l)) * 0.6931471805599453f, ps.inv);
        } else {
          mbar_arrive(smem_u32(&c.o_free[place]));
        }
      }
    }
    if (!ok) {
      atomicExch(a.status, ST_SOFTMAX);
      c.abort = 1;
    }
  }

  // a role that gave up leaves the others to run into their own bounded waits
  __syncwarp();
  __syncthreads();
  if (c.abort) {                           // copies in flight land before shared memory is given up
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kQkWarp) tmem_dealloc(tmem, 512);
}

template <bool kHalf, int D>
cudaError_t launch_one(const Params& p, const CUtensorMap& mk, const CUtensorMap& mv, const ShortArgs& sa, int sms,
                       cudaStream_t st) {
  constexpr size_t smem = one_smem_bytes<D>();
  const cudaError_t e = prepare_kernel(attend_tc5_one_kernel<kHalf, D>, smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(attend_tc5_one_kernel<kHalf, D>, dim3(sms), kOneThreads, smem, st, p, mk, mv, sa);
}

}  // namespace

cudaError_t launch_attend_one_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                  const int32_t* cu, const int32_t* list_counts, const int32_t* list_offsets,
                                  const int32_t* tile_prefix, const int32_t* row_list, __half* partial_out,
                                  float2* partial_lse, int32_t* work_counter, int32_t* status, int sms, cudaStream_t st) {
  CUtensorMap mk, mv;
  if (!make_kv_map(&mk, p.fp16 != 0, p.D, k, p.T, p.Hkv, p.sk_t, p.sk_h, kBN) ||
      !make_kv_map(&mv, p.fp16 != 0, p.D, v, p.T, p.Hkv, p.sv_t, p.sv_h, kBN))
    return cudaErrorNotSupported;
  ShortArgs sa;
  sa.a = KernelArgs{q, cu, list_counts, list_offsets, tile_prefix, row_list, partial_out, partial_lse,
                    work_counter, status, ((uintptr_t)partial_out & 31) == 0};
  sa.iq = item_queue(p, cu, list_counts, list_offsets, tile_prefix, row_list, work_counter, short_batch(p, 2 * sms, false), false, 0);
  switch (p.D) {
    case 64: return p.fp16 ? launch_one<true, 64>(p, mk, mv, sa, sms, st) : launch_one<false, 64>(p, mk, mv, sa, sms, st);
    case 96: return p.fp16 ? launch_one<true, 96>(p, mk, mv, sa, sms, st) : launch_one<false, 96>(p, mk, mv, sa, sms, st);
    case 128: return p.fp16 ? launch_one<true, 128>(p, mk, mv, sa, sms, st) : launch_one<false, 128>(p, mk, mv, sa, sms, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace moba
