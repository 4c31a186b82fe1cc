// dQ of the MoBA dense stage on the Blackwell tensor path (tcgen05.mma, accumulators in
// tensor memory, K/V tiles staged by TMA).
//
// Replaces, for the training path of the reference, the dq kernel of
//   _triton_varlen_backward   backends/_mthreads/ops/moba/attention.py:163-369
// as called for both branches by MixedAttention.backward (parallel.py:171-236): with the
// merged LSE and delta_i = sum_d dO_id O_id of the merged output,
//   p_ij = exp(s_ij * scale - lse_i),  dS_ij = p_ij (dO_i . V_j - delta_i),
//   dQ_i = scale * sum_j dS_ij K_j.
//
// Work items are those of the forward's tcgen05 dense stage: up to 256 query rows (two
// 128-row MMA tiles, "A" and "B") against the keys of one chunk, visited in tiles of 64 keys.
// Per tile step and row tile X the tensor core computes
//   S_X  = Q_X . K^T     (128 x 64, operands in shared memory)
//   dP_X = dO_X . V^T    (128 x 64, operands in shared memory)
//   dQ_X += dS_X . K     (128 x D, dS read from tensor memory, K as the MN-major operand)
// and one thread per row turns S and dP into dS (input dtype) in between.  Each item writes
// scale * dQ as an fp32 partial into the row's slot (own chunk = 0, rank r = r + 1); a later
// kernel adds a row's slots.  No atomics: the result is bit-identical run to run.
//
// Warp roles (512 threads), in one flat stream of items and key tiles without a CTA-wide barrier: warp 0 TMA
// producer (K tiles in three stages, V tiles in two), warp 1 MMA issuer and owner of the TMEM allocation,
// warp 2 draws and resolves the next item, warps 4-7 / 8-11 the rows of tile A / B, warps 12-15 copy a tile's Q
// and dO rows (cp.async) as soon as the last S / dP of the item before has executed.  When the row threads
// gathered their rows behind a barrier at the item's start the kernel took 950 us on 19456 tokens x 32 heads,
// chunk 512, 837 us this way.
// TMEM columns of row tile X: S 128X..128X+63 (dS, 16-bit, overwrites the first 32),
// dP 128X+64..128X+127, dQ 256+128X..; 512 columns in all, which is why a key step is 64 wide.
// Every wait is bounded; a wait that gives up sets a status word that the summing kernel
// turns into NaN results.
#include "common.cuh"
#include "short_items.cuh"
#include "sm100_ptx.cuh"

namespace moba {

// defined with the forward kernel: tiled map of a [T, Hkv, D] tensor, boxes of `box_rows` x 1 x 64
bool make_kv_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int Hkv, int64_t st,
                 int64_t sh, int box_rows);

namespace {

using namespace ptx;

constexpr int kThreads = 512;
constexpr int kTileM = 128;                 // rows per MMA tile
constexpr int kBN = 64;                     // keys per step
constexpr int kQBlockBytes = 128 * 64 * 2;  // one [128 rows][64 dims] swizzled block of Q or dO
constexpr int kQTileBytes = 2 * kQBlockBytes;
constexpr int kKvBlockBytes = kBN * 64 * 2; // one [64 keys][64 dims] swizzled block of K or V
constexpr int kKvTileBytes = 2 * kKvBlockBytes;
constexpr uint32_t kTmemCols = 512;
constexpr int kPrefixCache = 2048;          // ints of tile_prefix kept in shared memory
constexpr int kKStages = 3;                 // K tiles serve S (early) and dQ (late): three stages give the next one a full step of lead

template <bool kHalf> constexpr uint32_t kIdescS = idesc_16_f32(kHalf, 128, kBN, 0, 0);
template <bool kHalf, int D> constexpr uint32_t kIdescDQ = idesc_16_f32(kHalf, 128, D, 0, 1);

enum { ST_OK = 0, ST_PRODUCER = 11, ST_MMA = 12, ST_ROWS = 13 };

struct Ctrl {
  uint64_t k_full[kKStages], k_empty[kKStages], v_full[2], v_empty[2];
  uint64_t s_full[2], ds_full[2], dq_full[2];
  uint64_t rows_full[2], rows_free[2];       // per item: Q and dO of tile A / B landed; its last S / dP has executed
  uint64_t item_full[2], slot_free[2];
  uint32_t tmem_slot;
  volatile int32_t abort;
  Item item[2];                              // slot (n & 1) holds item n, described an item ahead
  int32_t done[2];
  int64_t qoff[2][2 * kTileM];               // element offset of the row in q
  int32_t grow[2][2 * kTileM];               // row index t * Hq + h (dO, lse and delta are indexed by it)
  int32_t entry[2][2 * kTileM];              // partial slot of the row, -1: no row
  int32_t prefix_cache[kPrefixCache];
};

constexpr size_t kSmemBytes = 1024 /*alignment slack*/ + 4 * kQTileBytes + (kKStages + 2) * kKvTileBytes + sizeof(Ctrl);
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");

struct KernelArgs {
  const __nv_bfloat16* q;
  const __nv_bfloat16* dout;                 // contiguous [T, Hq, D]
  const int32_t* cu;
  const int32_t* list_counts;
  const int32_t* list_offsets;
  const int32_t* tile_prefix;
  const int32_t* row_list;
  const float* lse2;                         // lse * log2(e), [rows]
  const float* delta;                        // [rows]
  float* partial_dq;
  int32_t* work_counter;
  int32_t* status;
  int32_t wide_store;                        // partial_dq is 32-byte aligned
};

// One warp, an item ahead of the others: draws the next item from the global queue, decodes it,
// resolves its rows into slot `slot` and publishes it.  False when the queue is empty.
__device__ __forceinline__ bool describe_item(const Params& p, const KernelArgs& a, Ctrl& c, int slot,
                                              int n_routed, int n_items) {
  const int lane = threadIdx.x & 31;
  Item it;
  it.valid = 0;
  int done = 0;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = c.abort ? 0x7fffffff : atomicAdd(a.work_counter, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= n_items) { done = 1; break; }
    it = decode_item(p, idx, n_routed, 2 * kTileM, a.cu, a.list_counts, a.list_offsets,
                     p.lists < kPrefixCache ? c.prefix_cache : a.tile_prefix);
    if (it.valid) break;
  }
  if (lane == 0) { c.item[slot] = it; c.done[slot] = done; }
  if (!done) {
    int32_t ent[2 * kTileM / 32];
#pragma unroll
    for (int u = 0; u < 2 * kTileM / 32; ++u) {
      const int r = lane + 32 * u;
      ent[u] = -1;
      if (r < it.nrows) {
        if (it.causal) ent[u] = (int32_t)(((int64_t)(it.tok0 - p.win_lo + r) * p.Hq + it.head) * p.NP);
        else ent[u] = __ldg(a.row_list + it.row_start + r);
      }
    }
#pragma unroll
    for (int u = 0; u < 2 * kTileM / 32; ++u) {
      const int r = lane + 32 * u;
      const int32_t e = ent[u];
      int64_t off = 0;
      int32_t row = 0;
      if (e >= 0) {
        row = e / p.NP;
        const int64_t t = row / p.Hq;
        off = t * p.sq_t + (row - t * p.Hq) * p.sq_h;
      }
      c.entry[slot][r] = e;
      c.qoff[slot][r] = off;
      c.grow[slot][r] = row;
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&c.item_full[slot]));
  return done == 0;
}

// Exponentials evaluated with the cubic on the FMA pipe instead of the special-function
// unit: kPolyPairs of every 8 column pairs (never in masked steps, where a masked column must
// give exactly zero).
#ifndef MOBA_BWD_POLY_PAIRS
#define MOBA_BWD_POLY_PAIRS 2
#endif
constexpr int kPolyPairs = MOBA_BWD_POLY_PAIRS;

// One step of one row: S and dP (64 fp32 columns each of this thread's TMEM lane) -> dS in
// the input dtype, written over the first 32 columns of S.
//   p = 2^(s * scale * log2 e - lse * log2 e),  dS = p * (dP - delta)
// Rows that do not exist carry lse = +inf, but their Q and dO rows are whatever the tile held before, NaN
// included: their dS and dQ rows may be anything, are never stored and are added to nothing (a row of the tile only
// enters its own row of S, dP and dQ).
template <bool kMasked, bool kHalf, bool kUnrolled>
__device__ __forceinline__ void ds_row(uint32_t tS, int key0, int lim, float sl2, float neg_lse2, float delta) {
  // 32 keys at a time: with sixteen warps a thread has 128 registers.  Unrolled, the step is ready a little earlier, which
  // counts where a step waits for it and for the tensor core in turn (head dim 96, 128, long items: 64 steps 106 -> 105
  // us); rolled it is less code to fetch, which counts at head dim 64 (16384 tokens x 16/4, chunk 4096 1024 -> 985) and for items of one or two steps.
  const uint64_t scale2 = pack2(sl2, sl2);
  const uint64_t nl2 = pack2(neg_lse2, neg_lse2);
  const uint64_t dl2 = pack2(delta, delta);
#pragma unroll(kUnrolled ? 2 : 1)
  for (int ch = 0; ch < 2; ++ch) {
    uint32_t s[32], g[32], pk[16];
    tmem_ld32(tS + ch * 32, s);
    tmem_ld32(tS + 64 + ch * 32, g);
    tmem_wait_ld();
    if (kMasked) {
#pragma unroll
      for (int i = 0; i < 32; ++i) s[i] = (i < lim - key0 - ch * 32) ? s[i] : 0xff800000u;   // -inf: p = 0
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int e = 2 * i;
      const uint64_t x = fma2(pack2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), scale2, nl2);
      uint64_t pr;
      if (!kMasked && (i & 7) < kPolyPairs) pr = ex2_poly2(x);
      else pr = pack2(ex2_approx(lo2(x)), ex2_approx(hi2(x)));
      const uint64_t d = mul2(pr, sub2(pack2(__uint_as_float(g[e]), __uint_as_float(g[e + 1])), dl2));
      pk[i] = pack2_16<kHalf>(lo2(d), hi2(d));
    }
    tmem_st16(tS + ch * 16, pk);
  }
  tmem_wait_st();
}

// Shared-memory descriptor words (128-byte swizzle).  Low word: start address >> 4 |
// (leading byte offset >> 4) << 16; high word: stride byte offset 1024 >> 4 | version 1 << 14
// | SWIZZLE_128B (2) << 29.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo_bytes) {
  return ((addr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
}
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);

// S_X = Q_X . K^T and dP_X = dO_X . V^T for one 64-key tile: D / 16 k-steps each; `dk`, `dv`:
// descriptor words of the K and V stage.
template <int X, bool kHalf, int D>
__device__ __forceinline__ void issue_s_dp(uint32_t tmem, uint32_t dq, uint32_t dg, uint32_t dk, uint32_t dv) {
  constexpr int kQBlock = kQBlockBytes >> 4, kQTile = kQTileBytes >> 4;
  constexpr int kKvBlock = kKvBlockBytes >> 4;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const uint32_t qo = (uint32_t)(X * kQTile + (ks >> 2) * kQBlock + (ks & 3) * 2);
    const uint32_t ko = (uint32_t)((ks >> 2) * kKvBlock + (ks & 3) * 2);
    mma_ss_lo<kDescHi>(tmem + X * 128, dq + qo, dk + ko, kIdescS<kHalf>, ks > 0);
  }
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const uint32_t qo = (uint32_t)(X * kQTile + (ks >> 2) * kQBlock + (ks & 3) * 2);
    const uint32_t ko = (uint32_t)((ks >> 2) * kKvBlock + (ks & 3) * 2);
    mma_ss_lo<kDescHi>(tmem + X * 128 + 64, dg + qo, dv + ko, kIdescS<kHalf>, ks > 0);
  }
}
// dQ_X (+)= dS_X . K for one 64-key tile: 4 k-steps of 16 keys, dS read from tensor memory,
// K read as the MN-major operand (`dkt`: descriptor word with the 64-dim block stride).
template <int X, bool kHalf, int D>
__device__ __forceinline__ void issue_dq(uint32_t tmem, uint32_t dkt, bool first) {
#pragma unroll
  for (int ks = 0; ks < kBN / 16; ++ks)
    mma_ts_lo<kDescHi>(tmem + 256 + X * 128, tmem + X * 128 + ks * 8,
                       dkt + ks * (2048 >> 4), kIdescDQ<kHalf, D>, (!first) || ks > 0);
}

template <bool kHalf, int D>
__global__ void __launch_bounds__(kThreads, 1)
bwd_dq_tc5_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const KernelArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);                       // Q tile A, Q tile B
  const uint32_t sG = sQ + 2 * kQTileBytes;                 // dO tile A, dO tile B
  const uint32_t sK = sG + 2 * kQTileBytes;                 // 3 stages
  const uint32_t sV = sK + kKStages * kKvTileBytes;         // 2 stages
  Ctrl& c = *reinterpret_cast<Ctrl*>(smem + 4 * kQTileBytes + (kKStages + 2) * kKvTileBytes);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kKStages; ++i) {
      mbar_init(smem_u32(&c.k_full[i]), 1);
      mbar_init(smem_u32(&c.k_empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.v_full[i]), 1);
      mbar_init(smem_u32(&c.v_empty[i]), 1);
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.ds_full[i]), kTileM);
      mbar_init(smem_u32(&c.dq_full[i]), 1);
      mbar_init(smem_u32(&c.rows_full[i]), 4 * 32);          // the copies of four warps' lanes
      mbar_init(smem_u32(&c.rows_free[i]), 1);
      mbar_init(smem_u32(&c.item_full[i]), 1);
      mbar_init(smem_u32(&c.slot_free[i]), 8);               // the row warps
    }
    c.abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&c.tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  if (p.hist > 0 && p.lists < kPrefixCache)
    for (int i = threadIdx.x; i <= (int)p.lists; i += kThreads) c.prefix_cache[i] = a.tile_prefix[i];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  const int n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
  const int n_items = n_routed + own_item_count(p.slots, p.Hq, p.C, 2 * kTileM);

  bool ok = true;                            // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  // item n: slot n & 1, phase n >> 1 of its barriers; false at the end of the queue (or after a wait gave up)
  auto take = [&](int n) { return wait(&c.item_full[n & 1], (n >> 1) & 1) && !c.done[n & 1]; };

  if (warp == 2) {
    // =============================================== describes the items
    for (int n = 0;; ++n) {
      if (n >= 2 && !wait(&c.slot_free[n & 1], ((n >> 1) - 1) & 1)) break;
      if (!describe_item(p, a, c, n & 1, n_routed, n_items)) break;
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 0) {
    // =============================================== K / V tiles, as far ahead as stages are free
    uint32_t g = 0;
    for (int n = 0; take(n); ++n) {
      const int ntiles = (c.item[n & 1].kv_len + kBN - 1) / kBN;
      const int tok0 = c.item[n & 1].kv_tok0, head = c.item[n & 1].kv_head;
      if (lane == 0)                         // one lane: requests go out a little earlier than behind a vote of the warp
        for (int j = 0; j < ntiles; ++j, ++g) {
          const int tok = tok0 + j * kBN;
          const uint32_t ks = g % kKStages, vs = g & 1;
          if (!(ok = mbar_wait(smem_u32(&c.k_empty[ks]), ((g / kKStages) & 1) ^ 1))) break;
          uint32_t bar = smem_u32(&c.k_full[ks]);
          mbar_expect_tx(bar, ((D + 63) / 64) * kKvBlockBytes);
          tma_load_3d(sK + ks * kKvTileBytes, &tmap_k, bar, 0, head, tok);
          if (D > 64) tma_load_3d(sK + ks * kKvTileBytes + kKvBlockBytes, &tmap_k, bar, 64, head, tok);
          if (!(ok = mbar_wait(smem_u32(&c.v_empty[vs]), ((g >> 1) & 1) ^ 1))) break;
          bar = smem_u32(&c.v_full[vs]);
          mbar_expect_tx(bar, ((D + 63) / 64) * kKvBlockBytes);
          tma_load_3d(sV + vs * kKvTileBytes, &tmap_v, bar, 0, head, tok);
          if (D > 64) tma_load_3d(sV + vs * kKvTileBytes + kKvBlockBytes, &tmap_v, bar, 64, head, tok);
        }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp >= 12) {
    // =============================================== Q and dO rows: a tile's as soon as the last S / dP of the
    // item before has executed, while its dQ is still being computed and written
    for (int n = 0; take(n); ++n) {
      const int slot = n & 1, nrows = c.item[slot].nrows;
      for (int x = 0; x < 2; ++x) {
        if (n > 0 && !wait(&c.rows_free[x], (n - 1) & 1)) break;
        const int rows = min(max(nrows - x * kTileM, 0), kTileM);
        copy_rows_async<D / 8, 4>(sQ + x * kQTileBytes, a.q, 0, warp - 12, rows,
                                  [&](int r) { return c.qoff[slot][x * kTileM + r]; });
        copy_rows_async<D / 8, 4>(sG + x * kQTileBytes, a.dout, 0, warp - 12, rows,
                                  [&](int r) { return (int64_t)c.grow[slot][x * kTileM + r] * D; });
        cp_async_mbar_arrive(smem_u32(&c.rows_full[x]));
      }
      if (!ok) break;
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 1) {
    // =============================================== MMA issuer: the whole warp runs convergent, one elected lane issues
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dg = __shfl_sync(0xffffffffu, desc_lo(sG, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, 16), 0);
    const uint32_t dkt = __shfl_sync(0xffffffffu, desc_lo(sK, kKvBlockBytes), 0);
    const uint32_t el = elect_one();
    constexpr uint32_t kStageDesc = kKvTileBytes >> 4;
    uint32_t g = 0;                          // key tiles whose dQ has been issued
    uint32_t pph0 = 0, pph1 = 0;             // ds_full phases of tile A / B
    // S and dP of tile x for the first step of item n, key tile `gt` of the CTA
    auto s_dp = [&](int x, int n, int ntiles, uint32_t gt) {
      if (!wait(&c.rows_full[x], n & 1)) return;
      fence_proxy_async_smem();                               // rows written by cp.async, read by the tensor core
      if (x == 0 && (!wait(&c.k_full[gt % kKStages], (gt / kKStages) & 1) || !wait(&c.v_full[gt & 1], (gt >> 1) & 1))) return;
      tc_fence_after();
      if (el) {
        const uint32_t ko = (gt % kKStages) * kStageDesc, vo = (gt & 1) * kStageDesc;
        if (x == 0) issue_s_dp<0, kHalf, D>(tm, dq, dg, dk + ko, dv + vo);
        else issue_s_dp<1, kHalf, D>(tm, dq, dg, dk + ko, dv + vo);
        tc_commit(smem_u32(&c.s_full[x]));
        if (ntiles == 1) tc_commit(smem_u32(&c.rows_free[x]));
        if (x == 1) tc_commit(smem_u32(&c.v_empty[gt & 1]));
      }
      __syncwarp();
    };
    if (take(0)) {
      int ntiles = (c.item[0].kv_len + kBN - 1) / kBN;
      s_dp(0, 0, ntiles, 0);
      if (ok) s_dp(1, 0, ntiles, 0);
      for (int n = 0; ok; ++n) {
        // All steps but the last, whose successor is of the same item.  The issue is part of the chain that a
        // step waits for, so this loop has nothing in it that depends on where the successor comes from (an item of
        // 64 steps at head dim 128 112 -> 107 us; one call site for both kinds of successor: 117).
        for (int j = 0; j + 1 < ntiles; ++j, ++g) {
          const uint32_t kcur = g % kKStages, g1 = g + 1, knxt = g1 % kKStages, vnxt = g1 & 1;
          if (!wait(&c.ds_full[0], pph0)) break;
          pph0 ^= 1;
          tc_fence_after();
          if (el) issue_dq<0, kHalf, D>(tm, dkt + kcur * kStageDesc, j == 0);
          __syncwarp();
          if (!wait(&c.k_full[knxt], (g1 / kKStages) & 1) || !wait(&c.v_full[vnxt], (g1 >> 1) & 1)) break;
          tc_fence_after();
          if (el) {
            issue_s_dp<0, kHalf, D>(tm, dq, dg, dk + knxt * kStageDesc, dv + vnxt * kStageDesc);
            tc_commit(smem_u32(&c.s_full[0]));
            if (j + 2 == ntiles) tc_commit(smem_u32(&c.rows_free[0]));
          }
          __syncwarp();
          if (!wait(&c.ds_full[1], pph1)) break;
          pph1 ^= 1;
          tc_fence_after();
          if (el) {
            issue_dq<1, kHalf, D>(tm, dkt + kcur * kStageDesc, j == 0);
            tc_commit(smem_u32(&c.k_empty[kcur]));
            issue_s_dp<1, kHalf, D>(tm, dq, dg, dk + knxt * kStageDesc, dv + vnxt * kStageDesc);
            tc_commit(smem_u32(&c.s_full[1]));
            if (j + 2 == ntiles) tc_commit(smem_u32(&c.rows_free[1]));
            tc_commit(smem_u32(&c.v_empty[vnxt]));
          }
          __syncwarp();
        }
        if (!ok) break;
        // the last step, followed by the first of the next item
        int next_tiles = 0;                  // key tiles of item n + 1 (0: there is none)
        const uint32_t kcur = g % kKStages;
        if (!wait(&c.ds_full[0], pph0)) break;
        pph0 ^= 1;
        tc_fence_after();
        if (el) {
          issue_dq<0, kHalf, D>(tm, dkt + kcur * kStageDesc, ntiles == 1);
          tc_commit(smem_u32(&c.dq_full[0]));
        }
        __syncwarp();
        if (take(n + 1)) next_tiles = (c.item[(n + 1) & 1].kv_len + kBN - 1) / kBN;
        if (!ok) break;
        if (next_tiles > 0) s_dp(0, n + 1, next_tiles, g + 1);
        if (!ok || !wait(&c.ds_full[1], pph1)) break;
        pph1 ^= 1;
        tc_fence_after();
        if (el) {
          issue_dq<1, kHalf, D>(tm, dkt + kcur * kStageDesc, ntiles == 1);
          tc_commit(smem_u32(&c.k_empty[kcur]));
          tc_commit(smem_u32(&c.dq_full[1]));
        }
        __syncwarp();
        if (next_tiles > 0) s_dp(1, n + 1, next_tiles, g + 1);
        ++g;
        if (next_tiles == 0) break;
        ntiles = next_tiles;
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else if (warp >= 4) {
    // =============================================== warps 4-11: one thread per row
    const int x = (warp - 4) >> 2;                       // 0: tile A, 1: tile B
    const int row = (warp & 3) * 32 + lane;              // row inside the tile = TMEM lane
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_base + x * 128;
    const uint32_t tDQ = tmem + lane_base + 256 + x * 128;
    const float scale = rsqrtf((float)D);
    const float sl2 = scale * 1.4426950408889634f;
    uint32_t sph = 0;                                    // s_full phase of this tile
    for (int n = 0; take(n); ++n) {
      const int slot = n & 1;
      const int32_t e = c.entry[slot][x * kTileM + row];
      const int kv_len = c.item[slot].kv_len, causal = c.item[slot].causal;
      const int rel = c.item[slot].tok0 + x * kTileM - c.item[slot].kv_tok0;   // own chunk: position of the tile's first row
      float neg_lse2 = -INFINITY, delta = 0.f;
      if (e >= 0) {
        const int32_t gr = c.grow[slot][x * kTileM + row];
        neg_lse2 = -__ldg(a.lse2 + gr);
        delta = __ldg(a.delta + gr);
      }
      const int ntiles = (kv_len + kBN - 1) / kBN;
      const int lim = causal ? min(kv_len, rel + row + 1) : kv_len;            // keys < lim are visible
      for (int j = 0; j < ntiles; ++j) {
        if (!wait(&c.s_full[x], sph)) break;
        sph ^= 1;
        // The item's S has run: every role but the other tile's row warps has read its description.  It is let go
        // four steps before the end, which is time enough to describe the item after the next; at the start of a
        // long item a CTA would draw two more ahead of CTAs that end before (8192 tokens x 8/2 heads, head_dim 128,
        // chunk 4096: 270 us, 251 this way).
        if (j == max(ntiles - 4, 0) && lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
        tc_fence_after();
        const int key0 = j * kBN;
        const bool masked = key0 + kBN > kv_len || (causal && key0 + kBN - 1 > rel);
        if (masked) ds_row<true, kHalf, (D > 64)>(tS, key0, lim, sl2, neg_lse2, delta);
        else ds_row<false, kHalf, (D > 64)>(tS, key0, lim, sl2, neg_lse2, delta);
        tc_fence_before();
        mbar_arrive(smem_u32(&c.ds_full[x]));
      }
      if (!ok || !wait(&c.dq_full[x], n & 1)) break;
      tc_fence_after();
      float* dst = a.partial_dq + (int64_t)(e >= 0 ? e : 0) * D;
#pragma unroll
      for (int ch = 0; ch < D; ch += 32) {
        uint32_t v[32];
        tmem_ld32(tDQ + ch, v);
        tmem_wait_ld();
        if (e >= 0) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint32_t o[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) o[u] = __float_as_uint(__uint_as_float(v[i + u]) * scale);
            if (a.wide_store) {
              store32(dst + ch + i, o);
            } else {
              *reinterpret_cast<uint4*>(dst + ch + i) = make_uint4(o[0], o[1], o[2], o[3]);
              *reinterpret_cast<uint4*>(dst + ch + i + 4) = make_uint4(o[4], o[5], o[6], o[7]);
            }
          }
        }
        __syncwarp();
      }
      tc_fence_before();
    }
    if (!ok) { atomicExch(a.status, ST_ROWS); c.abort = 1; }
  }
  __syncwarp();
  __syncthreads();

  // teardown: all roles are past their last wait; give in-flight copies time to land after
  // an abort, then release tensor memory
  if (c.abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------
// chunks of at most kDqShortChunk keys: one 128-row tile per work item
//
// With one chunk tile per item the kernel above spends most of an item on its hand-over (description,
// gather by the row threads, epilogue, two CTA-wide barriers).  Here the roles run through a flat stream
// of items without CTA-wide barriers, as in the forward's kernel for short items:
//   warp 0     describes the items, up to eight ahead
//   warps 2, 3 copy the Q / dO rows of an item (cp.async) into its slot (two slots, item n uses n & 1) as soon
//              as the last S / dP of item n - 2 has executed; warp 2 requests K and V of the chunk (TMA)
//              once per run of items on it
//   warp 1     issues the MMAs, the two slots in turn: dQ of a step and behind it S / dP of the slot's
//              next step, of its next item too
//   warps 4-7, 8-11  the rows of slot 0 / 1: dS of each 64-key step, then dQ from tensor memory to
//              32-byte stores, while the other slot computes
// Shared memory: Q and dO of two slots (128 KB), K and V of a chunk (64 KB).  TMEM per slot as above:
// S 64, dP 64, dQ 128 columns.
// Measured against the kernel above (as it was with its barriers), 8191 tokens x 16/4 heads, chunk 128: 328 -> 255 us.
// ---------------------------------------------------------------------------
constexpr int kSlotBytes = 2 * kQTileBytes;                   // Q tile, dO tile
constexpr int kChunkBlockBytes = kDqShortChunk * 64 * 2;      // one [128 keys][64 dims] swizzled block
constexpr int kChunkTileBytes = 2 * kChunkBlockBytes;

constexpr int kDqSlots = 8;                // item descriptions in flight (see the describing warp)

struct DqShortCtrl {
  static constexpr int kPrefix = kShortPrefix;
  uint64_t row_full[2];                      // Q and dO of the slot's item landed; once per item
  uint64_t row_free[2];                      // the last S / dP of the slot's item has executed
  uint64_t kv_full, kv_free;                 // K and V landed; every MMA that read them has executed (once per chunk followed by another)
  uint64_t s_full[2], ds_full[2], dq_full[2];
  uint64_t item_full[kDqSlots], slot_free[kDqSlots];
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;
  SlotRange own;
  ShortItem item[kDqSlots];
  alignas(16) int32_t entry[kDqSlots][kTileM];
  alignas(16) int32_t grow[kDqSlots][kTileM];    // row index t * Hq + h (dO, lse and delta are indexed by it)
  alignas(16) int64_t qoff[kDqSlots][kTileM];
  int32_t prefix_cache[kShortPrefix];
};
constexpr int kDqShortThreads = 384;
constexpr size_t kDqShortSmemBytes = 1024 + 2 * kSlotBytes + 2 * kChunkTileBytes + sizeof(DqShortCtrl);
static_assert(kDqShortSmemBytes <= 232448, "shared memory of one CTA");

struct DqShortArgs {
  KernelArgs a;
  ItemQueue iq;
};

// S_X = Q_X . K^T and dP_X = dO_X . V^T for the 64 keys at row `key0` of the chunk tiles
template <int X, bool kHalf, int D>
__device__ __forceinline__ void issue_s_dp_short(uint32_t tmem, uint32_t dq, uint32_t dk, uint32_t dv, int key0) {
  constexpr int kQBlock = kQBlockBytes >> 4, kSlot = kSlotBytes >> 4, kBlock = kChunkBlockBytes >> 4;
  const uint32_t rows = (uint32_t)(key0 * 128) >> 4;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const uint32_t qo = (uint32_t)(X * kSlot + (ks >> 2) * kQBlock + (ks & 3) * 2);
    const uint32_t ko = (uint32_t)((ks >> 2) * kBlock + (ks & 3) * 2);
    mma_ss_lo<kDescHi>(tmem + X * 128, dq + qo, dk + rows + ko, kIdescS<kHalf>, ks > 0);
  }
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    const uint32_t qo = (uint32_t)(X * kSlot + (kQTileBytes >> 4) + (ks >> 2) * kQBlock + (ks & 3) * 2);
    const uint32_t ko = (uint32_t)((ks >> 2) * kBlock + (ks & 3) * 2);
    mma_ss_lo<kDescHi>(tmem + X * 128 + 64, dq + qo, dv + rows + ko, kIdescS<kHalf>, ks > 0);
  }
}

template <bool kHalf, int D>
__global__ void __launch_bounds__(kDqShortThreads, 1)
bwd_dq_short_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const DqShortArgs sa) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);                       // slot 0: Q, dO; slot 1: Q, dO
  const uint32_t sK = sQ + 2 * kSlotBytes;
  const uint32_t sV = sK + kChunkTileBytes;
  DqShortCtrl& c = *reinterpret_cast<DqShortCtrl*>(smem + 2 * kSlotBytes + 2 * kChunkTileBytes);
  const KernelArgs& a = sa.a;
  constexpr int kNBlk = (D + 63) / 64;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.row_full[i]), 64);               // the copies of two warps' lanes
      mbar_init(smem_u32(&c.row_free[i]), 1);
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.ds_full[i]), kTileM);
      mbar_init(smem_u32(&c.dq_full[i]), 1);
    }
    mbar_init(smem_u32(&c.kv_full), 1);
    mbar_init(smem_u32(&c.kv_free), 1);
    for (int i = 0; i < kDqSlots; ++i) {
      mbar_init(smem_u32(&c.item_full[i]), 1);
      // The row warps of the item, once its first S is there.  Behind that S are the other readers of the description: the MMA
      // warp reads it in front of S, warps 2 and 3 before they arrive on row_full, which S waits for.
      mbar_init(smem_u32(&c.slot_free[i]), 4);
    }
    c.abort = 0;
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + own_item_count(c.own.n, p.Hq, p.C, kTileM);
    fence_barrier_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&c.tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kDqShortThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  bool ok = true;                            // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  if (warp == 0) {
    ok = describe_items<kDqSlots, 2, true, true>(p, sa.iq, c);
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 2 || warp == 3) {
    // ---- rows: warp 2 copies Q (and requests K and V), warp 3 dO
    uint32_t kv = 0;                         // chunks requested so far
    for (int n = 0; ok; ++n) {
      const int x = n & 1, slot = n % kDqSlots;
      if (!wait(&c.item_full[slot], (n / kDqSlots) & 1)) break;
      if (c.item[slot].done) break;
      const int tok0 = c.item[slot].tok0, head = c.item[slot].head, nrows = c.item[slot].nrows;
      const bool fresh = c.item[slot].new_kv != 0;
      if (n >= 2 && !wait(&c.row_free[x], ((n >> 1) - 1) & 1)) break;
      const uint32_t tile = sQ + x * kSlotBytes;
      if (warp == 2) copy_rows_async<D / 8, 1>(tile, a.q, 0, 0, nrows, [&](int r) { return c.qoff[slot][r]; });
      else copy_rows_async<D / 8, 1>(tile + kQTileBytes, a.dout, 0, 0, nrows, [&](int r) { return (int64_t)c.grow[slot][r] * D; });
      cp_async_mbar_arrive(smem_u32(&c.row_full[x]));
      if (warp == 2 && fresh) {
        if (kv > 0 && !wait(&c.kv_free, (kv - 1) & 1)) break;
        ++kv;
        if (lane == 0) {
          const uint32_t bar = smem_u32(&c.kv_full);
          mbar_expect_tx(bar, 2 * kNBlk * kChunkBlockBytes);
          tma_load_3d(sK, &tmap_k, bar, 0, head, tok0);
          if (D > 64) tma_load_3d(sK + kChunkBlockBytes, &tmap_k, bar, 64, head, tok0);
          tma_load_3d(sV, &tmap_v, bar, 0, head, tok0);
          if (D > 64) tma_load_3d(sV + kChunkBlockBytes, &tmap_v, bar, 64, head, tok0);
        }
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp runs convergent, one elected lane issues.
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, 16), 0);
    const uint32_t dkt = __shfl_sync(0xffffffffu, desc_lo(sK, kChunkBlockBytes), 0);
    const uint32_t el = elect_one();
    uint32_t kv = 0;                       // chunks consumed
    int next = 0;                          // the next item to start (item `next` goes to slot next & 1)
    bool end = false;
    // per slot: the key step whose dS is due and the steps of its item; 0 steps: empty
    int step0 = 0, step1 = 0, steps0 = 0, steps1 = 0;
    uint32_t dph0 = 0, dph1 = 0;           // ds_full phases
    auto s_dp = [&](int x, int step, int steps) {
      tc_fence_after();
      if (el) {
        if (x) issue_s_dp_short<1, kHalf, D>(tm, dq, dk, dv, step * kBN);
        else issue_s_dp_short<0, kHalf, D>(tm, dq, dk, dv, step * kBN);
        tc_commit(smem_u32(&c.s_full[x]));
        if (step + 1 == steps) tc_commit(smem_u32(&c.row_free[x]));
      }
      __syncwarp();
    };
    // starts item `next` in its slot, whose item before has issued its last dQ.  An item on another chunk waits
    // until the other slot has issued its last dQ too (`other_busy` false): K and V are then free.
    auto start = [&](bool other_busy) {
      if (end) return;
      const int slot = next % kDqSlots, x = next & 1;
      if (!wait(&c.item_full[slot], (next / kDqSlots) & 1)) return;
      if (c.item[slot].done) { end = true; return; }
      const bool fresh = c.item[slot].new_kv != 0;
      if (fresh) {
        if (other_busy) return;
        if (kv > 0) {
          if (el) tc_commit(smem_u32(&c.kv_free));
          __syncwarp();
        }
        if (!wait(&c.kv_full, kv & 1)) return;
        ++kv;
      }
      if (!wait(&c.row_full[x], (next >> 1) & 1)) return;
      fence_proxy_async_smem();                               // rows written by cp.async, read by the tensor core
      const int steps = (c.item[slot].kv_len + kBN - 1) / kBN;
      if (x) { steps1 = steps; step1 = 0; } else { steps0 = steps; step0 = 0; }
      s_dp(x, 0, steps);
      ++next;
    };
    start(false);
    if (ok) start(steps0 > 0);
    // slots in turn; a slot without an item starts the next one when it is that item's slot
    for (int turn = 0; ok && (steps0 > 0 || steps1 > 0); ++turn) {
      const int x = turn & 1;
      const int steps = x ? steps1 : steps0, step = x ? step1 : step0;
      if (steps > 0) {
        if (!wait(&c.ds_full[x], x ? dph1 : dph0)) break;
        if (x) dph1 ^= 1; else dph0 ^= 1;
        tc_fence_after();
        if (el) {
#pragma unroll
          for (int ks = 0; ks < kBN / 16; ++ks)
            mma_ts_lo<kDescHi>(tm + 256 + x * 128, tm + x * 128 + ks * 8, dkt + ((step * kBN + ks * 16) * 128 >> 4),
                               kIdescDQ<kHalf, D>, step > 0 || ks > 0);
          if (step + 1 == steps) tc_commit(smem_u32(&c.dq_full[x]));
        }
        __syncwarp();
        if (step + 1 < steps) {
          s_dp(x, step + 1, steps);
          if (x) ++step1; else ++step0;
        } else {
          if (x) steps1 = 0; else steps0 = 0;
        }
      }
      if (ok && (x ? steps1 : steps0) == 0 && (next & 1) == x) start((x ? steps0 : steps1) > 0);
      // the other slot may have been waiting for this one to let go of K and V
      if (ok && steps0 == 0 && steps1 == 0) start(false);
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else {
    // ---- one thread per row; warps 4-7: slot 0, 8-11: slot 1
    const int x = (warp - 4) >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_base + x * 128;
    const uint32_t tDQ = tmem + lane_base + 256 + x * 128;
    const float scale = rsqrtf((float)D);
    const float sl2 = scale * 1.4426950408889634f;
    uint32_t sph = 0;
    for (int n = x; ok; n += 2) {
      const int slot = n % kDqSlots;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.item_full[slot]), (n / kDqSlots) & 1));
      if (!ok) break;
      const ShortItem it = c.item[slot];
      if (it.done) break;
      const int32_t e = c.entry[slot][row];
      const bool active = (warp & 3) * 32 < it.nrows;
      float neg_lse2 = -INFINITY, delta = 0.f;
      if (e >= 0) {
        const int32_t gr = c.grow[slot][row];
        neg_lse2 = -__ldg(a.lse2 + gr);
        delta = __ldg(a.delta + gr);
      }
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      const int lim = it.causal ? min(it.kv_len, it.tok_rel + row + 1) : it.kv_len;   // keys < lim are visible
      for (int j = 0; j < ntiles; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.s_full[x]), sph));
        if (!ok) break;
        sph ^= 1;
        // the item's S has run: every role has read its description
        if (j == 0 && lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
        if (active) {
          tc_fence_after();
          const int key0 = j * kBN;
          const bool masked = key0 + kBN > it.kv_len || (it.causal && key0 + kBN - 1 > it.tok_rel);
          if (masked) ds_row<true, kHalf, false>(tS, key0, lim, sl2, neg_lse2, delta);
          else ds_row<false, kHalf, false>(tS, key0, lim, sl2, neg_lse2, delta);
          tc_fence_before();
        }
        mbar_arrive(smem_u32(&c.ds_full[x]));
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.dq_full[x]), (n >> 1) & 1));
      if (!ok) break;
      if (active) {
        tc_fence_after();
        float* dst = a.partial_dq + (int64_t)(e >= 0 ? e : 0) * D;
#pragma unroll 1
        for (int ch = 0; ch < D; ch += 32) {
          uint32_t v[32];
          tmem_ld32(tDQ + ch, v);
          tmem_wait_ld();
          if (e >= 0) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint32_t o[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) o[u] = __float_as_uint(__uint_as_float(v[i + u]) * scale);
              if (a.wide_store) {
                store32(dst + ch + i, o);
              } else {
                *reinterpret_cast<uint4*>(dst + ch + i) = make_uint4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<uint4*>(dst + ch + i + 4) = make_uint4(o[4], o[5], o[6], o[7]);
              }
            }
          }
          __syncwarp();
        }
        tc_fence_before();
      }
    }
    if (!ok) {
      atomicExch(a.status, ST_ROWS);
      c.abort = 1;
    }
  }

  __syncwarp();
  __syncthreads();
  if (c.abort) {                           // copies in flight land before shared memory is given up
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

}  // namespace

cudaError_t launch_bwd_dq_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                              const __nv_bfloat16* v, const __nv_bfloat16* dout, const int32_t* cu,
                              const int32_t* list_counts, const int32_t* list_offsets, const int32_t* tile_prefix,
                              const int32_t* row_list, const float* lse2, const float* delta, float* partial_dq,
                              int32_t* work_counter, int32_t* status, cudaStream_t st) {
  if (p.D != 64 && p.D != 96 && p.D != 128) return cudaErrorInvalidValue;
  CUtensorMap mk, mv;
  if (!make_kv_map(&mk, p.fp16 != 0, p.D, k, p.T, p.Hkv, p.sk_t, p.sk_h, kBN) ||
      !make_kv_map(&mv, p.fp16 != 0, p.D, v, p.T, p.Hkv, p.sv_t, p.sv_h, kBN))
    return cudaErrorNotSupported;
  const int sms = device_info().sms;
  const KernelArgs args{q, dout, cu, list_counts, list_offsets, tile_prefix, row_list, lse2, delta, partial_dq,
                        work_counter, status, ((uintptr_t)partial_dq & 31) == 0};
  if (bwd_dq_short_items(p)) {
    DqShortArgs sa;
    sa.a = args;
    sa.iq = item_queue(p, cu, list_counts, list_offsets, tile_prefix, row_list, work_counter, short_batch(p, sms, false), false, 0);
    if (!make_kv_map(&mk, p.fp16 != 0, p.D, k, p.T, p.Hkv, p.sk_t, p.sk_h, kDqShortChunk) ||
        !make_kv_map(&mv, p.fp16 != 0, p.D, v, p.T, p.Hkv, p.sv_t, p.sv_h, kDqShortChunk))
      return cudaErrorNotSupported;
    auto kern = p.D == 128 ? (p.fp16 ? bwd_dq_short_kernel<true, 128> : bwd_dq_short_kernel<false, 128>)
              : p.D == 96  ? (p.fp16 ? bwd_dq_short_kernel<true, 96> : bwd_dq_short_kernel<false, 96>)
                           : (p.fp16 ? bwd_dq_short_kernel<true, 64> : bwd_dq_short_kernel<false, 64>);
    const cudaError_t se = prepare_kernel(kern, kDqShortSmemBytes);
    if (se != cudaSuccess) return se;
    kern<<<sms, kDqShortThreads, kDqShortSmemBytes, st>>>(p, mk, mv, sa);
    return cudaGetLastError();
  }
  auto kernel = p.D == 128 ? (p.fp16 ? bwd_dq_tc5_kernel<true, 128> : bwd_dq_tc5_kernel<false, 128>)
              : p.D == 96  ? (p.fp16 ? bwd_dq_tc5_kernel<true, 96> : bwd_dq_tc5_kernel<false, 96>)
                           : (p.fp16 ? bwd_dq_tc5_kernel<true, 64> : bwd_dq_tc5_kernel<false, 64>);
  cudaError_t e = prepare_kernel(kernel, kSmemBytes);
  if (e != cudaSuccess) return e;
  kernel<<<sms, kThreads, kSmemBytes, st>>>(p, mk, mv, args);
  return cudaGetLastError();
}

}  // namespace moba
