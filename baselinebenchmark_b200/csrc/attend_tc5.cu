// Dense stage of MoBA on the Blackwell tensor path: block-sparse flash-attention
// forward with tcgen05.mma, accumulators in tensor memory (TMEM) and K/V tiles
// staged by TMA.
//
// Replaces, for the inference path of the reference,
//   _varlen_attn_fwd_kernel        backends/_mthreads/ops/moba/attention.py:53-160  (own chunk, causal)
//   native_moba.routed / MATE FMHA backends/_mthreads/ops/moba/native_moba.py:120-135
//   _routed_gqa_attn_fwd_kernel    attention.py:610-707                           (selected chunks)
// Templated on the element type (bf16, fp16) and the head dim (64, 96, 128); buffer
// strides in shared memory and TMEM are those of head dim 128.  At head dim 96 the second
// 64-dim block of a K / V tile is half filled (TMA fills dims 96-127 with zeros), Q.K^T runs
// six 16-dim steps and P.V writes 96 accumulator columns.
// Numerics follow attention.py:116-155 (fp32 scores * D^-0.5 * log2 e, P rounded
// to the input dtype before P.V, fp32 accumulation, natural-log LSE); the running maximum is
// only refreshed when it grows by more than 8 (factor 256), which changes the
// rounding pattern but not the value of the softmax.
//
// Work item = up to 256 query rows (two 128-row MMA tiles, "A" and "B") against
// the keys of one chunk.  Routed items gather their rows through row_list (the
// rows of all query heads of a GQA group share the K/V stream of their kv
// head); own-chunk items are 256 consecutive tokens of one head with a causal
// mask.  CTAs are persistent (one per SM) and draw items from a global counter.
//
// Warp roles (384 threads):
//   warp 0      TMA producer: K and V tiles of 128 keys, two stages each
//   warp 2      draws, decodes and resolves the next work item while the current one runs
//   warp 1      MMA issuer: S = Q.K^T into TMEM, O += P.V with P read from TMEM; the
//               warp runs convergent, one elected lane issues; owns the TMEM allocation
//   warps 4-7   softmax of tile A: one thread per row (TMEM lane)
//   warps 8-11  softmax of tile B
//   warps 4-11  also gather the Q rows into 128B-swizzled shared memory at the item start
// TMEM columns: S_A 0-127, S_B 128-255, O_A 256-383, O_B 384-511; the 16-bit P
// tile overwrites the first 64 columns of its S tile.
// The tensor core alternates  QK_A(j+1) | PV_B(j) | QK_B(j+1) | PV_A(j+1) ...
// so that the softmax of one tile runs while the MMAs of the other execute.
#include <mutex>

#include "attend_rows.cuh"
#include "common.cuh"
#include "short_items.cuh"
#include "sm100_ptx.cuh"

namespace moba {

namespace {

using namespace ptx;

constexpr int kThreads = 384;
constexpr uint32_t kTmemCols = 512;

constexpr int kPrefixCache = 6144;       // ints of tile_prefix kept in shared memory (24 KB)

struct Ctrl {
  static constexpr int kPrefix = kPrefixCache;
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t s_full[2], p_full[2], o_full[2];
  uint64_t item_ready[2];                  // slot filled by the prefetch warp (phase = fill count)
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;               // work items of the launch (routed tiles first), set by thread 0
  SlotRange own;                           // slots the own-chunk items run over
  // Work items are drawn and resolved one item ahead by a spare warp: slot (n & 1)
  // holds item n, its output entries and the offsets of its Q rows.
  Item item[2];
  int32_t done[2];
  int64_t qoff[2][2 * kTileM];
  int32_t entry[2][2 * kTileM];
  // tile_prefix sampled once per CTA (whole when it fits): decoding an item searches it, and with
  // short items (small chunks) eleven dependent global loads per item were the critical path
  int32_t prefix_cache[kPrefixCache];
  float row_inv[kTileM];                   // head dim 256: the row's factor (scale / row sum), handed to the warps that write the second half of O
};

constexpr size_t kSmemBytes = 1024 /*alignment slack*/ + 6 * kTileBytes + sizeof(Ctrl);

// Runs in one spare warp while the other warps work on the current item: draws the
// next item from the global queue (skipping empty own-chunk tiles), decodes it and
// resolves its rows (output entry and Q row offset) into prefetch slot `slot`.
template <int kItemRows, typename CtrlT>
__device__ __forceinline__ void prefetch_item(const Params& p, const KernelArgs& a, CtrlT& c, int slot) {
  const int lane = threadIdx.x & 31;
  const int n_routed = c.n_routed, n_items = c.n_items;
  const SlotRange own = c.own;
  Item it;
  it.valid = 0;
  int done = 0;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = c.abort ? 0x7fffffff : atomicAdd(a.work_counter, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= n_items) { done = 1; break; }
    it = decode_item(p, idx, n_routed, kItemRows, a.cu, a.list_counts, a.list_offsets, a.tile_prefix,
                     idx < n_routed ? find_list(c, a.tile_prefix, p.lists, idx) : 0, own);
    if (it.valid) break;
  }
  if (lane == 0) { c.item[slot] = it; c.done[slot] = done; }
  if (!done) {
    // the rows of a lane: all row_list loads in flight before any of them is used
    int32_t ent[kItemRows / 32];
#pragma unroll
    for (int u = 0; u < kItemRows / 32; ++u) {
      const int r = lane + 32 * u;
      ent[u] = -1;
      if (r < it.nrows) {
        if (!it.causal) ent[u] = __ldg(a.row_list + it.row_start + r);
        else if (r >= it.row_start)                            // rows before the query window stay absent
          ent[u] = (int32_t)(((int64_t)(it.tok0 - p.win_lo + r) * p.Hq + it.head) * p.NP);
      }
    }
#pragma unroll
    for (int u = 0; u < kItemRows / 32; ++u) {
      const int r = lane + 32 * u;
      const int32_t e = ent[u];
      int64_t off = 0;
      if (e >= 0) {
        // entries and rows fit 32 bits (checked on the host): unsigned 32-bit divisions, not the
        // 64-bit ones, which are a subroutine of a hundred instructions each
        const uint32_t row = (uint32_t)e / (uint32_t)p.NP;
        const uint32_t t = row / (uint32_t)p.Hq;
        off = (int64_t)t * p.sq_t + (int64_t)(row - t * (uint32_t)p.Hq) * p.sq_h;
      }
      c.entry[slot][r] = e;
      c.qoff[slot][r] = off;
      if (e >= 0) {                                            // the gather of the next item then hits L2
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.q + off));
        if (p.D > 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.q + off + 64));
        if (p.D > 128) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a.q + off + 128));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a.q + off + 192));
        }
      }
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&c.item_ready[slot]));   // the producer may look at the slot now
}

// Common head of an item, executed by all 384 threads: take the prefetched item
// of slot `slot`; the softmax warps (kGather) gather its Q rows into the two swizzled Q tiles.  Returns
// false when the queue is empty (or the kernel is aborting).
template <bool kGather, int D, int kItemRows = 2 * kTileM>
__device__ __forceinline__ bool next_item(const KernelArgs& a, Ctrl& c, unsigned char* smem, int slot, Item& it) {
  __syncthreads();                         // every role has finished the previous item; slot is filled
  if (c.done[slot]) return false;
  it = c.item[slot];
  const int32_t* entry = c.entry[slot];
  const int64_t* qoff = c.qoff[slot];
  // gather Q rows into two tiles of D/64 [128][64] blocks with the 128-byte swizzle TMA would
  // produce; the 256 softmax threads do it, each with its D/8 loads in flight at once
  if (kGather) {
    constexpr int kChunks = D / 8;                  // 16-byte pieces of a row
    constexpr int kPieces = kItemRows * kChunks / 256;   // pieces per thread
    const int t = threadIdx.x - 128;
    uint4 val[kPieces];
#pragma unroll
    for (int u = 0; u < kPieces; ++u) {
      const int i = t + u * 256;
      const int r = i / kChunks, ch = i % kChunks;
      val[u] = make_uint4(0, 0, 0, 0);
      if (entry[r] >= 0) val[u] = __ldg(reinterpret_cast<const uint4*>(a.q + qoff[r] + ch * 8));
    }
#pragma unroll
    for (int u = 0; u < kPieces; ++u) {
      const int i = t + u * 256;
      const int r = i / kChunks, ch = i % kChunks;
      const uint32_t dst = (uint32_t)((r >> 7) * kTileBytes + (ch >> 3) * kHalfBytes + (r & 127) * 128 +
                                      (((ch & 7) ^ (r & 7)) << 4));
      *reinterpret_cast<uint4*>(smem + dst) = val[u];
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  return true;
}

// One softmax step of one row: S (128 fp32 columns of this thread's TMEM lane)
// -> P (bf16, written over the first 64 columns), running max / sum updated.
// `before_rescale` runs (warp-uniformly) before the accumulator O is rescaled: a kernel whose
// previous P.V may still be executing at that point waits for it there.
template <bool kMasked, bool kHalf, int D, typename F>
__device__ __forceinline__ void softmax_row(uint32_t tS, uint32_t tO, int j, int key0, int lim, float sl2,
                                            float& m_ref, float& l, F&& before_rescale) {
  uint32_t v[128];
  tmem_ld128(tS, v);
  tmem_wait_ld();
  if (kMasked) {
#pragma unroll
    for (int i = 0; i < 128; ++i) v[i] = (key0 + i < lim) ? v[i] : 0xff800000u;   // -inf
  }
  float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
  for (int i = 0; i < 128; i += 8) {
    mx0 = max3(mx0, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
    mx1 = max3(mx1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
    mx2 = max3(mx2, __uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
    mx3 = max3(mx3, __uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
  }
  const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
  const float m_new = fmaxf(m_ref, mx * sl2);
  // a row's reference moves only when the row itself asks for it: its result does not depend on
  // the rows it shares a warp with
  const bool up = m_new > m_ref + 8.f;
  if (__any_sync(0xffffffffu, up)) {
    const float alpha = up ? ex2_approx(m_ref - m_new) : 1.f;
    if (j > 0) {
      before_rescale();
      uint32_t o[32];
#pragma unroll
      for (int ch = 0; ch < D / 32; ++ch) {
        tmem_ld32(tO + ch * 32, o);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
        tmem_st32(tO + ch * 32, o);
      }
    }
    l *= alpha;
    if (up) m_ref = m_new;
  }
  const uint64_t scale2 = pack2(sl2, sl2);
  const uint64_t negm2 = pack2(-m_ref, -m_ref);
  uint64_t sum_a = 0, sum_b = 0;           // two packed accumulators = four running sums
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int e = ch * 32 + 2 * i;
      const uint64_t x = fma2(pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), scale2, negm2);
      uint64_t pr;
      if ((i & 7) < kPolyPairs) {
        pr = ex2_poly2(x);
      } else {
        pr = pack2(ex2_approx(lo2(x)), ex2_approx(hi2(x)));
      }
      if (i & 1) sum_b = add2(sum_b, pr); else sum_a = add2(sum_a, pr);
      pk[i] = pack2_16<kHalf>(lo2(pr), hi2(pr));
    }
    tmem_st16(tS + ch * 16, pk);
  }
  const uint64_t sum = add2(sum_a, sum_b);
  l += lo2(sum) + hi2(sum);
  tmem_wait_st();
}

// S_X = Q_X . K^T for one K tile: 8 k-steps of 16 dims; X and STAGE are compile-time
// so every descriptor is the base word plus an immediate.
template <int X, int STAGE, bool kHalf, int D>
__device__ __forceinline__ void issue_qk(uint32_t tmem, uint32_t dq, uint32_t dk) {
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    constexpr int kBlock = kHalfBytes >> 4, kTile = kTileBytes >> 4;
    const uint32_t koff = (uint32_t)((ks >> 2) * kBlock + (ks & 3) * 2);
    mma_ss(tmem + X * kBN, desc64(dq + X * kTile + koff), desc64(dk + STAGE * kTile + koff), kIdescQK<kHalf>, ks > 0);
  }
}
// O_X (+)= P_X . V for one V tile: 8 k-steps of 16 keys, P read from tensor memory.
template <int X, int STAGE, bool kHalf, int D>
__device__ __forceinline__ void issue_pv(uint32_t tmem, uint32_t dv, bool first) {
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    mma_ts(tmem + 256 + X * 128, tmem + X * kBN + ks * 8,
           desc64(dv + STAGE * (kTileBytes >> 4) + ks * (2048 >> 4)), kIdescPV<kHalf, D>, (!first) || ks > 0);
}

template <bool kHalf, int D>
__global__ void __launch_bounds__(kThreads, 1)
attend_tc5_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const KernelArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);                       // tile A, tile B
  const uint32_t sK = sQ + 2 * kTileBytes;                  // 2 stages
  const uint32_t sV = sK + 2 * kTileBytes;                  // 2 stages
  Ctrl& c = *reinterpret_cast<Ctrl*>(smem + 6 * kTileBytes);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp index, uniform

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.k_full[i]), 1);
      mbar_init(smem_u32(&c.k_empty[i]), 1);
      mbar_init(smem_u32(&c.v_full[i]), 1);
      mbar_init(smem_u32(&c.v_empty[i]), 1);
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.p_full[i]), kTileM);
      mbar_init(smem_u32(&c.o_full[i]), 1);
      mbar_init(smem_u32(&c.item_ready[i]), 1);
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
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + own_item_count(c.own.n, p.Hq, p.C, 2 * kTileM);
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;
  Item it;

  if (warp < 4) {
    // =============================================== warps 0-3: TMA producer, MMA issuer, two spare warps
    setmaxnreg_dec<72>();
    uint32_t kc = 0, vc = 0;               // K / V tiles produced (warp 0) or consumed (warp 1) so far
    uint32_t pph0 = 0, pph1 = 0;           // p_full phases of tile A / B
    int pre = 0;                           // producer: tiles of the coming item already requested
    // warp-uniform copies of the TMEM base and of the low words of the shared-memory
    // descriptors of the first Q / K / V block (every other block or k-step is a
    // compile-time offset from these), and the lane that issues
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    for (int n = 0;; ++n) {
      // warp 2 runs one item ahead: it fills slot n & 1 while the others still work on item n - 1
      if (warp == 2) prefetch_item<2 * kTileM>(p, a, c, n & 1);
      if (!next_item<false, D>(a, c, smem, n & 1, it)) break;
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      if (warp == 0 && lane == 0) {
        // K and V tile `j` of item `w` into the next free stages; false after a timeout
        auto load_tile = [&](const Item& w, int j) -> bool {
          const int tok = w.kv_tok0 + j * kBN;
          {
            const uint32_t s = kc & 1;
            if (!mbar_wait(smem_u32(&c.k_empty[s]), ((kc >> 1) & 1) ^ 1)) return false;
            const uint32_t bar = smem_u32(&c.k_full[s]);
            mbar_expect_tx(bar, ((D + 63) / 64) * kHalfBytes);
            tma_load_3d(sK + s * kTileBytes, &tmap_k, bar, 0, w.kv_head, tok);
            if (D > 64) tma_load_3d(sK + s * kTileBytes + kHalfBytes, &tmap_k, bar, 64, w.kv_head, tok);
            ++kc;
          }
          {
            const uint32_t s = vc & 1;
            if (!mbar_wait(smem_u32(&c.v_empty[s]), ((vc >> 1) & 1) ^ 1)) return false;
            const uint32_t bar = smem_u32(&c.v_full[s]);
            mbar_expect_tx(bar, ((D + 63) / 64) * kHalfBytes);
            tma_load_3d(sV + s * kTileBytes, &tmap_v, bar, 0, w.kv_head, tok);
            if (D > 64) tma_load_3d(sV + s * kTileBytes + kHalfBytes, &tmap_v, bar, 64, w.kv_head, tok);
            ++vc;
          }
          return true;
        };
        bool alive = true;
        for (int j = pre; alive && j < ntiles; ++j) alive = load_tile(it, j);
        pre = 0;
        // The first tiles of the next item are requested as soon as stages free up, while the
        // tail of this item still computes: the prefetch warp has the next item ready by then.
        if (alive) {
          const int s1 = (n + 1) & 1;
          alive = mbar_wait(smem_u32(&c.item_ready[s1]), ((n + 1) >> 1) & 1);
          if (alive && !c.done[s1]) {
            const Item nx = c.item[s1];
            const int nt = min(2, (nx.kv_len + kBN - 1) / kBN);
            for (; alive && pre < nt; ++pre) alive = load_tile(nx, pre);
          }
        }
        if (!alive) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
      } else if (warp == 1) {
        // MMA issuer.  The whole warp runs this code so that addresses and descriptors
        // stay warp-uniform (uniform registers); one elected lane executes the
        // tcgen05 instructions.  Issued from a single-lane branch instead, every MMA
        // costs a dozen dependent vector instructions and the issuer starves for
        // issue slots next to the softmax warps of its scheduler partition.
        bool ok = true;
        tc_fence_after();
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.k_full[kc & 1]), (kc >> 1) & 1));
        if (ok) {
          tc_fence_after();
          if (el) {
            if (kc & 1) { issue_qk<0, 1, kHalf, D>(tm, dq, dk); tc_commit(smem_u32(&c.s_full[0])); issue_qk<1, 1, kHalf, D>(tm, dq, dk); }
            else        { issue_qk<0, 0, kHalf, D>(tm, dq, dk); tc_commit(smem_u32(&c.s_full[0])); issue_qk<1, 0, kHalf, D>(tm, dq, dk); }
            tc_commit(smem_u32(&c.s_full[1]));
            tc_commit(smem_u32(&c.k_empty[kc & 1]));
          }
          __syncwarp();
          ++kc;
        }
        // K tile j+1 and V tile j always sit in opposite stages (kc == vc + 1 here)
        for (int j = 0; ok && j < ntiles; ++j) {
          const bool more = j + 1 < ntiles;
          const uint32_t vs = vc & 1, ks = vs ^ 1;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.v_full[vs]), (vc >> 1) & 1));
          if (!ok) break;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.p_full[0]), pph0));
          if (!ok) break;
          pph0 ^= 1;
          tc_fence_after();
          if (el) { if (vs) issue_pv<0, 1, kHalf, D>(tm, dv, j == 0); else issue_pv<0, 0, kHalf, D>(tm, dv, j == 0); }
          __syncwarp();
          if (more) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.k_full[ks]), (kc >> 1) & 1));
            if (!ok) break;
            tc_fence_after();
            if (el) {
              if (ks) issue_qk<0, 1, kHalf, D>(tm, dq, dk); else issue_qk<0, 0, kHalf, D>(tm, dq, dk);
              tc_commit(smem_u32(&c.s_full[0]));
            }
          } else if (el) {
            tc_commit(smem_u32(&c.o_full[0]));
          }
          __syncwarp();
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.p_full[1]), pph1));
          if (!ok) break;
          pph1 ^= 1;
          tc_fence_after();
          if (el) {
            if (vs) issue_pv<1, 1, kHalf, D>(tm, dv, j == 0); else issue_pv<1, 0, kHalf, D>(tm, dv, j == 0);
            tc_commit(smem_u32(&c.v_empty[vs]));
            if (more) {
              if (ks) issue_qk<1, 1, kHalf, D>(tm, dq, dk); else issue_qk<1, 0, kHalf, D>(tm, dq, dk);
              tc_commit(smem_u32(&c.s_full[1]));
              tc_commit(smem_u32(&c.k_empty[ks]));
            } else {
              tc_commit(smem_u32(&c.o_full[1]));
            }
          }
          __syncwarp();
          ++vc;
          if (more) ++kc;
        }
        if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
      }
      __syncwarp();
    }
  } else {
    // =============================================== warps 4-11: softmax + epilogue, one thread per row
    setmaxnreg_inc<216>();
    const int x = (warp - 4) >> 2;                       // 0: tile A, 1: tile B
    const int row = (warp & 3) * 32 + lane;              // row inside the tile = TMEM lane
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + lane_base + x * kBN;
    const uint32_t tO = tmem + lane_base + 256 + x * 128;
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    uint32_t sph = 0, oph = 0;                           // s_full / o_full phases of this tile
    for (int n = 0; next_item<true, D>(a, c, smem, n & 1, it); ++n) {
      const int32_t* entries = c.entry[n & 1];
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      const int qpos = it.tok0 + x * kTileM + row;
      const int lim = it.causal ? min(it.kv_len, qpos - it.kv_tok0 + 1) : it.kv_len;   // keys < lim are visible
      float m_ref = -INFINITY, l = 0.f;
      bool ok = true;
      for (int j = 0; ok && j < ntiles; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.s_full[x]), sph));   // warp-uniform exit
        if (!ok) break;
        sph ^= 1;
        tc_fence_after();
        const int key0 = j * kBN;
        const bool masked = key0 + kBN > it.kv_len ||
                            (it.causal && it.kv_tok0 + key0 + kBN - 1 > it.tok0 + x * kTileM);
        // S of the next step is only computed after this tile's P.V: O is quiet here
        if (masked) softmax_row<true, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, [] {});
        else softmax_row<false, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, [] {});
        tc_fence_before();
        mbar_arrive(smem_u32(&c.p_full[x]));
      }
      if (ok) ok = mbar_wait(smem_u32(&c.o_full[x]), oph);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        oph ^= 1;
        tc_fence_after();
        const int32_t e = entries[x * kTileM + row];
        // the row's largest magnitude decides the power of two its fp16 copy is scaled by
        uint32_t v0[32], v1[32];
        float amax = 0.f;
#pragma unroll
        for (int ch = 0; ch < D / 32; ++ch) {
          tmem_ld32(tO + ch * 32, v0);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            amax = max3(amax, fabsf(__uint_as_float(v0[i])), fabsf(__uint_as_float(v0[i + 1])));
        }
        const float inv = 1.f / l;
        const PartialScale ps = partial_scale(amax * inv);
        const float mul = inv * ps.scale;
        // O rows go through this warp's 8 KB of the (now idle) Q tile so that every global
        // store instruction writes whole 128-byte pieces of four rows: 64 columns at a
        // time, rows 144 bytes apart in shared memory (conflict-free both ways).
        unsigned char* stage = smem + x * kTileBytes + (warp & 3) * 8192;
#pragma unroll
        for (int ch = 0; ch < (D + 63) / 64; ++ch) {
          constexpr int kLast = D % 64 == 0 ? 64 : D % 64;      // columns of the last piece (head dim 96: 32)
          const int cols = ch == (D + 63) / 64 - 1 ? kLast : 64;
          tmem_ld32(tO + ch * 64, v0);
          if (cols > 32) tmem_ld32(tO + ch * 64 + 32, v1);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (i * 8 < cols) {
              const uint32_t* s8 = i < 4 ? v0 + 8 * i : v1 + 8 * (i - 4);
              *reinterpret_cast<uint4*>(stage + lane * 144 + i * 16) =
                  make_uint4(pack2_half(__uint_as_float(s8[0]) * mul, __uint_as_float(s8[1]) * mul),
                             pack2_half(__uint_as_float(s8[2]) * mul, __uint_as_float(s8[3]) * mul),
                             pack2_half(__uint_as_float(s8[4]) * mul, __uint_as_float(s8[5]) * mul),
                             pack2_half(__uint_as_float(s8[6]) * mul, __uint_as_float(s8[7]) * mul));
            }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rl = i * 4 + (lane >> 3), c16 = lane & 7;
            const int32_t er = __shfl_sync(0xffffffffu, e, rl);
            const uint4 val = *reinterpret_cast<const uint4*>(stage + rl * 144 + c16 * 16);
            if (er >= 0 && c16 * 8 < cols)
              __stcs(reinterpret_cast<uint4*>(a.partial_out + (int64_t)er * D + ch * 64 + c16 * 8), val);
          }
          __syncwarp();
        }
        if (e >= 0) a.partial_lse[e] = make_float2((m_ref + log2f(l)) * 0.6931471805599453f, ps.inv);
        tc_fence_before();
      } else {
        atomicExch(a.status, ST_SOFTMAX);
        c.abort = 1;
      }
    }
  }

  // teardown: all roles are past their last wait; give in-flight copies time to
  // land after an abort, then release tensor memory
  if (c.abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------
// head dim 256, chunks of more than kSmallChunk keys
//
// One 128-row tile per work item.  Operands keep the shapes of the kernel above: Q, K and V are
// handled as two 128-dim halves ("lo", "hi"); S = Q_lo.K_lo^T + Q_hi.K_hi^T (16 k-steps into one
// accumulator), O_lo += P.V_lo and O_hi += P.V_hi (two 128-column accumulators).
// TMEM columns: S buffers 0-127 and 128-255 (tile g of the CTA uses buffer g & 1), O 256-511.
// Shared memory: Q 64 KB (lo, hi), the K halves in two 32 KB slots, the V halves in two.
// With S double-buffered Q.K^T of tile j+1 runs while the softmax of tile j does.  Per tile the
// tensor core has 2048 cycles of MMAs against about 1700 of softmax, so one softmax warpgroup
// keeps it busy.  Order on the tensor core: QK(0) QK(1) PV(0) QK(2) PV(1) ...; the producer
// requests K and V in that order.  The P.V of a tile may still be executing when the softmax
// of the next tile wants to rescale O: that (rare) path waits for it first.
// Warps 8-11 take no part in the softmax: they gather Q rows and write the hi half of O.
// ---------------------------------------------------------------------------
template <int SB, int H, bool kHalf>
__device__ __forceinline__ void issue_qk_wide(uint32_t tmem, uint32_t dq, uint32_t dk) {
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    constexpr int kBlock = kHalfBytes >> 4, kTile = kTileBytes >> 4;
    const uint32_t koff = (uint32_t)(H * kTile + (ks >> 2) * kBlock + (ks & 3) * 2);
    mma_ss(tmem + SB * kBN, desc64(dq + koff), desc64(dk + koff), kIdescQK<kHalf>, (H | ks) > 0);
  }
}
template <int SB, int H, bool kHalf>
__device__ __forceinline__ void issue_pv_wide(uint32_t tmem, uint32_t dv, bool first) {
#pragma unroll
  for (int ks = 0; ks < 8; ++ks)
    mma_ts(tmem + 256 + H * 128, tmem + SB * kBN + ks * 8,
           desc64(dv + H * (kTileBytes >> 4) + ks * (2048 >> 4)), kIdescPV<kHalf, 128>, (!first) || ks > 0);
}

__device__ __forceinline__ void bar_sync_256() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

template <bool kHalf>
__global__ void __launch_bounds__(kThreads, 1)
attend_tc5_wide_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const KernelArgs a) {
  constexpr int D = 256;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);                       // lo, hi
  const uint32_t sK = sQ + 2 * kTileBytes;                  // lo, hi
  const uint32_t sV = sK + 2 * kTileBytes;                  // lo, hi
  Ctrl& c = *reinterpret_cast<Ctrl*>(smem + 6 * kTileBytes);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.k_full[i]), 1);
      mbar_init(smem_u32(&c.k_empty[i]), 1);
      mbar_init(smem_u32(&c.v_full[i]), 1);
      mbar_init(smem_u32(&c.v_empty[i]), 1);
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.p_full[i]), kTileM);
      mbar_init(smem_u32(&c.o_full[i]), 1);
      mbar_init(smem_u32(&c.item_ready[i]), 1);
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
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + own_item_count(c.own.n, p.Hq, p.C, kTileM);
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;
  Item it;
  // c.o_full[0] completes once per tile, when its P.V has executed; "tile g" counts the CTA's tiles

  if (warp < 4) {
    setmaxnreg_dec<72>();
    uint32_t kt = 0, vt = 0;               // K / V tiles produced (warp 0) or consumed (warp 1) so far
    uint32_t g = 0, gp = 0;                // tiles whose Q.K^T / P.V has been issued (warp 1)
    bool pre_k0 = false, pre_v0 = false;   // producer: K(0) / V(0) of the coming item already requested
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    for (int n = 0;; ++n) {
      if (warp == 2) prefetch_item<kTileM>(p, a, c, n & 1);
      if (!next_item<false, D, kTileM>(a, c, smem, n & 1, it)) break;
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      if (warp == 0 && lane == 0) {
        // both halves of K (V) tile `j` of item `w`, each into its slot; false after a timeout
        auto load_k = [&](const Item& w, int j) -> bool {
          const int tok = w.kv_tok0 + j * kBN;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!mbar_wait(smem_u32(&c.k_empty[h]), (kt & 1) ^ 1)) return false;
            const uint32_t bar = smem_u32(&c.k_full[h]);
            mbar_expect_tx(bar, kTileBytes);
            tma_load_3d(sK + h * kTileBytes, &tmap_k, bar, h * 128, w.kv_head, tok);
            tma_load_3d(sK + h * kTileBytes + kHalfBytes, &tmap_k, bar, h * 128 + 64, w.kv_head, tok);
          }
          ++kt;
          return true;
        };
        auto load_v = [&](const Item& w, int j) -> bool {
          const int tok = w.kv_tok0 + j * kBN;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!mbar_wait(smem_u32(&c.v_empty[h]), (vt & 1) ^ 1)) return false;
            const uint32_t bar = smem_u32(&c.v_full[h]);
            mbar_expect_tx(bar, kTileBytes);
            tma_load_3d(sV + h * kTileBytes, &tmap_v, bar, h * 128, w.kv_head, tok);
            tma_load_3d(sV + h * kTileBytes + kHalfBytes, &tmap_v, bar, h * 128 + 64, w.kv_head, tok);
          }
          ++vt;
          return true;
        };
        // in the order the tensor core consumes them: K(0), then K(j + 1), V(j) for every tile j
        bool alive = pre_k0 ? true : load_k(it, 0);
        for (int j = 0; alive && j < ntiles; ++j) {
          if (j + 1 < ntiles) alive = load_k(it, j + 1);
          if (alive && !(j == 0 && pre_v0)) alive = load_v(it, j);
        }
        pre_k0 = pre_v0 = false;
        // K(0) and V(0) of the next item go into the slots the tail of this item frees (K(1)
        // would need a slot that only the next item's own first MMAs free: not before it starts)
        if (alive) {
          const int s1 = (n + 1) & 1;
          alive = mbar_wait(smem_u32(&c.item_ready[s1]), ((n + 1) >> 1) & 1);
          if (alive && !c.done[s1]) {
            const Item nx = c.item[s1];
            alive = load_k(nx, 0);
            pre_k0 = alive;
            if (alive) { alive = load_v(nx, 0); pre_v0 = alive; }
          }
        }
        if (!alive) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
      } else if (warp == 1) {
        bool ok = true;
        tc_fence_after();
        // S(g & 1) = Q.K^T for the next K tile
        auto qk = [&]() -> bool {
          if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&c.k_full[0]), kt & 1))) return false;
          tc_fence_after();
          if (el) {
            if (g & 1) issue_qk_wide<1, 0, kHalf>(tm, dq, dk); else issue_qk_wide<0, 0, kHalf>(tm, dq, dk);
            tc_commit(smem_u32(&c.k_empty[0]));
          }
          __syncwarp();
          if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&c.k_full[1]), kt & 1))) return false;
          tc_fence_after();
          if (el) {
            if (g & 1) issue_qk_wide<1, 1, kHalf>(tm, dq, dk); else issue_qk_wide<0, 1, kHalf>(tm, dq, dk);
            tc_commit(smem_u32(&c.k_empty[1]));
            tc_commit(smem_u32(&c.s_full[g & 1]));
          }
          __syncwarp();
          ++kt;
          ++g;
          return true;
        };
        ok = qk();
        if (ok && ntiles > 1) ok = qk();
        for (int j = 0; ok && j < ntiles; ++j) {
          // O += P.V: P of tile gp sits in S buffer gp & 1
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.v_full[0]), vt & 1));
          if (!ok) break;
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.p_full[0]), gp & 1));
          if (!ok) break;
          tc_fence_after();
          if (el) {
            if (gp & 1) issue_pv_wide<1, 0, kHalf>(tm, dv, j == 0); else issue_pv_wide<0, 0, kHalf>(tm, dv, j == 0);
            tc_commit(smem_u32(&c.v_empty[0]));
          }
          __syncwarp();
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.v_full[1]), vt & 1));
          if (!ok) break;
          tc_fence_after();
          if (el) {
            if (gp & 1) issue_pv_wide<1, 1, kHalf>(tm, dv, j == 0); else issue_pv_wide<0, 1, kHalf>(tm, dv, j == 0);
            tc_commit(smem_u32(&c.v_empty[1]));
            tc_commit(smem_u32(&c.o_full[0]));
          }
          __syncwarp();
          ++vt;
          ++gp;
          if (j + 2 < ntiles) ok = qk();
        }
        if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
      }
      __syncwarp();
    }
  } else {
    setmaxnreg_inc<216>();
    const int xg = (warp - 4) >> 2;                      // 0: softmax + lo half of O, 1: hi half of O
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tO = tmem + lane_base + 256;
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    uint32_t g = 0;                                      // tiles of this CTA before the current one
    for (int n = 0; next_item<true, D, kTileM>(a, c, smem, n & 1, it); ++n) {
      const int32_t* entries = c.entry[n & 1];
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      float m_ref = -INFINITY, l = 0.f;
      bool ok = true;
      if (xg == 0) {
        const int qpos = it.tok0 + row;
        const int lim = it.causal ? min(it.kv_len, qpos - it.kv_tok0 + 1) : it.kv_len;
        for (int j = 0; ok && j < ntiles; ++j, ++g) {
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.s_full[g & 1]), (g >> 1) & 1));
          if (!ok) break;
          tc_fence_after();
          const uint32_t tS = tmem + lane_base + (g & 1) * kBN;
          const int key0 = j * kBN;
          const bool masked = key0 + kBN > it.kv_len || (it.causal && it.kv_tok0 + key0 + kBN - 1 > it.tok0);
          // the P.V of tile g - 1 must have executed before O is touched (tile g - 2 is known to have)
          auto wait_pv = [&] {
            if (!mbar_wait(smem_u32(&c.o_full[0]), (g - 1) & 1)) ok = false;
            tc_fence_after();
          };
          if (masked) softmax_row<true, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, wait_pv);
          else softmax_row<false, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, wait_pv);
          // keeps the completions of o_full at most one behind, so that a wait on the parity of a
          // tile index can never be answered by an older phase
          if (j > 0 && !mbar_wait(smem_u32(&c.o_full[0]), (g - 1) & 1)) ok = false;
          ok = __all_sync(0xffffffffu, ok);
          tc_fence_before();
          mbar_arrive(smem_u32(&c.p_full[0]));
        }
      } else {
        g += (uint32_t)ntiles;
      }
      bar_sync_256();                                    // the last P has been published
      if (ok) ok = mbar_wait(smem_u32(&c.o_full[0]), (g - 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      const int32_t e = entries[row];
      uint32_t v0[32], v1[32];
      if (ok) tc_fence_after();
      if (ok && xg == 0) {
        // the row's largest magnitude over all 256 dims decides the power of two of its fp16 copy
        float amax = 0.f;
#pragma unroll
        for (int ch = 0; ch < D / 32; ++ch) {
          tmem_ld32(tO + ch * 32, v0);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 2)
            amax = max3(amax, fabsf(__uint_as_float(v0[i])), fabsf(__uint_as_float(v0[i + 1])));
        }
        const float inv = 1.f / l;
        const PartialScale ps = partial_scale(amax * inv);
        c.row_inv[row] = inv * ps.scale;
        if (e >= 0) a.partial_lse[e] = make_float2((m_ref + log2f(l)) * 0.6931471805599453f, ps.inv);
      }
      bar_sync_256();                                    // the rows' factors are visible to warps 8-11
      if (ok) {
        const float mul = c.row_inv[row];
        // as above: O rows pass through this warp's 8 KB of the idle Q tile; warps 4-7 write
        // dims 0-127, warps 8-11 dims 128-255
        unsigned char* stage = smem + xg * kTileBytes + (warp & 3) * 8192;
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          tmem_ld32(tO + xg * 128 + ch * 64, v0);
          tmem_ld32(tO + xg * 128 + ch * 64 + 32, v1);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t* s8 = i < 4 ? v0 + 8 * i : v1 + 8 * (i - 4);
            *reinterpret_cast<uint4*>(stage + lane * 144 + i * 16) =
                make_uint4(pack2_half(__uint_as_float(s8[0]) * mul, __uint_as_float(s8[1]) * mul),
                           pack2_half(__uint_as_float(s8[2]) * mul, __uint_as_float(s8[3]) * mul),
                           pack2_half(__uint_as_float(s8[4]) * mul, __uint_as_float(s8[5]) * mul),
                           pack2_half(__uint_as_float(s8[6]) * mul, __uint_as_float(s8[7]) * mul));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rl = i * 4 + (lane >> 3), c16 = lane & 7;
            const int32_t er = __shfl_sync(0xffffffffu, e, rl);
            const uint4 val = *reinterpret_cast<const uint4*>(stage + rl * 144 + c16 * 16);
            if (er >= 0)
              __stcs(reinterpret_cast<uint4*>(a.partial_out + (int64_t)er * D + xg * 128 + ch * 64 + c16 * 8), val);
          }
          __syncwarp();
        }
        tc_fence_before();
      } else {
        atomicExch(a.status, ST_SOFTMAX);
        c.abort = 1;
      }
    }
  }

  if (c.abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------
// short items: chunks of at most kShortChunk keys (kShortChunkFew in all but long calls, see tc5_short_items), and query windows
// with at most 128 rows per kv head.  One 128-row tile per work item, two CTAs per SM.  (Most chunks of 96 to 128 keys:
// attend_one_tc5.cu; windows of at most eight rows at head dims 96 and 128: attend_few_tc5.cu.)
//
// Such an item is one to eight key tiles (or, in a small window, a long chunk for some
// rows), so what counts is that nothing of its hand-over is waited for.  The roles of a CTA run
// through one flat stream of key tiles, without a CTA-wide barrier between items:
//   warp 4     describes the items, up to four ahead (a chain of dependent global loads and divisions as
//              long as an item: it does nothing else)
//   warps 6, 7 copy the Q rows of the next item into the swizzled tile (cp.async) as soon as the last
//              Q.K^T of the item before has executed; warp 6 also requests K/V tiles (TMA).  An item on the
//              chunk of the item before it (the row tiles of one list are consecutive) finds K and V in
//              place when the chunk is one tile
//   warp 5     issues QK(0) PV(0) QK(1) PV(1) ...: QK of the next tile, of the next item
//              too, directly behind the PV that consumed P
//   warps 0-3, 8-11  softmax, and the epilogue: one thread per row, O from tensor memory through
//              registers to 32-byte stores (whole sectors, no staging in shared memory).  The two
//              warpgroups take the items in turn: one computes the softmax of an item while the other
//              writes the rows of the item before it (o_free: O may be overwritten)
// Per CTA: one Q, one K and one V tile (32 KB each), 256 TMEM columns (S 0-127, O 128-255); two CTAs per SM
// overlap each other's softmax, MMA and stores.
// With one warpgroup for both, softmax and epilogue of an item took most of its time, one after the other (see
// softmax_row_rolled); with two, dense stage of 2 x 4096 tokens x 16 heads, chunk 128 142 -> 134 us, 13311 x 16/4 at
// head_dim 64 162 -> 145.  An item now takes 7000 cycles of a CTA, the chain Q.K^T, S, softmax, P.V and the copy of the next Q rows.
// Measured (chunk 128 where it ran them, and decode steps where it did) against the kernel with CTA-wide barriers between items and unrolled code: dense stage of
// 2 x 4096 tokens x 16 heads, chunk 128 199 -> 146 us (whole call 347 -> 279); 13311 tokens x 16/4 heads,
// head_dim 64 233 -> 172; 32768 x 32/8 1651 -> 1094.  A decode step (chunk 4096, 131072-token prefix, 32/8 heads), in
// place of the 256-row kernel: 132 -> 90.  The rolled loops alone: 205 -> 146 on the first.
// ---------------------------------------------------------------------------
constexpr int kShortThreads = 384;

struct ShortCtrl {
  static constexpr int kPrefix = kShortPrefix;
  uint64_t q_full, k_full, v_full;         // tiles landed
  uint64_t q_free;                         // per item: its last Q.K^T has executed
  uint64_t k_free;                         // per other key tile of an item: its Q.K^T has executed
  uint64_t v_free;                         // per key tile that a new V tile follows: its P.V has executed
  uint64_t s_full[2], p_full[2], o_full[2];  // [softmax warpgroup]
  uint64_t o_free;                         // per item: its rows of O have been read
  uint64_t item_full[kShortSlots], slot_free[kShortSlots];
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;
  SlotRange own;
  ShortItem item[kShortSlots];
  alignas(16) int32_t entry[kShortSlots][kTileM];
  alignas(16) int64_t qoff[kShortSlots][kTileM];
  int32_t prefix_cache[kShortPrefix];
};
constexpr size_t kShortSmemBytes = 1024 + 3 * kTileBytes + sizeof(ShortCtrl);
static_assert(2 * (kShortSmemBytes + 1024) <= 232448, "two CTAs per SM");

template <bool kHalf, int D>
__global__ void __launch_bounds__(kShortThreads, 2)
attend_tc5_short_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const ShortArgs sa) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);
  const uint32_t sK = sQ + kTileBytes;
  const uint32_t sV = sK + kTileBytes;
  ShortCtrl& c = *reinterpret_cast<ShortCtrl*>(smem + 3 * kTileBytes);
  const KernelArgs& a = sa.a;
  constexpr uint32_t kCols = 256;
  constexpr int kNBlk = (D + 63) / 64;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&c.q_full), 64);                        // the copies of two warps' lanes
    mbar_init(smem_u32(&c.k_full), 1);
    mbar_init(smem_u32(&c.v_full), 1);
    mbar_init(smem_u32(&c.q_free), 1);
    mbar_init(smem_u32(&c.k_free), 1);
    mbar_init(smem_u32(&c.v_free), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.s_full[i]), 1);
      mbar_init(smem_u32(&c.p_full[i]), kTileM);
      mbar_init(smem_u32(&c.o_full[i]), 1);
    }
    mbar_init(smem_u32(&c.o_free), kTileM);
    for (int i = 0; i < kShortSlots; ++i) {
      mbar_init(smem_u32(&c.item_full[i]), 1);
      // The softmax warps of the item, once its first S is there.  Behind that S are the other readers of the description:
      // the MMA warp reads it in front of Q.K^T, warps 6 and 7 before they arrive on q_full, which Q.K^T waits for.
      mbar_init(smem_u32(&c.slot_free[i]), 4);
    }
    c.abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&c.tmem_slot), kCols);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] << sa.iq.tile_shift : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + (sa.iq.grouped ? c.own.n * p.Hkv : own_item_count(c.own.n, p.Hq, p.C, kTileM));
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kShortThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  bool ok = true;                          // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  if (warp == 4) {
    if (p.C <= kBN) ok = describe_items<kShortSlots, 2, true, false>(p, sa.iq, c);
    else ok = describe_items<kShortSlots, 2, false, false>(p, sa.iq, c);
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 6 || warp == 7) {
    // ---- Q rows; K/V tiles
    uint32_t kt = 0, vt = 0;               // k_free phases waited for, V tiles requested
    for (int n = 0; ok; ++n) {
      const int slot = n % kShortSlots;
      if (!wait(&c.item_full[slot], (n / kShortSlots) & 1)) break;
      if (c.item[slot].done) break;
      const int tok0 = c.item[slot].tok0, head = c.item[slot].head;
      const int ntiles = (c.item[slot].kv_len + kBN - 1) / kBN;
      const bool fresh = c.item[slot].new_kv != 0;
      auto load = [&](uint32_t dst, const CUtensorMap* m, uint64_t* full, int j) {
        if (lane == 0) {
          const uint32_t bar = smem_u32(full);
          mbar_expect_tx(bar, kNBlk * kHalfBytes);
          tma_load_3d(dst, m, bar, 0, head, tok0 + j * kBN);
          if (D > 64) tma_load_3d(dst + kHalfBytes, m, bar, 64, head, tok0 + j * kBN);
        }
      };
      if (n > 0 && !wait(&c.q_free, (n - 1) & 1)) break;
      if (warp == 6 && fresh) load(sK, &tmap_k, &c.k_full, 0);
      copy_rows_async<D / 8, 2>(sQ, a.q, 0, warp - 6, c.item[slot].nrows, [&](int r) { return c.qoff[slot][r]; });
      cp_async_mbar_arrive(smem_u32(&c.q_full));
      if (warp == 6)
        for (int j = 0; j < ntiles; ++j) {
          if (j > 0) {
            if (!wait(&c.k_free, kt & 1)) break;
            ++kt;
            load(sK, &tmap_k, &c.k_full, j);
          }
          if (!fresh) break;                                   // (one tile, in place)
          if (vt > 0 && !wait(&c.v_free, (vt - 1) & 1)) break;
          ++vt;
          load(sV, &tmap_v, &c.v_full, j);
        }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 5) {
    // ---- MMA issuer: the whole warp runs this code, one elected lane issues.  Predicated MMAs instead of a branch around them:
    // dense stage of 700 tokens behind 50021, 32/8 heads, chunk 1024 139 -> 134.5 us; 20000 x 16/4 at
    // head dim 64, chunk 1024 887 -> 858; 32768 x 32/8, chunk 512 2.58 -> 2.46 ms
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    uint32_t kt = 0, vt = 0;               // K / V tiles consumed
    uint32_t pph[2] = {0, 0};              // p_full phases
    // Q.K^T of tile j of item n; `fresh`: the K tile is a new one
    auto qk = [&](int n, int j, int ntiles, bool fresh) {
      if (j == 0) {
        if (!wait(&c.q_full, n & 1)) return;
        fence_proxy_async_smem();                             // rows written by cp.async, read by the tensor core
      }
      if (fresh) {
        if (!wait(&c.k_full, kt & 1)) return;
        ++kt;
      }
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint32_t koff = (uint32_t)((ks >> 2) * (kHalfBytes >> 4) + (ks & 3) * 2);
        mma_ss_el<kDescHi>(el, tm, dq + koff, dk + koff, kIdescQK<kHalf>, ks > 0);
      }
      tc_commit_el(el, smem_u32(&c.s_full[n & 1]));
      tc_commit_el(el, smem_u32(j + 1 == ntiles ? &c.q_free : &c.k_free));
    };
    int n = 0;
    if (wait(&c.item_full[0], 0) && !c.item[0].done) {
      int ntiles = (c.item[0].kv_len + kBN - 1) / kBN;
      bool fresh = c.item[0].new_kv != 0;
      qk(0, 0, ntiles, fresh);
      while (ok) {
        int next_tiles = 0;
        bool next_fresh = false, more = true;
        for (int j = 0; ok && j < ntiles; ++j) {
          if (fresh) {
            if (!wait(&c.v_full, vt & 1)) break;
            ++vt;
          }
          const int x = n & 1;
          if (!wait(&c.p_full[x], x ? pph[1] : pph[0])) break;
          if (x) pph[1] ^= 1; else pph[0] ^= 1;
          if (j == 0 && n > 0 && !wait(&c.o_free, (n - 1) & 1)) break;
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            mma_ts_el<kDescHi>(el, tm + 128, tm + ks * 8, dv + ks * (2048 >> 4), kIdescPV<kHalf, D>, j > 0 || ks > 0);
          tc_commit_el(el, smem_u32(j + 1 == ntiles ? &c.o_full[x] : &c.v_free));
          if (j + 1 < ntiles) {
            qk(n, j + 1, ntiles, true);
          } else {
            const int s1 = (n + 1) % kShortSlots;
            if (!wait(&c.item_full[s1], ((n + 1) / kShortSlots) & 1)) break;
            more = !c.item[s1].done;
            next_tiles = (c.item[s1].kv_len + kBN - 1) / kBN;
            next_fresh = c.item[s1].new_kv != 0;
            if (more) {
              if (next_fresh) tc_commit_el(el, smem_u32(&c.v_free));
              qk(n + 1, 0, next_tiles, next_fresh);
            }
          }
        }
        if (!ok || !more) break;
        ntiles = next_tiles;
        fresh = next_fresh;
        ++n;
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else {
    // ---- softmax + epilogue, one thread per row; warpgroup x takes items x, x + 2, ...
    const int x = warp >> 3;
    const int row0 = (warp & 3) * 32, row = row0 + lane;
    const uint32_t lane_base = (uint32_t)row0 << 16;
    const uint32_t tS = tmem + lane_base;
    const uint32_t tO = tmem + lane_base + 128;
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    uint32_t sph = 0;                      // phase of s_full[x]
    for (int n = x; ok; n += 2) {
      const int slot = n % kShortSlots;
      if (!wait(&c.item_full[slot], (n / kShortSlots) & 1)) break;
      if (c.item[slot].done) break;
      const int kv_len = c.item[slot].kv_len, tok_rel = c.item[slot].tok_rel, group = c.item[slot].group;
      const bool causal = c.item[slot].causal != 0;
      const bool active = row0 < c.item[slot].nrows;     // warps without rows only keep the barriers going
      const int32_t e = c.entry[slot][row];
      const int ntiles = (kv_len + kBN - 1) / kBN;
      const int qrel = tok_rel + (group == 1 ? row : row / group);              // own chunk: position in the chunk
      const int lim = causal ? min(kv_len, qrel + 1) : kv_len;                  // keys < lim are visible
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < ntiles; ++j) {
        if (!wait(&c.s_full[x], sph)) break;
        sph ^= 1;
        // the item's Q.K^T has run: every role has read its description
        if (j == 0 && lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
        if (active) {
          tc_fence_after();
          const int key0 = j * kBN;
          const bool masked = key0 + kBN > kv_len || (causal && key0 + kBN - 1 > tok_rel);
          // S of the next tile is only computed after this tile's P.V: O is quiet here
          if (masked) softmax_row_rolled<true, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, [] {});
          else softmax_row_rolled<false, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, [] {});
          tc_fence_before();
        }
        mbar_arrive(smem_u32(&c.p_full[x]));
      }
      if (!ok || !wait(&c.o_full[x], (n >> 1) & 1)) break;
      if (active) {
        tc_fence_after();
        // the row's largest magnitude decides the power of two its fp16 copy is scaled by
        const float amax = amax_row_rolled<D>(tO, tO + 64);
        const float inv = 1.f / l;
        const PartialScale ps = partial_scale(amax * inv);
        store_row_rolled<D>(tO, tO + 64, a.partial_out + (int64_t)(e >= 0 ? e : 0) * D, inv * ps.scale, e >= 0, a.wide_store != 0,
                            [&] {
                              tc_fence_before();
                              mbar_arrive(smem_u32(&c.o_free));   // O may be overwritten
                            });
        if (e >= 0) a.partial_lse[e] = make_float2((m_ref + log2f(l)) * 0.6931471805599453f, ps.inv);
      } else {
        mbar_arrive(smem_u32(&c.o_free));
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
  if (warp == 5) tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------------------
// head dim 256, chunks of at most kSmallChunk keys
//
// The operands, tensor memory and order of MMAs of attend_tc5_wide_kernel, with the roles of the kernel
// above: one 128-row tile per work item, one CTA per SM, one flat stream of items and key tiles.  The
// halves of Q, of K and of V have 32 KB slots of their own, each refilled as soon as the MMAs that read it
// have executed.  Two softmax warpgroups take the items in turn: one computes the next item's softmax
// while the other waits for its P.V and writes its rows.  The P.V of a tile can still be executing when
// the softmax of the item's next tile wants to rescale O: that path waits for it.  The Q rows of the next item are
// copied by the warpgroup whose item's last Q.K^T has just executed, in front of its last softmax step: with a
// warp of its own for each half of Q the MMAs waited half of an item's time for 64 copies a lane (281 -> 228 us; one tile
// of 128 dims waits for softmax instead, and there two warps of their own are better: 126 against 154).  Measured
// against the wide kernel, 2 x 4096 tokens x 16 heads, chunk 128: 446 -> 228 us.  Long chunks stay with the wide kernel: 295 tokens behind
// 22411, 16 heads, chunk 4096 take 200 us there and 236 here.
// ---------------------------------------------------------------------------
// warp 0 describes the items, 1 issues MMAs, 2 requests K, 3 requests V; 4-7, 8-11: softmax of the even / odd items, and the Q rows
// of the item behind
constexpr int kWideShortThreads = 384;

struct WideShortCtrl {
  static constexpr int kPrefix = kShortPrefix;
  uint64_t q_full[2], k_full[2], v_full[2];        // halves landed
  uint64_t q_free[2];                              // per item: its last Q.K^T has read the halves
  uint64_t k_free[2];                              // per other key tile of an item: its Q.K^T has read the half of K
  uint64_t v_free[2];                              // per key tile that a new V follows: its P.V has read the half
  uint64_t s_full[2][2];                           // [warpgroup][S buffer]
  uint64_t p_full[2], pv_full[2];                  // [warpgroup], once per key tile
  uint64_t o_free;                                 // once per item: its rows of O have been read
  uint64_t item_full[kShortSlots], slot_free[kShortSlots];
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;
  SlotRange own;
  ShortItem item[kShortSlots];
  alignas(16) int32_t entry[kShortSlots][kTileM];
  alignas(16) int64_t qoff[kShortSlots][kTileM];
  int32_t prefix_cache[kShortPrefix];
};
constexpr size_t kWideShortSmemBytes = 1024 + 6 * kTileBytes + sizeof(WideShortCtrl);
static_assert(kWideShortSmemBytes <= 232448, "shared memory of one CTA");

template <bool kHalf>
__global__ void __launch_bounds__(kWideShortThreads, 1)
attend_tc5_wide_short_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k,
                       const __grid_constant__ CUtensorMap tmap_v, const ShortArgs sa) {
  constexpr int D = 256;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sQ = smem_u32(smem);                       // lo, hi
  const uint32_t sK = sQ + 2 * kTileBytes;                  // lo, hi
  const uint32_t sV = sK + 2 * kTileBytes;                  // lo, hi
  WideShortCtrl& c = *reinterpret_cast<WideShortCtrl*>(smem + 6 * kTileBytes);
  const KernelArgs& a = sa.a;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.q_full[i]), kTileM + 1);          // the copies of a warpgroup; warp 2
      mbar_init(smem_u32(&c.k_full[i]), 1);
      mbar_init(smem_u32(&c.v_full[i]), 1);
      mbar_init(smem_u32(&c.q_free[i]), 1);
      mbar_init(smem_u32(&c.k_free[i]), 1);
      mbar_init(smem_u32(&c.v_free[i]), 1);
      mbar_init(smem_u32(&c.s_full[i][0]), 1);
      mbar_init(smem_u32(&c.s_full[i][1]), 1);
      mbar_init(smem_u32(&c.p_full[i]), kTileM);
      mbar_init(smem_u32(&c.pv_full[i]), 1);
    }
    mbar_init(smem_u32(&c.o_free), kTileM);
    for (int i = 0; i < kShortSlots; ++i) {
      mbar_init(smem_u32(&c.item_full[i]), 1);
      // The readers of a description and what orders each before the slot's next item: the MMA warp reads it in front of
      // Q.K^T, warp 2 and the warpgroup that copies the Q rows before they arrive on q_full, which Q.K^T waits for; the
      // softmax warps of the item arrive here once its first S is there, behind all of these.  Warp 3 requests V, which no
      // Q.K^T waits for: it arrives here itself.
      mbar_init(smem_u32(&c.slot_free[i]), 5);
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
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] << sa.iq.tile_shift : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + (sa.iq.grouped ? c.own.n * p.Hkv : own_item_count(c.own.n, p.Hq, p.C, kTileM));
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kWideShortThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  bool ok = true;                          // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  if (warp == 0) {
    if (p.C <= kBN) ok = describe_items<kShortSlots, 2, true, false>(p, sa.iq, c);
    else ok = describe_items<kShortSlots, 2, false, false>(p, sa.iq, c);
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 2 || warp == 3) {
    // ---- warp 2: K tiles, warp 3: V tiles
    uint32_t kt = 0, vt = 0;               // k_free phases waited for, V tiles requested
    for (int n = 0; ok; ++n) {
      const int slot = n % kShortSlots;
      if (!wait(&c.item_full[slot], (n / kShortSlots) & 1)) break;
      if (c.item[slot].done) break;
      const int tok0 = c.item[slot].tok0, head = c.item[slot].head;
      const int ntiles = (c.item[slot].kv_len + kBN - 1) / kBN;
      const bool fresh = c.item[slot].new_kv != 0;
      __syncwarp();                                             // every lane has read the description
      if (warp == 3 && lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
      auto load = [&](uint32_t dst, const CUtensorMap* m, uint64_t* full, int h, int j) {
        if (lane == 0) {
          const uint32_t bar = smem_u32(full);
          mbar_expect_tx(bar, kTileBytes);
          tma_load_3d(dst, m, bar, h * 128, head, tok0 + j * kBN);
          tma_load_3d(dst + kHalfBytes, m, bar, h * 128 + 64, head, tok0 + j * kBN);
        }
      };
      if (warp == 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (n > 0 && !wait(&c.q_free[h], (n - 1) & 1)) break;
          if (lane == 0) mbar_arrive(smem_u32(&c.q_full[h]));   // (nobody runs past a phase this warp waits for)
          if (fresh) load(sK + h * kTileBytes, &tmap_k, &c.k_full[h], h, 0);
        }
        for (int j = 1; ok && j < ntiles; ++j, ++kt)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!wait(&c.k_free[h], kt & 1)) break;
            load(sK + h * kTileBytes, &tmap_k, &c.k_full[h], h, j);
          }
      } else {
        if (fresh)
          for (int j = 0; ok && j < ntiles; ++j, ++vt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (vt > 0 && !wait(&c.v_free[h], (vt - 1) & 1)) break;
              load(sV + h * kTileBytes, &tmap_v, &c.v_full[h], h, j);
            }
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 1) {
    // ---- MMA issuer
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sK, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    // the two streams: Q.K^T runs one key tile ahead of P.V
    uint32_t gq = 0, kt = 0, vt = 0;       // key tiles whose Q.K^T has been issued; K, V tiles consumed
    int nq = 0, jq = 0, tiles_q = 0;       // item and tile of the next Q.K^T; tiles of that item (0: not looked at yet)
    bool fresh_q = false, end = false;
    // Q.K^T of the next key tile; false when there is none (or a wait gave up)
    auto qk = [&]() -> bool {
      if (end) return false;
      if (jq == 0) {
        const int slot = nq % kShortSlots;
        if (!wait(&c.item_full[slot], (nq / kShortSlots) & 1)) return false;
        if (c.item[slot].done) { end = true; return false; }
        tiles_q = (c.item[slot].kv_len + kBN - 1) / kBN;
        fresh_q = c.item[slot].new_kv != 0;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (jq == 0) {
          if (!wait(&c.q_full[h], nq & 1)) return false;
          fence_proxy_async_smem();                           // rows written by cp.async, read by the tensor core
        }
        if (fresh_q && !wait(&c.k_full[h], kt & 1)) return false;
        tc_fence_after();
        if (el) {
          if (h == 0) { if (gq & 1) issue_qk_wide<1, 0, kHalf>(tm, dq, dk); else issue_qk_wide<0, 0, kHalf>(tm, dq, dk); }
          else        { if (gq & 1) issue_qk_wide<1, 1, kHalf>(tm, dq, dk); else issue_qk_wide<0, 1, kHalf>(tm, dq, dk); }
          if (h == 1) tc_commit(smem_u32(&c.s_full[nq & 1][gq & 1]));
          tc_commit(smem_u32(jq + 1 == tiles_q ? &c.q_free[h] : &c.k_free[h]));
        }
        __syncwarp();
      }
      if (fresh_q) ++kt;
      ++gq;
      if (++jq == tiles_q) { jq = 0; ++nq; }
      return true;
    };
    uint32_t pph[2] = {0, 0};              // p_full phases
    bool have = qk();
    int np = 0, jp = 0, tiles_p = tiles_q;
    uint32_t gp = 0;
    bool fresh_p = fresh_q;
    while (ok && have) {
      const bool next = qk();
      if (!ok) break;
      const int x = np & 1;
      if (!wait(&c.p_full[x], x ? pph[1] : pph[0])) break;
      if (x) pph[1] ^= 1; else pph[0] ^= 1;
      if (jp == 0 && np > 0 && !wait(&c.o_free, (np - 1) & 1)) break;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (fresh_p && !wait(&c.v_full[h], vt & 1)) break;
        tc_fence_after();
        if (el) {
          if (h == 0) { if (gp & 1) issue_pv_wide<1, 0, kHalf>(tm, dv, jp == 0); else issue_pv_wide<0, 0, kHalf>(tm, dv, jp == 0); }
          else        { if (gp & 1) issue_pv_wide<1, 1, kHalf>(tm, dv, jp == 0); else issue_pv_wide<0, 1, kHalf>(tm, dv, jp == 0); }
          if (next && fresh_q) tc_commit(smem_u32(&c.v_free[h]));       // (the stream is one tile ahead: fresh_q is the next tile's)
          if (h == 1) tc_commit(smem_u32(&c.pv_full[x]));
        }
        __syncwarp();
      }
      if (!ok) break;
      if (fresh_p) ++vt;
      ++gp;
      if (++jp == tiles_p) { jp = 0; ++np; tiles_p = tiles_q; }
      fresh_p = fresh_q;
      have = next;
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else {
    // ---- softmax + epilogue, one thread per row; warpgroup x takes items x, x + 2, ...
    const int x = (warp >> 2) - 1;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tO = tmem + lane_base + 256;
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    uint32_t sph0 = 0, sph1 = 0, pvph = 0;                     // phases of s_full[x][0], [1] and pv_full[x]
    // Q rows of item m; the last Q.K^T of the item before has executed
    auto copy_rows = [&](int m) {
      const int slot = m % kShortSlots;
      if (!wait(&c.item_full[slot], (m / kShortSlots) & 1) || c.item[slot].done) return;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        copy_rows_async<16, 4>(sQ + h * kTileBytes, a.q, 16 * h, warp & 3, c.item[slot].nrows, [&](int r) { return c.qoff[slot][r]; });
        cp_async_mbar_arrive(smem_u32(&c.q_full[h]));
      }
    };
    if (x == 1) copy_rows(0);
    for (int n = x; ok; n += 2) {
      const int slot = n % kShortSlots;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.item_full[slot]), (n / kShortSlots) & 1));
      if (!ok) break;
      const ShortItem it = c.item[slot];
      if (it.done) break;
      const int32_t e = c.entry[slot][row];
      const bool active = (warp & 3) * 32 < it.nrows;         // warps without rows only keep the barriers going
      const int ntiles = (it.kv_len + kBN - 1) / kBN;
      const int qrel = it.tok_rel + (it.group == 1 ? row : row / it.group);
      const int lim = it.causal ? min(it.kv_len, qrel + 1) : it.kv_len;
      float m_ref = -INFINITY, l = 0.f;
      for (int j = 0; j < ntiles; ++j) {
        const uint32_t buf = (uint32_t)(it.tile0 + j) & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.s_full[x][buf]), buf ? sph1 : sph0));
        if (!ok) break;
        if (buf) sph1 ^= 1; else sph0 ^= 1;
        // the item's Q.K^T has run: every role but warp 3 has read its description
        if (j == 0 && lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
        if (j + 1 == ntiles) copy_rows(n + 1);
        if (!ok) break;
        // the P.V of the tile before must have executed before O is touched
        bool waited = j == 0;
        auto wait_pv = [&] {
          if (!waited && !mbar_wait(smem_u32(&c.pv_full[x]), pvph)) ok = false;
          waited = true;
          tc_fence_after();
        };
        if (active) {
          tc_fence_after();
          const int key0 = j * kBN;
          const bool masked = key0 + kBN > it.kv_len || (it.causal && key0 + kBN - 1 > it.tok_rel);
          const uint32_t tS = tmem + lane_base + buf * kBN;
          if (masked) softmax_row_rolled<true, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, wait_pv);
          else softmax_row_rolled<false, kHalf, D>(tS, tO, j, key0, lim, sl2, m_ref, l, wait_pv);
        }
        // every completion of pv_full is waited for before the next P is published, so that a phase is
        // never passed by
        if (j > 0) {
          wait_pv();
          pvph ^= 1;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_before();
        mbar_arrive(smem_u32(&c.p_full[x]));
      }
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.pv_full[x]), pvph));
      if (!ok) break;
      pvph ^= 1;
      if (active) {
        tc_fence_after();
        // the row's largest magnitude over all 256 dims decides the power of two of its fp16 copy
        const float amax = amax_row_rolled<D>(tO, tO + 64);
        const float inv = 1.f / l;
        const PartialScale ps = partial_scale(amax * inv);
        store_row_rolled<D>(tO, tO + 64, a.partial_out + (int64_t)(e >= 0 ? e : 0) * D, inv * ps.scale, e >= 0, a.wide_store != 0, [&] {
          tc_fence_before();
          mbar_arrive(smem_u32(&c.o_free));                   // O may be overwritten
        });
        if (e >= 0) a.partial_lse[e] = make_float2((m_ref + log2f(l)) * 0.6931471805599453f, ps.inv);
      } else {
        mbar_arrive(smem_u32(&c.o_free));
      }
    }
    if (!ok) {
      atomicExch(a.status, ST_SOFTMAX);
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

// One warp waits, with the same bounded wait every role of the dense stage uses, on a barrier
// nobody ever arrives on: the wait gives up after `limit_ns`, the status word is set like the
// kernel would set it, and the warp returns.  Lets a test see the give-up path without a fault.
__global__ void bounded_wait_probe_kernel(int32_t* status, unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (!mbar_wait(smem_u32(&bar), 0, limit_ns) && threadIdx.x == 0) atomicExch(status, ST_SOFTMAX);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

}  // namespace

// [T, H, D] 16-bit tensor with element strides (st, sh, 1): boxes of `box_rows` tokens x `box_heads` heads x
// 64 dims, 128-byte swizzle; elements outside the tensor read as zero
bool make_tile_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int H, int64_t st,
                   int64_t sh, int box_heads, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)T};
  const cuuint64_t strides[2] = {(cuuint64_t)sh * 2, (cuuint64_t)st * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_heads, (cuuint32_t)box_rows};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_kv_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int Hkv, int64_t st, int64_t sh,
                 int box_rows) {
  return make_tile_map(m, fp16, D, base, T, Hkv, st, sh, 1, box_rows);
}

cudaError_t launch_bounded_wait_probe(int32_t* status, unsigned long long limit_ns, cudaStream_t st) {
  bounded_wait_probe_kernel<<<1, 32, 0, st>>>(status, limit_ns);
  return cudaGetLastError();
}

cudaError_t launch_attend_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k,
                              const __nv_bfloat16* v, const int32_t* cu, const int32_t* list_counts,
                              const int32_t* list_offsets, const int32_t* tile_prefix,
                              const int32_t* row_list, __half* partial_out, float2* partial_lse,
                              int32_t* work_counter, int32_t* status, cudaStream_t st) {
  if (p.D != 64 && p.D != 96 && p.D != 128 && p.D != 256) return cudaErrorInvalidValue;
  const int sms = device_info().sms;
  const int which = tc5_kernel(p);
  if (which == MOBA_KERNEL_ONE_TILE)
    return launch_attend_one_tc5(p, q, k, v, cu, list_counts, list_offsets, tile_prefix, row_list, partial_out, partial_lse,
                                 work_counter, status, sms, st);
  if (which == MOBA_KERNEL_FEW_ROWS)
    return launch_attend_few_tc5(p, q, k, v, cu, list_counts, list_offsets, tile_prefix, row_list, partial_out, partial_lse,
                                 work_counter, status, sms, st);
  CUtensorMap mk, mv;
  if (!make_kv_map(&mk, p.fp16 != 0, p.D, k, p.T, p.Hkv, p.sk_t, p.sk_h, kBN) || !make_kv_map(&mv, p.fp16 != 0, p.D, v, p.T, p.Hkv, p.sv_t, p.sv_h, kBN))
    return cudaErrorNotSupported;
  const KernelArgs args{q, cu, list_counts, list_offsets, tile_prefix, row_list, partial_out, partial_lse,
                        work_counter, status, ((uintptr_t)partial_out & 31) == 0};
  cudaError_t e;
  if (which == MOBA_KERNEL_WIDE_SHORT || which == MOBA_KERNEL_SHORT) {
    auto kern = p.D == 256 ? (p.fp16 ? attend_tc5_wide_short_kernel<true> : attend_tc5_wide_short_kernel<false>)
              : p.D == 128 ? (p.fp16 ? attend_tc5_short_kernel<true, 128> : attend_tc5_short_kernel<false, 128>)
              : p.D == 96  ? (p.fp16 ? attend_tc5_short_kernel<true, 96> : attend_tc5_short_kernel<false, 96>)
                           : (p.fp16 ? attend_tc5_short_kernel<true, 64> : attend_tc5_short_kernel<false, 64>);
    const int threads = p.D == 256 ? kWideShortThreads : kShortThreads, ctas = p.D == 256 ? sms : 2 * sms;
    const size_t smem = p.D == 256 ? kWideShortSmemBytes : kShortSmemBytes;
    e = prepare_kernel(kern, smem);
    if (e != cudaSuccess) return e;
    ShortArgs sa;
    sa.a = args;
    const bool grouped = p.Tq * p.G <= kTileM;
    // (a window's lists have one tile of either size)
    const int tile_shift = p.D == 256 || tc5_small_tiles(p.D, p.C) || grouped ? 0 : 1;
    sa.iq = item_queue(p, cu, list_counts, list_offsets, tile_prefix, row_list, work_counter, short_batch(p, ctas, grouped), grouped,
                       tile_shift);
    return launch_pdl(kern, dim3(sa.iq.grouped ? window_ctas(p, ctas) : ctas), threads, smem, st, p, mk, mv, sa);
  }
  auto kernel = p.D == 256 ? (p.fp16 ? attend_tc5_wide_kernel<true> : attend_tc5_wide_kernel<false>)
              : p.D == 128 ? (p.fp16 ? attend_tc5_kernel<true, 128> : attend_tc5_kernel<false, 128>)
              : p.D == 96  ? (p.fp16 ? attend_tc5_kernel<true, 96> : attend_tc5_kernel<false, 96>)
                           : (p.fp16 ? attend_tc5_kernel<true, 64> : attend_tc5_kernel<false, 64>);
  e = prepare_kernel(kernel, kSmemBytes);
  if (e != cudaSuccess) return e;
  return launch_pdl(kernel, dim3(sms), kThreads, kSmemBytes, st, p, mk, mv, args);
}

}  // namespace moba
