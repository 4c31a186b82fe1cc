// Dense stage of a decode step: query windows of at most eight rows per kv head (head dim 96 or 128).
//
// A list then has a handful of rows, and an item is a whole chunk of K and V for them: the stage is bound by the bytes of K and V
// as long as the chain of a key tile is shorter than the tile takes to arrive (64 KB, about 3000 cycles with all SMs loading).
// With rows as the lanes of tensor memory, as in the other kernels, one warp of an SM has rows at all and works through 128 scores
// of each in one thread: 3900 cycles a tile.  Here the operands change places:
//   S^T = K . Q^T      keys are the 128 lanes, rows the 16 columns: a thread has one key, for all rows
//   O^T += V^T . P^T   dims are the lanes; P goes through shared memory (a B operand of 16 rows x 128 keys)
// Results are the other kernels' bit for bit: an element of a product is summed over the same operands in the same steps of 16,
// the maximum, the reference of a row and the exponentials are the same, the largest magnitude of a row too, and
// the sum of a row is added in their order (four running sums over every fourth key), by a warp of its own.
//
// Roles (256 threads, two CTAs per SM):
//   warps 0-3   softmax: one thread per key; epilogue: one thread per dim
//   warp 4      row sums
//   warp 5      describes the items
//   warp 6      Q rows (cp.async); issues QK(g + 1) PV(g), g running through the key tiles of all items
//   warp 7      K and V tiles (TMA), in the order in which they are used: K0 K1 V0 K2 V1 ...
// Dense stage of one decode step, chunk 4096, against attend_tc5_short_kernel (us; whole step in brackets):
//   131072 tokens, 32/8 heads   83.4 -> 57 (107 -> 80)   344 MB of K and V: 52 at the measured copy bandwidth
//   131072, 16/16               74.4 -> 45.1 (98 -> 71)
//   131072, 8/1, top-k 12       71.5 -> 47.8 (95 -> 70)    few items: the chain of a tile, 2700 cycles
//   34816, 8/1, chunk 2048, head dim 96   38.2 -> 27.2 (58 -> 46)
//   65536, 32/8, chunk 1024     30.2 -> 21.0;  20479, chunk 512 19.7 -> 16.3;  5000, chunk 128 12.3 -> 12.0
// Eight rows, because the exponentials of more do not fit beside three K/V tiles and a second CTA.  Head dim 64 stays with the kernel for
// short items: a form of this one for it (O^T with M = 64, tiles of half the bytes) has not been built.
// Six K/V tiles instead of three where one CTA per SM has all items, chunk 4096: 131072 and 65536 tokens, 16/16 and 8/8 heads 47.1 -> 45.1 us (whole
// step 143.4 -> 141.8, 80.9 -> 79.4); 20479 tokens, 16/4 49.2 both; chunk 1024 20.5 both; 8/1, top-k 12 50.2 / 51.2.
#include "attend_rows.cuh"
#include "common.cuh"
#include "short_items.cuh"
#include "sm100_ptx.cuh"

namespace moba {

bool make_kv_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int Hkv, int64_t st,
                 int64_t sh, int box_rows);

namespace {

constexpr int kFewThreads = 256;
constexpr int kFewSlots = 4;               // item descriptions in flight
constexpr int kFewMaxStages = 6;           // K and V tiles: three where two CTAs share an SM, six for one
constexpr int kFewN = 16;                  // columns of S and O (rows behind kFewRows are never read)
constexpr int kFewBlock = kFewN * 128;     // bytes of 64 dims of Q, or of P for 64 keys
constexpr int kSumStride = kBN + 4;        // floats of a row of exponentials: reads of every fourth one by eight rows spread over the banks

template <bool kHalf> constexpr uint32_t kIdescFewQK = idesc_16_f32(kHalf, 128, kFewN, 0, 0);
template <bool kHalf> constexpr uint32_t kIdescFewPV = idesc_16_f32(kHalf, 128, kFewN, 1, 0);

struct FewItem {
  ShortItem s;
  int32_t rows_at, qhead;                  // see short_pick
};

struct FewCtrl {
  static constexpr int kPrefix = 64;
  uint64_t full[kFewMaxStages], empty[kFewMaxStages];
  uint64_t q_full, q_free;                 // per item
  uint64_t s_full[2];                      // [tile mod 2]
  uint64_t p_full, pv_done, sum_done;      // per tile
  uint64_t o_full;                         // per item
  uint64_t exchange;                       // the four softmax warps, one lane each
  uint64_t item_full[kFewSlots], slot_free[kFewSlots];
  uint32_t tmem_slot;
  volatile int32_t abort;
  int32_t n_routed, n_items;
  SlotRange own;
  FewItem item[kFewSlots];
  alignas(16) float warp_max[2][kFewRows][4];
  float alpha[2][kFewRows], row_sum[kFewRows];
  int32_t prefix_cache[kPrefix];
  float p32[kFewRows][kSumStride];         // exponentials of the tile
};
template <int kStages> constexpr size_t few_smem_bytes() { return 1024 + kStages * kTileBytes + 4 * kFewBlock + sizeof(FewCtrl); }
static_assert(2 * (few_smem_bytes<3>() + 1024) <= 233472, "two CTAs per SM");
static_assert(few_smem_bytes<kFewMaxStages>() <= 232448, "shared memory of one CTA");

__device__ __forceinline__ float redux_max(float x) {          // over the warp; NaN only if all are
  float y;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

template <bool kHalf, int D, int kStages>
__global__ void __launch_bounds__(kFewThreads, 2)
attend_tc5_few_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const ShortArgs sa) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sKV = smem_u32(smem);
  const uint32_t sQ = sKV + kStages * kTileBytes;          // two blocks of 64 dims
  const uint32_t sP = sQ + 2 * kFewBlock;                     // two blocks of 64 keys
  FewCtrl& c = *reinterpret_cast<FewCtrl*>(smem + kStages * kTileBytes + 4 * kFewBlock);
  const KernelArgs& a = sa.a;
  constexpr uint32_t kCols = 64;           // S of the even and the odd tiles at 0 and 16, O at 32
  constexpr uint32_t kO = 32;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&c.full[i]), 1);
      mbar_init(smem_u32(&c.empty[i]), 1);
    }
    mbar_init(smem_u32(&c.q_full), 32);
    mbar_init(smem_u32(&c.q_free), 1);
    mbar_init(smem_u32(&c.s_full[0]), 1);
    mbar_init(smem_u32(&c.s_full[1]), 1);
    mbar_init(smem_u32(&c.p_full), kBN);
    mbar_init(smem_u32(&c.pv_done), 1);
    mbar_init(smem_u32(&c.sum_done), 1);
    mbar_init(smem_u32(&c.o_full), 1);
    mbar_init(smem_u32(&c.exchange), 4);
    for (int i = 0; i < kFewSlots; ++i) {
      mbar_init(smem_u32(&c.item_full[i]), 1);
      mbar_init(smem_u32(&c.slot_free[i]), 7);                 // every warp but the describing one, when it has read the description
    }
    c.abort = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 6) {
    tmem_alloc(smem_u32(&c.tmem_slot), kCols);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    c.n_routed = p.hist > 0 ? a.tile_prefix[p.lists] : 0;
    c.own = own_slot_range(p, a.cu);
    c.n_items = c.n_routed + c.own.n * p.Hkv;
  }
  if (p.hist > 0) fill_prefix_cache(c, a.tile_prefix, p.lists, kFewThreads);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  bool ok = true;                          // false: a wait of this role gave up
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity));
    return ok;
  };
  // The next item's description, for every warp but the one that writes them; false at the end (or when a wait gave up).
  int items = 0;                           // taken
  FewItem it;
  auto next_item = [&]() {
    const int slot = items % kFewSlots;
    if (!wait(&c.item_full[slot], (items / kFewSlots) & 1)) return false;
    it = c.item[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&c.slot_free[slot]));
    ++items;
    return __shfl_sync(0xffffffffu, it.s.done, 0) == 0;
  };
  auto tiles_of = [&]() { return __shfl_sync(0xffffffffu, (it.s.kv_len + kBN - 1) / kBN, 0); };

  if (warp == 5) {
    // ---- descriptions
    ShortQueue w;
    short_start(sa.iq, c, w);
    int n = 0;
    for (bool done = false; ok && !done;) {
      FewItem o;
      short_pick<true>(p, sa.iq, c, w, o.s, o.s.tok0, o.s.head, o.rows_at, o.qhead);
      done = o.s.done;
      // (the lists of a selection that names a chunk for several ranks of a row are longer than the window has rows)
      int rows = o.s.nrows;
      do {
        o.s.nrows = min(rows, kFewRows);
        const int slot = n % kFewSlots;
        if (n >= kFewSlots && !wait(&c.slot_free[slot], (n / kFewSlots - 1) & 1)) break;
        if (lane == 0) {
          c.item[slot] = o;
          mbar_arrive(smem_u32(&c.item_full[slot]));
        }
        __syncwarp();
        ++n;
        o.rows_at += kFewRows;
        rows -= kFewRows;
      } while (rows > 0);
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 7) {
    // ---- K and V tiles: K of a tile in front of V of the tile before it
    int g = 0;                             // tiles requested
    auto load = [&](const CUtensorMap* m, int head, int tok) {
      const int st = g % kStages;
      if (g >= kStages && !wait(&c.empty[st], (g / kStages - 1) & 1)) return false;
      ++g;
      if (lane == 0) {
        const uint32_t bar = smem_u32(&c.full[st]), dst = sKV + st * kTileBytes;
        mbar_expect_tx(bar, kTileBytes);
        tma_load_3d(dst, m, bar, 0, head, tok);
        tma_load_3d(dst + kHalfBytes, m, bar, 64, head, tok);
      }
      __syncwarp();
      return true;
    };
    int v_tok = -1, v_head = 0;            // V that is still to be requested
    while (ok && next_item()) {
      const int n = tiles_of();
      for (int j = 0; j < n; ++j) {
        const int tok = it.s.tok0 + j * kBN;
        if (!load(&tmap_k, it.s.head, tok)) break;
        if (v_tok >= 0 && !load(&tmap_v, v_head, v_tok)) break;
        v_tok = tok;
        v_head = it.s.head;
      }
    }
    if (ok && v_tok >= 0) load(&tmap_v, v_head, v_tok);
    if (!ok && lane == 0) { atomicExch(a.status, ST_PRODUCER); c.abort = 1; }
  } else if (warp == 6) {
    // ---- Q rows and MMAs: the whole warp runs this code, one elected lane issues
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t dq = __shfl_sync(0xffffffffu, desc_lo(sQ, 16), 0);
    const uint32_t dp = __shfl_sync(0xffffffffu, desc_lo(sP, 16), 0);
    const uint32_t dk = __shfl_sync(0xffffffffu, desc_lo(sKV, 16), 0);
    const uint32_t dv = __shfl_sync(0xffffffffu, desc_lo(sKV, kHalfBytes), 0);
    const uint32_t el = elect_one();
    int g = 0, at = 0;                     // Q.K^T issued, ring tiles taken
    auto copy_q = [&]() {                  // rows of item `it`; the Q.K^T of the item before have executed
      constexpr int kPieces = D / 8;
      const int g_ = it.s.group;
      int64_t off = 0;
      if (lane < it.s.nrows) {
        if (it.s.causal) {
          const int x = lane / g_;
          off = (int64_t)(it.rows_at + x) * p.sq_t + (int64_t)(it.qhead + lane - x * g_) * p.sq_h;
        } else {
          off = entry_qoff(p, sa.iq, __ldg(a.row_list + it.rows_at + lane));
        }
      }
#pragma unroll
      for (int i = lane; i < kFewRows * kPieces; i += 32) {
        const int r = i / kPieces, ch = i % kPieces;
        const int64_t o = __shfl_sync(0xffffffffu, off, r);
        cp_async_16(sQ + (uint32_t)((ch >> 3) * kFewBlock + r * 128 + (((ch & 7) ^ (r & 7)) << 4)), a.q + o + ch * 8);
      }
      cp_async_mbar_arrive(smem_u32(&c.q_full));
    };
    static_assert(kFewRows * (D / 8) % 32 == 0, "whole warps copy");
    auto qk = [&](bool first, bool last) {
      if (first) {
        if (items > 1 && !wait(&c.q_free, (items - 2) & 1)) return;
        copy_q();
        if (!wait(&c.q_full, (items - 1) & 1)) return;
        fence_proxy_async_smem();                             // rows written by cp.async, read by the tensor core
      }
      const int st = at % kStages;
      if (!wait(&c.full[st], (at / kStages) & 1)) return;
      ++at;
      tc_fence_after();
      const uint32_t k = dk + (uint32_t)st * (kTileBytes >> 4);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        mma_ss_el<kDescHi>(el, tm + (uint32_t)(g & 1) * kFewN, k + (uint32_t)((ks >> 2) * (kHalfBytes >> 4) + (ks & 3) * 2),
                           dq + (uint32_t)((ks >> 2) * (kFewBlock >> 4) + (ks & 3) * 2), kIdescFewQK<kHalf>, ks > 0);
      tc_commit_el(el, smem_u32(&c.s_full[g & 1]));
      tc_commit_el(el, smem_u32(&c.empty[st]));
      if (last) tc_commit_el(el, smem_u32(&c.q_free));
      ++g;
    };
    auto pv = [&](int m, bool first, bool last) {             // m: tile, of all items
      const int st = at % kStages;
      if (!wait(&c.full[st], (at / kStages) & 1)) return;
      ++at;
      if (!wait(&c.p_full, m & 1)) return;
      tc_fence_after();
      const uint32_t v = dv + (uint32_t)st * (kTileBytes >> 4);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        mma_ss_el<kDescHi>(el, tm + kO, v + ks * (2048 >> 4), dp + (uint32_t)((ks >> 2) * (kFewBlock >> 4) + (ks & 3) * 2),
                           kIdescFewPV<kHalf>, !first || ks > 0);
      tc_commit_el(el, smem_u32(&c.pv_done));
      tc_commit_el(el, smem_u32(&c.empty[st]));
      if (last) tc_commit_el(el, smem_u32(&c.o_full));
    };
    bool pending = false, p_first = false, p_last = false;    // P.V of the tile whose Q.K^T was issued last
#pragma unroll 1
    while (ok && next_item()) {
      const int n = tiles_of();
#pragma unroll 1
      for (int j = 0; j < n && ok; ++j) {
        qk(j == 0, j + 1 == n);
        if (!ok) break;
        if (pending) pv(g - 2, p_first, p_last);
        pending = true;
        p_first = j == 0;
        p_last = j + 1 == n;
      }
    }
    if (ok && pending) pv(g - 1, p_first, p_last);
    if (!ok && lane == 0) { atomicExch(a.status, ST_MMA); c.abort = 1; }
  } else if (warp == 4) {
    // ---- row sums: four lanes a row, each with every fourth key of the tile
    const int q = lane >> 2, r = lane & 3;
    int g = 0;
    while (ok && next_item()) {
      const int n = tiles_of();
      float l = 0.f;
      for (int j = 0; j < n; ++j, ++g) {
        if (!wait(&c.p_full, g & 1)) break;
        float x[kBN / 4];
#pragma unroll
        for (int i = 0; i < kBN / 4; ++i) x[i] = c.p32[q][r + 4 * i];
        const float alpha = c.alpha[g & 1][q];
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < kBN / 4; ++i) acc = __fadd_rn(acc, x[i]);
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 2));
        acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, 1));
        l = __fadd_rn(__fmul_rn(l, alpha), acc);
        if (r == 0) c.row_sum[q] = l;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&c.sum_done));
      }
    }
    if (!ok && lane == 0) { atomicExch(a.status, ST_SOFTMAX); c.abort = 1; }
  } else {
    // ---- softmax, one thread per key; epilogue, one thread per dim
    const int key = threadIdx.x;           // of the tile; and dim
    const uint32_t tl = tmem + ((uint32_t)(warp * 32) << 16);
    const float sl2 = rsqrtf((float)D) * 1.4426950408889634f;
    const bool poly = ((key >> 1) & 7) < kPolyPairs;           // this key's exponentials are the cubic's
    unsigned char* const p_at = smem + (sP - sKV) + (key >> 6) * kFewBlock + (key & 7) * 2;
    int g = 0;
    uint32_t xph = 0;                      // phase of `exchange`
    // largest of x[r] over the four warps, for all rows
    auto all_max = [&](float (&x)[kFewRows], int nrows) {
      const int buf = xph;
#pragma unroll
      for (int r = 0; r < kFewRows; ++r)
        if (r < nrows) {
          const float m = redux_max(x[r]);
          if (lane == 0) c.warp_max[buf][r][warp] = m;
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c.exchange));
      if (!wait(&c.exchange, xph)) return;
      xph ^= 1;
#pragma unroll
      for (int r = 0; r < kFewRows; ++r)
        if (r < nrows) {
          const float4 m = *reinterpret_cast<const float4*>(c.warp_max[buf][r]);
          x[r] = fmaxf(fmaxf(m.x, m.y), fmaxf(m.z, m.w));
        }
    };
    while (ok && next_item()) {
      const int nrows = it.s.nrows, kv_len = it.s.kv_len, group = it.s.group, rows_at = it.rows_at, qhead = it.qhead;
      const bool causal = it.s.causal != 0;
      const int tok_rel = it.s.tok_rel;
      const int n = tiles_of();
      float m_ref[kFewRows];
      int lim[kFewRows];                   // keys < lim are visible to the row
#pragma unroll
      for (int r = 0; r < kFewRows; ++r) {
        m_ref[r] = -INFINITY;
        lim[r] = causal ? min(kv_len, tok_rel + r / group + 1) : kv_len;
      }
      for (int j = 0; j < n; ++j, ++g) {
        if (!wait(&c.s_full[g & 1], (g >> 1) & 1)) break;
        tc_fence_after();
        uint32_t v[kFewRows];
        tmem_ld8(tl + (uint32_t)(g & 1) * kFewN, v);
        tmem_wait_ld();
        float x[kFewRows];
        const int at = j * kBN + key;
#pragma unroll
        for (int r = 0; r < kFewRows; ++r) {
          if (at >= lim[r]) v[r] = 0xff800000u;                // -inf
          x[r] = __uint_as_float(v[r]);
        }
        all_max(x, nrows);
        if (!ok) break;
        bool any = false;
        float alpha[kFewRows];
#pragma unroll
        for (int r = 0; r < kFewRows; ++r) {
          alpha[r] = 1.f;
          if (r < nrows) {
            const float m_new = fmaxf(m_ref[r], x[r] * sl2);
            if (m_new > m_ref[r] + 8.f) {
              alpha[r] = ex2_approx(m_ref[r] - m_new);
              m_ref[r] = m_new;
              any = true;
            }
          }
        }
        // P.V of the tile before has run: O may be rescaled and P overwritten; the tile's sums are done: so may the exponentials
        if (g > 0 && (!wait(&c.pv_done, (g - 1) & 1) || !wait(&c.sum_done, (g - 1) & 1))) break;
        if (any && j > 0) {
          tc_fence_after();
          uint32_t o[kFewRows];
          tmem_ld8(tl + kO, o);
          tmem_wait_ld();
#pragma unroll
          for (int r = 0; r < kFewRows; ++r) o[r] = __float_as_uint(__uint_as_float(o[r]) * alpha[r]);
          tmem_st8(tl + kO, o);
          tmem_wait_st();
        }
        if (key == 0) {
#pragma unroll
          for (int r = 0; r < kFewRows; ++r) c.alpha[g & 1][r] = alpha[r];
        }
#pragma unroll
        for (int r = 0; r < kFewRows; r += 2) {
          if (r < nrows) {
            const uint64_t y = fma2(pack2(__uint_as_float(v[r]), __uint_as_float(v[r + 1])), pack2(sl2, sl2),
                                    pack2(-m_ref[r], -m_ref[r + 1]));
            const uint64_t cubic = ex2_poly2(y);
            const float e0 = poly ? lo2(cubic) : ex2_approx(lo2(y)), e1 = poly ? hi2(cubic) : ex2_approx(hi2(y));
            const uint32_t pk = pack2_16<kHalf>(e0, e1);
            c.p32[r][key] = e0;
            c.p32[r + 1][key] = e1;
            unsigned char* dst = p_at + r * 128;
            *reinterpret_cast<uint16_t*>(dst + ((((key & 63) >> 3) ^ r) << 4)) = (uint16_t)pk;
            *reinterpret_cast<uint16_t*>(dst + 128 + ((((key & 63) >> 3) ^ (r + 1)) << 4)) = (uint16_t)(pk >> 16);
          }
        }
        fence_proxy_async_smem();                              // P, read by the tensor core
        tc_fence_before();
        mbar_arrive(smem_u32(&c.p_full));
      }
      if (!ok || !wait(&c.o_full, (items - 1) & 1) || !wait(&c.sum_done, (g - 1) & 1)) break;
      tc_fence_after();
      uint32_t o[kFewRows];
      tmem_ld8(tl + kO, o);
      tmem_wait_ld();
      tc_fence_before();
      float amax[kFewRows];
#pragma unroll
      for (int r = 0; r < kFewRows; ++r) amax[r] = fabsf(__uint_as_float(o[r]));
      all_max(amax, nrows);
      if (!ok) break;
#pragma unroll
      for (int r = 0; r < kFewRows; ++r)
        if (r < nrows) {
          const int xg = r / group;
          const int32_t e = causal ? (int32_t)(((int64_t)(rows_at + xg) * p.Hq + qhead + r - xg * group) * p.NP)
                                   : __ldg(a.row_list + rows_at + r);
          const float l = c.row_sum[r];
          const float inv = 1.f / l;
          // the row's largest magnitude decides the power of two its fp16 copy is scaled by
          const PartialScale ps = partial_scale(fmaxf(amax[r], 0.f) * inv);
          if (D == 128 || key < D) a.partial_out[(int64_t)e * D + key] = __float2half_rn(__uint_as_float(o[r]) * (inv * ps.scale));
          if (key == r) a.partial_lse[e] = make_float2((m_ref[r] + log2f(l)) * 0.6931471805599453f, ps.inv);
        }
      // (the sums of the next item are written behind a p_full that these threads arrive on)
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
  if (warp == 6) tmem_dealloc(tmem, kCols);
}

}  // namespace

cudaError_t launch_attend_few_tc5(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                                  const int32_t* cu, const int32_t* list_counts, const int32_t* list_offsets,
                                  const int32_t* tile_prefix, const int32_t* row_list, __half* partial_out,
                                  float2* partial_lse, int32_t* work_counter, int32_t* status, int sms, cudaStream_t st) {
  CUtensorMap mk, mv;
  if (!make_kv_map(&mk, p.fp16 != 0, p.D, k, p.T, p.Hkv, p.sk_t, p.sk_h, kBN) ||
      !make_kv_map(&mv, p.fp16 != 0, p.D, v, p.T, p.Hkv, p.sv_t, p.sv_h, kBN))
    return cudaErrorNotSupported;
  ShortArgs sa;
  sa.a = KernelArgs{q, cu, list_counts, list_offsets, tile_prefix, row_list, partial_out, partial_lse,
                    work_counter, status, 0};
  sa.iq = item_queue(p, cu, list_counts, list_offsets, tile_prefix, row_list, work_counter, 1, true, 0);
  // As many CTAs as there can be items, up to two per SM.  Where one per SM is enough, each has twice the tiles in flight
  const int ctas = window_ctas(p, 2 * sms);
  const bool one = ctas <= sms;
  auto kern = p.D == 128 ? (p.fp16 ? (one ? attend_tc5_few_kernel<true, 128, 6> : attend_tc5_few_kernel<true, 128, 3>)
                                   : (one ? attend_tc5_few_kernel<false, 128, 6> : attend_tc5_few_kernel<false, 128, 3>))
                         : (p.fp16 ? (one ? attend_tc5_few_kernel<true, 96, 6> : attend_tc5_few_kernel<true, 96, 3>)
                                   : (one ? attend_tc5_few_kernel<false, 96, 6> : attend_tc5_few_kernel<false, 96, 3>));
  const size_t smem = one ? few_smem_bytes<6>() : few_smem_bytes<3>();
  const cudaError_t e = prepare_kernel(kern, smem);
  if (e != cudaSuccess) return e;
  return launch_pdl(kern, dim3(ctas), kFewThreads, smem, st, p, mk, mv, sa);
}

}  // namespace moba
