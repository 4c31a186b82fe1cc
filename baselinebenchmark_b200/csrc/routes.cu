// Compaction of the per-(token, head) selections into per-(chunk slot, kv head)
// query lists, and the LSE-weighted merge of the partial results.
//
// Replaces, for the inference path of the reference,
//   _count_sparse_routes_kernel / _exclusive_prefix_sum_triton /
//   _scatter_sparse_routes_device_kernel / _build_route_block_descriptors_kernel
//                              backends/_mthreads/ops/moba/routing.py:1311-1429, 1561-1718
//   _fused_merge_softmax_kernel                      attention.py:787-889
//
// Differences by design: lists are keyed by (slot, kv head) so the query heads
// of a GQA group share one K/V stream; all ranks are compacted at once (the
// reference loops over rank passes, parallel.py:335); tile descriptors are not
// materialised, the dense stage finds its tile by binary search in a prefix of
// tile counts; the merge sees every partial of a row at once and rounds once.
#include "common.cuh"

namespace moba {

// ---------------------------------------------------------------------------
// rows of an append: a 16-byte piece of K and of V per thread
// ---------------------------------------------------------------------------
constexpr int kAppendThreads = 256;

__global__ void __launch_bounds__(kAppendThreads)
append_rows_kernel(Params p, const __nv_bfloat16* __restrict__ k_new, const __nv_bfloat16* __restrict__ v_new,
                   int64_t kn_t, int64_t kn_h, int64_t vn_t, int64_t vn_h, __nv_bfloat16* __restrict__ k,
                   __nv_bfloat16* __restrict__ v, int32_t* __restrict__ cu) {
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) { cu[0] = 0; cu[1] = (int32_t)p.T; }
  const int pieces = p.D / 8;
  const int64_t total = p.Tq * p.Hkv * pieces;
  for (int64_t i = (int64_t)blockIdx.x * kAppendThreads + threadIdx.x; i < total; i += (int64_t)gridDim.x * kAppendThreads) {
    const int64_t r = i / pieces;
    const int c = (int)(i - r * pieces) * 8;
    const int64_t t = r / p.Hkv;
    const int64_t h = r - t * p.Hkv;
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(k_new + t * kn_t + h * kn_h + c));
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(v_new + t * vn_t + h * vn_h + c));
    *reinterpret_cast<uint4*>(k + (p.win_lo + t) * p.sk_t + h * p.sk_h + c) = a;
    *reinterpret_cast<uint4*>(v + (p.win_lo + t) * p.sv_t + h * p.sv_h + c) = b;
  }
}

cudaError_t launch_append_rows(const Params& p, const __nv_bfloat16* k_new, const __nv_bfloat16* v_new, int64_t kn_t,
                               int64_t kn_h, int64_t vn_t, int64_t vn_h, __nv_bfloat16* k, __nv_bfloat16* v,
                               int32_t* cu, cudaStream_t st) {
  int64_t blocks = (p.Tq * p.Hkv * (p.D / 8) + kAppendThreads - 1) / kAppendThreads;
  if (blocks > 148 * 16) blocks = 148 * 16;
  return launch_pdl(append_rows_kernel, dim3((unsigned)blocks), kAppendThreads, 0, st, p, k_new, v_new, kn_t, kn_h, vn_t,
                    vn_h, k, v, cu);
}

// ---------------------------------------------------------------------------
// exclusive prefix sums over the lists (single CTA, any number of lists)
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads) scan_lists_kernel(const ListScan a) {
  pdl_wait();
  pdl_trigger();
  __shared__ int scratch[2 * kScanThreads / 32];
  scan_lists<kScanThreads, 1>(a, scratch);
}

// ---------------------------------------------------------------------------
// scatter: grid (token tiles of one sequence, kv head, sequence), like the
// gating kernel, so a CTA touches the lists of one (sequence, kv head) only and
// can reserve list space with one global atomic per list.
// ---------------------------------------------------------------------------
constexpr int kScatterThreads = 256;
constexpr int kScatterTokens = 64;

__global__ void __launch_bounds__(kScatterThreads)
scatter_routes_kernel(Params p, const int32_t* __restrict__ cu, const int32_t* __restrict__ selected,
                      const int32_t* __restrict__ offsets, int32_t* __restrict__ cursors,
                      int32_t* __restrict__ row_list, float2* __restrict__ partial_lse) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ int32_t sm[];
  int32_t* cnt_s = sm;               // [mc] rows of this CTA per list, then running index
  int32_t* base_s = sm + p.mc;       // [mc] first position reserved for this CTA
  const int b = blockIdx.z, hk = blockIdx.y;
  const int s0 = cu[b], s1 = cu[b + 1];
  const int x = blockIdx.x + window_tile0(p, s0, kScatterTokens);
  const int tok_lo = max(s0 + x * kScatterTokens, p.win_lo);
  const int tok_hi = min(min(s0 + (x + 1) * kScatterTokens, s1), p.win_lo + (int)p.Tq);
  if (tok_lo >= tok_hi) return;
  const int ntok = tok_hi - tok_lo;
  const int loc = tok_lo - p.win_lo;             // window-relative token of the first row
  const int slot0 = b * p.mc;
  const int n = p.hist * p.G * ntok;             // entries (rank, head, token), token fastest
  for (int i = threadIdx.x; i < p.mc; i += kScatterThreads) cnt_s[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kScatterThreads) {
    const int tl = i % ntok, rh = i / ntok;
    const int hl = rh % p.G, r = rh / p.G;
    const int slot = selected[(int64_t)r * p.sel_rs + (int64_t)(hk * p.G + hl) * p.Tq + loc + tl];
    if (slot >= 0) atomicAdd(&cnt_s[slot - slot0], 1);
  }
  __syncthreads();
  for (int c = threadIdx.x; c < p.mc; c += kScatterThreads) {
    const int m = cnt_s[c];
    base_s[c] = m > 0 ? atomicAdd(&cursors[(int64_t)(slot0 + c) * p.Hkv + hk], m) : 0;
    cnt_s[c] = 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kScatterThreads) {
    const int tl = i % ntok, rh = i / ntok;
    const int hl = rh % p.G, r = rh / p.G;
    const int head = hk * p.G + hl;
    const int slot = selected[(int64_t)r * p.sel_rs + (int64_t)head * p.Tq + loc + tl];
    const int64_t entry = ((int64_t)(loc + tl) * p.Hq + head) * p.NP + r + 1;
    if (slot >= 0) {
      const int c = slot - slot0;
      const int pos = offsets[(int64_t)slot * p.Hkv + hk] + base_s[c] + atomicAdd(&cnt_s[c], 1);
      row_list[pos] = (int32_t)entry;
    } else {
      partial_lse[entry] = make_float2(-INFINITY, 0.f);   // this rank contributes nothing to the merge
    }
  }
}

cudaError_t launch_compact(const Params& p, const int32_t* cu, const int32_t* selected,
                           const int32_t* list_counts, int32_t* list_offsets, int32_t* tile_prefix,
                           int32_t* cursors, int32_t* row_list, float2* partial_lse, int tile_rows,
                           cudaStream_t st) {
  const ListScan scan{list_counts, list_offsets, tile_prefix, cursors, p.lists, tile_rows};
  const cudaError_t e = launch_pdl(scan_lists_kernel, dim3(1), kScanThreads, 0, st, scan);
  if (e != cudaSuccess) return e;
  return launch_scatter(p, cu, selected, list_offsets, cursors, row_list, partial_lse, st);
}

cudaError_t launch_scatter(const Params& p, const int32_t* cu, const int32_t* selected, const int32_t* list_offsets,
                           int32_t* cursors, int32_t* row_list, float2* partial_lse, cudaStream_t st) {
  const size_t smem = (size_t)p.mc * 2 * sizeof(int32_t);
  if (smem > 200 * 1024) return cudaErrorInvalidConfiguration;
  if (smem > 48 * 1024) {
    const cudaError_t e = prepare_kernel(scatter_routes_kernel, smem);
    if (e != cudaSuccess) return e;
  }
  dim3 grid(window_tiles(p, kScatterTokens), p.Hkv, p.B);
  return launch_pdl(scatter_routes_kernel, grid, kScatterThreads, smem, st, p, cu, selected, list_offsets, cursors,
                    row_list, partial_lse);
}

// ---------------------------------------------------------------------------
// merge: a (token, head) row is combined by D / 8 lanes (rounded up to a power of two: one row a warp at
// head dim 256, two at 128 and 96, four at 64), or, from 17 partials on, by a whole warp.
//   lse_tot = log sum_j exp(lse_j);  out = sum_j O_j * exp(lse_j - lse_tot)
// (exponentials through ex2.approx: relative error 2^-22, far below the rounding of the output)
// Bound by HBM by bytes, with few partials in practice by issue slots: a whole warp per row spends as many
// instructions on reducing a handful of LSEs and adding its groups' sums as on the partial rows.  With many it
// reads more of a row in one go, and 64 LSEs fit its registers.  Measured, us, 131072 rows:
//   partials                  3     8    16    32    64
//   head dim 128, rows of 16 lanes   34.5  63.6   107     -     -
//                 rows of a warp     62.9  70.3   105   179   333
//   head dim 64,  rows of 8 lanes    17.7  35.5  61.3     -     -
//                 rows of a warp     52.4  64.0  71.4   105   180
// (reading the LSEs again for each partial where they do not fit the registers: 209 / 812 us at 128 with 32 / 64,
// 236 / 451 at 64), so the line lies at 16.  A row must come out the same bits however many chunks max_seqlen allows
// for, and the two add its partials in different orders.  So a top-k above 16 with few partials also runs on a
// part of a warp, but with the sums of the other's groups (kSums of them, added up in its order).
// ---------------------------------------------------------------------------
constexpr int kMergeThreads = 256;
constexpr int kMergeNarrow = 16;                 // most partials of a row on a part of a warp

// A partial row is D/8 pieces of eight fp16 values (16 bytes), one per lane of a group of lanes.  A row has
// kW lanes: one group, which takes the partials of the row in turn, or all 32 lanes of a warp, whose groups take
// every second (head dim 96, 128) or fourth (64) partial and add their sums at the end.
// kAhead partials of a group are in flight, kPairs LSEs in each lane.  kSums: sums a group keeps, partial j in sum
// j mod kSums.
template <int D> constexpr int kMergeGroup = D <= 64 ? 8 : D <= 128 ? 16 : 32;
template <bool kHalf, int D, int kW, int kPairs, int kAhead, int kCtas, int kSums = 1>
__global__ void __launch_bounds__(kMergeThreads, kCtas)
merge_kernel(Params p, const __half* __restrict__ partial_out, const float2* __restrict__ partial_lse,
             const int32_t* __restrict__ status, __nv_bfloat16* __restrict__ out, float* __restrict__ lse_out, int trigger) {
  pdl_wait();
  if (trigger) pdl_trigger();                    // see launch_chained
  constexpr int kGroup = kMergeGroup<D>, kGroups = kW / kGroup;
  constexpr int kPieces = D / 8;                 // lanes of a group that hold data (head dim 96: 12 of 16)
  constexpr int kRowsPerBlock = kMergeThreads / kW;
  static_assert(kPairs == 1 || kPairs == 2, "LSEs of a lane");
  static_assert(kW % (kGroups * kAhead) == 0, "the partials of a round lie on one side of kW");
  static_assert(kAhead % kSums == 0 && (kSums == 1 || kGroups == 1), "sums by the place in a round");
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kW - 1);               // lane of the row
  const int grp = sub / kGroup, piece = sub & (kGroup - 1);
  const unsigned base_lane = lane & ~(kW - 1);
  // a dense stage that gave up on a wait leaves a non-zero status: poison the result
  const bool failed = status != nullptr && *status != 0;
  const int64_t stride = (int64_t)gridDim.x * kRowsPerBlock;
  // Lane j holds {lse, 1 / scale} of the partials j and j + kW (there are at most kPairs * kW), and the pairs
  // of the next row are requested before this row is worked on, so that a row starts with its
  // partial rows as the only loads it has to wait for.
  int64_t row = (int64_t)blockIdx.x * kRowsPerBlock + threadIdx.x / kW;
  const float2 none = make_float2(-INFINITY, 0.f);
  float2 next0 = none, next1 = none;
  auto fetch = [&](int64_t r) {
    next0 = none;
    next1 = none;
    if (r < p.rows) {
      if (sub < p.NP) next0 = __ldg(partial_lse + r * p.NP + sub);
      if (kPairs > 1 && sub + kW < p.NP) next1 = __ldg(partial_lse + r * p.NP + sub + kW);
    }
  };
  fetch(row);
  // the rows of a warp end together: a row past the end is worked on without loads or stores
  for (int64_t row0 = row - threadIdx.x / kW + (threadIdx.x >> 5) * (32 / kW); row0 < p.rows; row0 += stride, row += stride) {
    const bool real = row < p.rows;
    const float2 cur0 = next0, cur1 = next1;
    fetch(row + stride);
    float mx = kPairs > 1 ? fmaxf(cur0.x, cur1.x) : cur0.x;
#pragma unroll
    for (int o = kW / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e0 = __expf(cur0.x - mx), e1 = kPairs > 1 ? __expf(cur1.x - mx) : 0.f;   // 0 past the partials (lse -inf)
    float tot = e0 + e1;
#pragma unroll
    for (int o = kW / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const float inv = failed ? __int_as_float(0x7fc00000) : 1.f / tot;
    // weights of this lane's partials; the row's power-of-two scale is undone with them
    const float w0 = e0 * cur0.y * inv, w1 = kPairs > 1 ? e1 * cur1.y * inv : 0.f;
    float2 sums[kSums][4];
#pragma unroll
    for (int a = 0; a < kSums; ++a)
#pragma unroll
      for (int i = 0; i < 4; ++i) sums[a][i] = make_float2(0.f, 0.f);
    const uint4* src = reinterpret_cast<const uint4*>(partial_out + row * p.NP * D) + piece;
#pragma unroll 1
    for (int j0 = 0; j0 < p.NP; j0 += kGroups * kAhead) {
      float w[kAhead];
      uint4 o[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int j = j0 + u * kGroups + grp;
        o[u] = make_uint4(0u, 0u, 0u, 0u);
        w[u] = 0.f;
        // Rows of a warp: a branch, the same for all lanes (head dim 128, 32 partials: 205 us with the loads
        // predicated only, 179 with it).  Rows of a part of it have no such branch (8 partials: 64 against 85).
        if (kW < 32 || j0 + u * kGroups < p.NP) {
          w[u] = __shfl_sync(0xffffffffu, kPairs == 1 || j0 < kW ? w0 : w1, base_lane + (j & (kW - 1)));
          // (a weight of NaN marks a failed dense stage: it must reach the sum, but the row is not read)
          if (real && j < p.NP && piece < kPieces && w[u] != 0.f && !failed) o[u] = __ldg(src + j * kPieces);
        }
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const uint32_t words[4] = {o[u].x, o[u].y, o[u].z, o[u].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&words[i]));
          sums[u % kSums][i].x += w[u] * a.x;
          sums[u % kSums][i].y += w[u] * a.y;
        }
      }
    }
    // the sums of a group, and of the groups
#pragma unroll
    for (int o = kSums / 2; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < o; ++a)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sums[a][i].x += sums[a + o][i].x;
          sums[a][i].y += sums[a + o][i].y;
        }
    float2(&acc)[4] = sums[0];
#pragma unroll
    for (int o = kW / 2; o >= kGroup; o >>= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i].x += __shfl_xor_sync(0xffffffffu, acc[i].x, o);
        acc[i].y += __shfl_xor_sync(0xffffffffu, acc[i].y, o);
      }
    const int64_t t = row / p.Hq;
    const int h = (int)(row - t * p.Hq);
    if (real && grp == 0 && piece < kPieces) {
      uint4 pk;
      pk.x = pack2_16<kHalf>(acc[0].x, acc[0].y);
      pk.y = pack2_16<kHalf>(acc[1].x, acc[1].y);
      pk.z = pack2_16<kHalf>(acc[2].x, acc[2].y);
      pk.w = pack2_16<kHalf>(acc[3].x, acc[3].y);
      *reinterpret_cast<uint4*>(out + t * p.so_t + (int64_t)h * p.so_h + piece * 8) = pk;
    }
    if (real && lse_out != nullptr && sub == 0) lse_out[(int64_t)h * p.Tq + t] = logf(tot) + mx;
  }
}

template <bool kHalf, int D>
static cudaError_t launch_merge_dim(const Params& p, const __half* partial_out, const float2* partial_lse,
                                    const int32_t* status, __nv_bfloat16* out, float* lse_out, cudaStream_t st, bool trigger) {
  auto launch = [&](auto* kernel, int lanes) {
    const int rows_per_block = kMergeThreads / lanes;
    int64_t blocks = (p.rows + rows_per_block - 1) / rows_per_block;
    if (blocks > 148 * 64) blocks = 148 * 64;
    const bool chained = p.rows * p.NP * D * (int64_t)sizeof(__half) <= kChainedMergeBytes;
    return launch_chained(chained, kernel, dim3((unsigned)blocks), kMergeThreads, 0, st, p, partial_out, partial_lse, status,
                          out, lse_out, (int)trigger);
  };
  constexpr int kGroup = kMergeGroup<D>, kSums = 32 / kGroup;
  const bool many = p.topk > kMergeNarrow;                   // (few partials of a top-k whose rows are on a warp elsewhere)
  if constexpr (D == 64) {
    // Eight partials in flight up to three waves of rows, where a row's own latency counts (16 partials: 11200 rows 5.3
    // against 6.5 us with four), four and more CTAs from there on (131072 rows: 61 against 68).
    if (p.NP <= kMergeNarrow) {
      if (p.rows <= 148 * 3 * 3 * (kMergeThreads / kGroup))
        return many ? launch(merge_kernel<kHalf, D, kGroup, 2, 4, 3, kSums>, kGroup) : launch(merge_kernel<kHalf, D, kGroup, 2, 8, 3>, kGroup);
      return many ? launch(merge_kernel<kHalf, D, kGroup, 2, 4, 4, kSums>, kGroup) : launch(merge_kernel<kHalf, D, kGroup, 2, 4, 5>, kGroup);
    }
  } else if constexpr (D < 256) {
    // two sums leave four CTAs: ahead of a warp per row up to 8 partials (3: 40 against 63 us, 8: 72 against 70, 16: 117 / 105)
    if (many && p.NP <= kMergeNarrow / 2) return launch(merge_kernel<kHalf, D, kGroup, 1, 4, 4, kSums>, kGroup);
    // (eight in flight for one wave of rows: 16 partials, 256 rows 3.6 against 4.3 us; 8, 11200 rows 6.1 against 5.5)
    if (!many)
      return p.rows <= 148 * 3 * (kMergeThreads / kGroup) ? launch(merge_kernel<kHalf, D, kGroup, 1, 8, 3>, kGroup)
                                                         : launch(merge_kernel<kHalf, D, kGroup, 1, 4, 5>, kGroup);
  } else {
    // one LSE a lane leaves registers for a fifth CTA (131072 rows, 32 partials: 335 -> 323 us)
    if (p.NP <= 32) return launch(merge_kernel<kHalf, D, 32, 1, 4, 5>, 32);
  }
  return launch(merge_kernel<kHalf, D, 32, 2, 4, 4>, 32);
}

cudaError_t launch_merge(const Params& p, const __half* partial_out, const float2* partial_lse,
                         const int32_t* status, __nv_bfloat16* out, float* lse_out, cudaStream_t st, bool trigger) {
#define MOBA_MERGE(DIM)                                                                                          \
  return p.fp16 ? launch_merge_dim<true, DIM>(p, partial_out, partial_lse, status, out, lse_out, st, trigger)    \
                : launch_merge_dim<false, DIM>(p, partial_out, partial_lse, status, out, lse_out, st, trigger)
  switch (p.D) {
    case 64: MOBA_MERGE(64);
    case 96: MOBA_MERGE(96);
    case 128: MOBA_MERGE(128);
    case 256: MOBA_MERGE(256);
    default: return cudaErrorInvalidValue;
  }
#undef MOBA_MERGE
}

}  // namespace moba
