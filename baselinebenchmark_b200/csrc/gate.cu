// Gating stage of MoBA: chunk slot tables, mean-pooled keys, q.mean scores with
// the causal chunk mask and a per-(token, head) top-k.
//
// Replaces, for the inference path of the reference,
//   _dense_chunk_metadata_kernel            backends/_mthreads/ops/moba/routing.py:553-592
//   _dense_chunk_mean_kernel                routing.py:690-737
//   _chunk_topk_batched_streaming_kernel    routing.py:1056-1182
//
// K and Q are read once.  The selection is defined by one fixed fp32 summation
// order, so that a CPU restatement reproduces it bit for bit; the scores of all
// candidates are first estimated on the tensor core and only the candidates the
// estimate cannot rank with certainty are evaluated in that order (see the
// scores section below):
//   mean : row r of a chunk is added to accumulator r % 32 in increasing r, the
//          32 accumulators are added in increasing index, the total is divided
//          by C and rounded to bf16 (round to nearest even);
//   score: products of two 16-bit values are exact in fp32; each block of 8
//          dims is added left to right, then a halving tree combines the D/8
//          block sums (for D = 128: block l + block l+8, then l + l+4, l + l+2,
//          l + l+1); a block count that is no power of two (D = 96) is padded
//          with blocks of +0.0 to the next one.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "topk_network.cuh"

namespace moba {

// ---------------------------------------------------------------------------
// slot tables
// ---------------------------------------------------------------------------
__global__ void chunk_metadata_kernel(Params p, const int32_t* __restrict__ cu,
                                      int32_t* __restrict__ cu_chunk,
                                      int32_t* __restrict__ chunk_end,
                                      int8_t* __restrict__ valid) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) cu_chunk[p.slots] = cu[p.B];
  if (s >= p.slots) return;
  const int b = s / p.mc, j = s - b * p.mc;
  const Slot sl = slot_of(cu, b, j, p.C);
  cu_chunk[s] = sl.start;
  chunk_end[s] = sl.historical ? sl.end : 0;
  valid[s] = sl.historical ? 1 : 0;
}

cudaError_t launch_chunk_metadata(const Params& p, const int32_t* cu, int32_t* cu_chunk,
                                  int32_t* chunk_end, int8_t* valid, cudaStream_t st) {
  const int threads = 256;
  chunk_metadata_kernel<<<cdiv_i(p.slots, threads), threads, 0, st>>>(p, cu, cu_chunk, chunk_end, valid);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// chunk means: one CTA per (slot, kv head), 32 row lanes x D/8 dim lanes (16-byte loads), or, when
// that leaves the chip mostly idle (few long chunks, or the one chunk a decode step completes), one
// CTA per 32 dims of it with four times the rows in flight.  A row lane adds its C / 32 rows
// one after the other (the order is the contract's), so what a long chunk waits for is the latency of that
// chain: kAhead rows of it are in flight.  Measured: one 4096-key chunk x 8 heads of a decode step 50 -> 20 us; the
// seven of a 32768-token sequence 58 -> 54 us, where 56 CTAs were enough to half fill HBM.
// kCtas: CTAs per SM the registers are held to.  Many short chunks (a CTA adds one or two rows a lane) want all of an
// SM's threads resident: at head dim 64, 42 registers left five CTAs instead of eight (2048 chunks of 64 keys x
// 16 heads 107 us, 80 with 32).  Few long ones want their loads in flight: with 512 CTAs on chunks of 4096 keys, 268 MB,
// a call took 340 us with 32 registers, 330 with 54.  So 32 it is where more CTAs come than fit with 48.
// Split over the dims, 64 registers (eight CTAs) hold ten rows; 106 held sixteen, in four CTAs.
// Where even that leaves most SMs without a CTA (the chunk a decode step completes), 16 dims a CTA, 8 bytes a load and 64 rows in
// flight: all of a 4096-key chunk is requested in two goes.  One 4096-key chunk x 8
// heads, whole decode step 114 -> 107 us (kernel 14.3 -> 8.3), x 16 heads 105 -> 98, x 4 heads at head dim 256 113 -> 110; chunks of
// 1024 (65536 tokens) 56.7 -> 55.5, of 2048 55.7 -> 55.3.  From 16 rows a lane on: shorter chains are one round either way.
// Head dim 256: 64 dims a CTA.  With all of them its 1024 threads were two CTAs to an SM, which loaded and added up in step: 8192 tokens x
// 16 heads, chunk 128 26.6 -> 20.4 us, 40000 x 8, chunk 1024 45.1 -> 41.0 (at 128 dims it makes no difference).
// kVec: dims of a load.
// ---------------------------------------------------------------------------
template <int D> constexpr int kMeanDims = D < 256 ? D : 64;
template <int kVec> struct MeanLoad;
template <> struct MeanLoad<8> { using T = uint4; };
template <> struct MeanLoad<4> { using T = uint2; };
template <bool kHalf>
__device__ __forceinline__ void unpack_mean(const uint4 x, float (&f)[8]) { unpack8<kHalf>(x, f); }
template <bool kHalf>
__device__ __forceinline__ void unpack_mean(const uint2 x, float (&f)[4]) {
  const float2 a = unpack2<kHalf>(x.x), b = unpack2<kHalf>(x.y);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}
template <bool kHalf, int D, int kDims, int kAhead, int kCtas, int kVec = 8>
__global__ void __launch_bounds__(kMeanLanes * (kDims / kVec), kCtas)
chunk_mean_kernel(Params p, int slot_begin, const __nv_bfloat16* __restrict__ k, const int32_t* __restrict__ cu,
                  __nv_bfloat16* __restrict__ means, int32_t* __restrict__ zero, int64_t zero_words) {
  pdl_wait();
  pdl_trigger();
  // the counters that the kernels behind this one add to
  for (int64_t i = (((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
       i < zero_words; i += (int64_t)gridDim.x * gridDim.y * gridDim.z * blockDim.x)
    zero[i] = 0;
  const int slot = slot_begin + blockIdx.x, hk = blockIdx.y, dim0 = blockIdx.z * kDims;
  const int b = slot / p.mc, j = slot - b * p.mc;
  const Slot sl = slot_of(cu, b, j, p.C);
  constexpr int kDimLanes = kDims / kVec;
  using Load = typename MeanLoad<kVec>::T;
  const int dl = threadIdx.x % kDimLanes;  // dims dim0 + kVec * dl ...
  const int rl = threadIdx.x / kDimLanes;  // row lane 0..31
  __nv_bfloat16* dst = means + ((int64_t)slot * p.Hkv + hk) * D + dim0;

  __shared__ float part[kMeanLanes][kDims + 4];
  float acc[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) acc[i] = 0.f;

  if (sl.historical) {                     // historical chunks are always full: C rows
    const __nv_bfloat16* base = k + (int64_t)sl.start * p.sk_t + (int64_t)hk * p.sk_h + dim0 + dl * kVec;
    int r = rl;
    // kAhead rows in flight per thread, accumulated in increasing r
    for (; r + (kAhead - 1) * kMeanLanes < p.C; r += kAhead * kMeanLanes) {
      Load x[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        x[u] = __ldg(reinterpret_cast<const Load*>(base + (int64_t)(r + u * kMeanLanes) * p.sk_t));
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        float f[kVec];
        unpack_mean<kHalf>(x[u], f);
#pragma unroll
        for (int i = 0; i < kVec; ++i) acc[i] += f[i];
      }
    }
    if constexpr (kAhead > 16) {           // a quarter as many for what is left
      for (; r + (kAhead / 4 - 1) * kMeanLanes < p.C; r += kAhead / 4 * kMeanLanes) {
        Load x[kAhead / 4];
#pragma unroll
        for (int u = 0; u < kAhead / 4; ++u)
          x[u] = __ldg(reinterpret_cast<const Load*>(base + (int64_t)(r + u * kMeanLanes) * p.sk_t));
#pragma unroll
        for (int u = 0; u < kAhead / 4; ++u) {
          float f[kVec];
          unpack_mean<kHalf>(x[u], f);
#pragma unroll
          for (int i = 0; i < kVec; ++i) acc[i] += f[i];
        }
      }
    }
    for (; r < p.C; r += kMeanLanes) {
      const Load x = __ldg(reinterpret_cast<const Load*>(base + (int64_t)r * p.sk_t));
      float f[kVec];
      unpack_mean<kHalf>(x, f);
#pragma unroll
      for (int i = 0; i < kVec; ++i) acc[i] += f[i];
    }
  }
#pragma unroll
  for (int i = 0; i < kVec; ++i) part[rl][dl * kVec + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < kDims) {
    float tot = part[0][threadIdx.x];
#pragma unroll
    for (int a = 1; a < kMeanLanes; ++a) tot += part[a][threadIdx.x];
    const float mean = sl.historical ? __fdiv_rn(tot, (float)p.C) : 0.f;
    if (kHalf) reinterpret_cast<__half*>(dst)[threadIdx.x] = __float2half_rn(mean);
    else dst[threadIdx.x] = __float2bfloat16_rn(mean);
  }
}

// Means of the slots [slot_begin, slot_end) only (context-parallel ranks compute those of their own chunks).
cudaError_t launch_chunk_means_range(const Params& p, int slot_begin, int slot_end, const __nv_bfloat16* k,
                                     const int32_t* cu, __nv_bfloat16* means, cudaStream_t st, int32_t* zero,
                                     int64_t zero_words) {
  if (slot_end <= slot_begin)
    return zero_words > 0 ? cudaMemsetAsync(zero, 0, (size_t)zero_words * sizeof(int32_t), st) : cudaSuccess;
  // Split over the dims when the (slot, head) pairs alone give the SMs fewer than two CTAs each and the
  // chunk is long enough for several batches of rows.
  const int64_t pairs = (int64_t)(slot_end - slot_begin) * p.Hkv;
  const bool split = pairs < 2 * 148 && p.C >= 8 * kMeanLanes;
  const bool many = pairs * (kMeanLanes * (p.D / 8)) > 148 * 1280;         // (the same kernel at head dim 256)
  // The split one again where 16 dims a CTA fit two CTAs per SM.
  const bool few = pairs * (p.D / 16) <= 2 * 148 && p.C >= 16 * kMeanLanes;
#define MOBA_MEANS(HALF, DIM)                                                                                          \
  return few ? launch_pdl(chunk_mean_kernel<HALF, DIM, 16, 64, 1, 4>, dim3(slot_end - slot_begin, p.Hkv, DIM / 16),    \
                          kMeanLanes * 4, 0, st, p, slot_begin, k, cu, means, zero, zero_words)                        \
       : split ? launch_pdl(chunk_mean_kernel<HALF, DIM, 32, 16, 8>, dim3(slot_end - slot_begin, p.Hkv, DIM / 32),     \
                            kMeanLanes * 4, 0, st, p, slot_begin, k, cu, means, zero, zero_words)                      \
               : launch_pdl(many ? chunk_mean_kernel<HALF, DIM, kMeanDims<DIM>, 4, DIM < 256 ? 2048 / (kMeanLanes * (DIM / 8)) : 6>  \
                                 : chunk_mean_kernel<HALF, DIM, kMeanDims<DIM>, 4, DIM < 256 ? 1 : 6>,                  \
                            dim3(slot_end - slot_begin, p.Hkv, DIM / kMeanDims<DIM>), kMeanLanes * (kMeanDims<DIM> / 8), 0, st, p, \
                            slot_begin, k, cu, means, zero, zero_words)
  switch (p.D) {
    case 64:  if (p.fp16) MOBA_MEANS(true, 64);  else MOBA_MEANS(false, 64);
    case 96:  if (p.fp16) MOBA_MEANS(true, 96);  else MOBA_MEANS(false, 96);
    case 128: if (p.fp16) MOBA_MEANS(true, 128); else MOBA_MEANS(false, 128);
    case 256: if (p.fp16) MOBA_MEANS(true, 256); else MOBA_MEANS(false, 256);
    default: return cudaErrorInvalidValue;
  }
#undef MOBA_MEANS
}

cudaError_t launch_chunk_means(const Params& p, const __nv_bfloat16* k, const int32_t* cu,
                               __nv_bfloat16* means, cudaStream_t st) {
  return launch_chunk_means_range(p, 0, p.slots, k, cu, means, st);
}

// ---------------------------------------------------------------------------
// scores + mask + top-k
//
// Two steps per (token, head) row, with the same result as scoring every
// candidate in the contract order above:
//
//   1. estimate on the tensor core.  A row tile is 128 rows: the tokens of a
//      tile x the query heads of one kv head.  Persistent CTAs (128 threads)
//      walk the row tiles; TMA brings the Q rows of a tile and a tile of up to
//      256 candidate means into shared memory in the 128-byte swizzled K-major
//      layout, tcgen05.mma multiplies them (fp32 accumulators in tensor
//      memory, one lane per row), and thread r reads the estimates a_c of its
//      row 32 at a time and keeps the L = hist + 1 (+ 3 when a row can have
//      more than 32 candidates) largest, sorted, in shared memory.  For
//      L <= 32 the five lowest bits of the 32 estimates hold their position
//      (a change of less than 2^-18 of the score, counted in eps), a
//      compare-exchange network over the 32 registers brings the largest 8, 16
//      or 32 to the front, and they are merged with the list; longer
//      lists are kept as a min-heap of order-preserving integer keys.
//   2. recheck.  With e_c the score in the contract order, |a_c - e_c| <= eps
//      for every candidate of the row (bound below).  If neighbours in the
//      sorted list differ by more than 2 eps down to the entry after the
//      hist-th, the order of the a_c is the order of the e_c and the list is
//      the answer.  Otherwise the candidates with a_c >= a_(hist) - 2 eps (the
//      only ones that can be among the hist best e_c) are scored again by the
//      warp on CUDA cores in the contract order, one candidate per lane, and
//      ranked by the packed key of the reference
//      (order-preserving score bits << 32 | 0xFFFFFFFF - slot,
//      routing.py:778-784, :1151-1153: ties go to the lower slot).  A row
//      whose near-ties overflow the list, whose scores are not finite, or
//      whose tensor-core result did not arrive is ranked over all its
//      candidates the same way.
//
// Error bound.  Products of two 16-bit inputs are exact in fp32, so both
// results differ from the real dot product by summation error only.  Contract
// order: 7 + log2(D/8) roundings on a path, each <= 2^-24 of a partial sum
// that is <= S = sum_i |q_i m_i|.  Tensor core: per 16-dim step the 16
// products and the accumulator are aligned to the largest exponent and
// truncated; assuming no more than one unit of the 24-bit significand of that
// exponent is lost per term and one more when the sum is normalised, a step
// loses <= 18 * 2^-23 * S.  Together eps = ((18 * D/16 + 16) * 2^-23 + 2^-18) * S
// with S <= |q|_2 |m|_2 (Cauchy-Schwarz, the largest norm over the staged means),
// plus 2^-100 for products flushed to zero.  The recheck step measures
// |a_c - e_c| / eps on every candidate it scores again (optional statistics
// output), so the assumption is observable: on random inputs the largest
// ratio seen is below 0.01.
// ---------------------------------------------------------------------------
namespace {

using namespace ptx;

constexpr int kGateThreads = 128;         // one thread per row = one TMEM lane
constexpr int kGateRows = 128;            // (token, head) rows per tile
constexpr int kListExtra = 3;             // list places beyond hist + 1 that absorb near-ties at the cut
constexpr int kCntSmemMax = 4096;         // chunks per sequence up to which the list histogram is kept in shared memory
constexpr int kQBlockBytes = 128 * 128;   // one [128 rows][64 dims] swizzled block of 16-bit values
// floats per row of the score scratch, for the values a network leaves (w) or, without one (0), all 32 of a step: an odd
// number of 16-byte pieces, so that 16-byte stores are free of conflicts
__host__ __device__ constexpr int scratch_stride(int w) { return (w > 0 ? w : 32) + 4; }
// (rows of one step of 32 candidates have nothing to merge)
__host__ __device__ constexpr bool has_scratch(int mc, int w) { return w == 0 || mc - 1 > 32; }

__device__ __forceinline__ uint32_t float_key(float x) {      // routing.py:778-784
  const uint32_t b = __float_as_uint(x);
  return b ^ ((b & 0x80000000u) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {      // inverse of float_key
  return __uint_as_float(k ^ ((k & 0x80000000u) ? 0x80000000u : 0xFFFFFFFFu));
}
__device__ __forceinline__ float dot8(const float (&q)[8], const float (&m)[8]) {
  float s = __fmul_rn(q[0], m[0]);
#pragma unroll
  for (int i = 1; i < 8; ++i) s = __fmaf_rn(q[i], m[i], s);
  return s;
}

// shared-memory matrix descriptor of a K-major, 128-byte swizzled tile (8-row groups 1024 bytes apart)
__device__ __forceinline__ uint64_t gate_desc(uint32_t addr) {
  constexpr uint64_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return (hi << 32) | (uint64_t)(((addr & 0x3FFFFu) >> 4) | (1u << 16));
}

// byte offset of the 16-byte piece `ch` of row `r` inside a tile of [rows][64]-element blocks
__device__ __forceinline__ uint32_t swz_piece(int r, int ch, int block_bytes) {
  return (uint32_t)((ch >> 3) * block_bytes + r * 128 + (((ch & 7) ^ (r & 7)) << 4));
}

struct GateCtrl {
  uint64_t q_full[2];
  uint64_t b_full;
  uint64_t mma_done;
  uint32_t tmem_slot;
  int32_t mean_ssq_max;                    // largest squared norm over the means seen so far of this (sequence, kv head)
  unsigned long long exact[kGateThreads / 32][64];   // per warp: keys of the row being ranked exactly
};

// Squared norm of row `r` of a swizzled tile.
template <bool kHalf, int D>
__device__ __forceinline__ float row_ssq(const unsigned char* tile, int r, int block_bytes) {
  float ssq = 0.f;
#pragma unroll 4
  for (int ch = 0; ch < D / 8; ++ch) {
    float f[8];
    unpack8<kHalf>(*reinterpret_cast<const uint4*>(tile + swz_piece(r, ch, block_bytes)), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) ssq = __fmaf_rn(f[e], f[e], ssq);
  }
  return ssq;
}
// Squared norm of the D values at `row` (global memory).
template <bool kHalf, int D>
__device__ __forceinline__ float global_ssq(const __nv_bfloat16* row) {
  float ssq = 0.f;
#pragma unroll 4
  for (int ch = 0; ch < D / 8; ++ch) {
    float f[8];
    unpack8<kHalf>(__ldg(reinterpret_cast<const uint4*>(row + ch * 8)), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) ssq = __fmaf_rn(f[e], f[e], ssq);
  }
  return ssq;
}

// Score of the row at `qrow` against the mean at `mrow` (global memory), in the contract order: one
// candidate per lane.
// (not inlined: it is called from rarely taken recheck paths, and one copy keeps the
// kernel's hot loop small in the instruction cache)
template <bool kHalf, int D>
__device__ __noinline__ float contract_score(const __nv_bfloat16* qrow, const __nv_bfloat16* mrow) {
  constexpr int kNB = D / 8;
  constexpr int kNBPad = kNB <= 8 ? 8 : (kNB <= 16 ? 16 : 32);
  uint4 mraw[kNB];
#pragma unroll
  for (int l = 0; l < kNB; ++l) mraw[l] = __ldg(reinterpret_cast<const uint4*>(mrow + l * 8));
  float b[kNBPad];
#pragma unroll
  for (int l = 0; l < kNBPad; ++l) {
    if (l < kNB) {
      float qf[8], mf[8];
      unpack8<kHalf>(__ldg(reinterpret_cast<const uint4*>(qrow + l * 8)), qf);
      unpack8<kHalf>(mraw[l], mf);
      b[l] = dot8(qf, mf);
    } else {
      b[l] = 0.f;
    }
  }
#pragma unroll
  for (int h = kNBPad / 2; h >= 1; h >>= 1)
#pragma unroll
    for (int l = 0; l < h; ++l) b[l] = __fadd_rn(b[l], b[l + h]);
  return b[0];
}

// The same score, a block of 8 dims per lane: the groups of kNBPad lanes of a warp each score a candidate, and
// the first lane of a group has the result.  For the few candidates of a run of near-ties: one load of the mean
// and eight multiply-adds in a row in place of sixteen and 128 (6200 cycles a row).
template <int D> constexpr int kScoreLanes = D <= 64 ? 8 : D <= 128 ? 16 : 32;
template <bool kHalf, int D>
__device__ __forceinline__ float contract_score_group(const __nv_bfloat16* qrow, const __nv_bfloat16* mrow) {
  const int l = threadIdx.x & (kScoreLanes<D> - 1);
  float b = 0.f;
  if (l < D / 8) {
    float qf[8], mf[8];
    unpack8<kHalf>(__ldg(reinterpret_cast<const uint4*>(qrow + l * 8)), qf);
    unpack8<kHalf>(__ldg(reinterpret_cast<const uint4*>(mrow + l * 8)), mf);
    b = dot8(qf, mf);
  }
#pragma unroll
  for (int h = kScoreLanes<D> / 2; h >= 1; h >>= 1) b = __fadd_rn(b, __shfl_down_sync(0xffffffffu, b, h));
  return b;
}

// Min-heap of {chunk, key} on the key: `heap[0]` is the smallest key kept.  Replaces the
// root by (key, chunk) and restores the heap.
__device__ __forceinline__ void heap_replace_root(uint2* heap, int n, uint32_t key, uint32_t chunk) {
  int k = 0;
  for (;;) {
    const int l = 2 * k + 1;
    if (l >= n) break;
    uint2 child = heap[l];
    int s = l;
    if (l + 1 < n) {
      const uint2 right = heap[l + 1];
      if (right.y < child.y) { child = right; s = l + 1; }
    }
    if (!(child.y < key)) break;
    heap[k] = child;
    k = s;
  }
  heap[k] = make_uint2(chunk, key);
}

enum { GATE_FORCE_EXACT = 1, GATE_FORCE_RECHECK = 2 };
// marks in the chunk word of a list entry (chunk indices are below 2^24; an empty place is 0xFFFFFFFF)
constexpr uint32_t kTied = 1u << 30, kRunStart = 1u << 29, kChunkMask = 0x00FFFFFFu;

// Resident CTAs per SM the register budget is set for: four with the narrow network (its
// working set is small and the kernel is bound by the latency of dependent instructions, which
// more warps hide), three otherwise (a fourth would spill the 32 values of the wide network).
template <int kW> constexpr int kGateMinCtas = kW == 8 ? 4 : 3;

struct GateTile {
  int valid, b, hk, s0, tok_lo, ntok, max_cand;
};

__device__ __forceinline__ GateTile gate_tile(const Params& p, const int32_t* __restrict__ cu, int i, int tiles_x,
                                              int tokens_per_cta) {
  GateTile t;
  const int rest = i / tiles_x;
  t.hk = rest % p.Hkv;
  t.b = rest / p.Hkv;
  t.s0 = cu[t.b];
  const int s1 = cu[t.b + 1];
  const int x = i - rest * tiles_x + window_tile0(p, t.s0, tokens_per_cta);
  // tokens of the tile, clipped to the sequence and to the query window
  t.tok_lo = max(t.s0 + x * tokens_per_cta, p.win_lo);
  const int tok_hi = min(min(t.s0 + (x + 1) * tokens_per_cta, s1), p.win_lo + (int)p.Tq);
  t.valid = t.tok_lo < tok_hi;
  t.ntok = tok_hi - t.tok_lo;
  // candidates of the last token of the tile bound the chunks to stage
  t.max_cand = t.valid ? (tok_hi - 1 - t.s0) / p.C : 0;
  return t;
}

// eps of a row is this times |q|_2 max|m|_2 (see the head of this section); kPosition: the estimates hold their
// position in their low bits
template <int D, bool kPosition> constexpr float gate_kappa =
    ((18.f * (D / 16) + 16.f) / 8388608.f + (kPosition ? 1.f / 262144.f : 0.f)) * 1.001f;

// ---- rows that the estimates alone do not settle ------------------------------------------------------------
struct GateLists {
  uint2* lists;                            // [128][lstride] {chunk, estimate (kFloats) or its key}, the largest first
  int lstride, list_len;
  unsigned long long* exact;               // [64] keys, of this warp
};
// The warp ranks the rows of its lanes with mode != 0: 1 all n_surv entries of the list, 2 all ncand candidates, 3 the runs of
// near-ties marked in the list.  The calling lane's row is `row` of the tile, at `qrow` in global memory; eps: its error bound.
// kShort: the loops over the entries of a row are not unrolled.  Code that few rows come to is mostly fetched: 32768 x 32/8, at most 32
// candidates, lists of 8: gating kernel 218 -> 214 us, head dim 256 552 -> 522, a decode step with a near-tie 60 -> 58.
// Where many rows do, it costs (top-k 28 of 256 candidates at head dim 256, half of the rows: 1936 -> 2056).
// kFloats: the list holds the estimates themselves, not order-preserving integer keys.
template <bool kHalf, int D, bool kShort, bool kFloats>
__device__ __forceinline__ void rank_rows(const Params& p, const GateLists& g, const GateTile& t, const __nv_bfloat16* qrow,
                                          int row, int mode, int n_surv, int n_keep, int ncand, float eps,
                                          const __nv_bfloat16* __restrict__ means, int32_t* __restrict__ stats) {
  const int lane = threadIdx.x & 31;
  const int hist = p.hist, lstride = g.lstride;
  const int slot0 = t.b * p.mc;
  auto estimate = [](uint32_t y) { return kFloats ? __uint_as_float(y) : key_float(y); };
  uint2* lists = g.lists;
  unsigned need = __ballot_sync(0xffffffffu, mode != 0);
  unsigned long long* lx = g.exact;
  while (need) {
    const int src = __ffs(need) - 1;
    need &= need - 1;
    const int r = (row & ~31) + src;
    const int r_mode = __shfl_sync(0xffffffffu, mode, src);
    const int r_total = r_mode == 2 ? __shfl_sync(0xffffffffu, ncand, src) : __shfl_sync(0xffffffffu, n_surv, src);
    const int r_keep = __shfl_sync(0xffffffffu, n_keep, src);
    const float r_eps = __shfl_sync(0xffffffffu, eps, src);
    const __nv_bfloat16* r_q =
        reinterpret_cast<const __nv_bfloat16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(qrow), src));
    uint2* rlist = lists + (size_t)r * lstride;
    if (r_mode == 3) {
      // runs of near-ties: one marked entry per lane (at most 32), exact keys, rank inside the run
      int cnt = 0, runs = 0, my_e = -1, my_run = 0;
      for (int e0 = 0; e0 < r_total; e0 += 32) {
        const int e = e0 + lane;
        const uint32_t x = e < r_total ? rlist[e].x : 0u;
        const unsigned bt = __ballot_sync(0xffffffffu, (x & kTied) != 0 && x != 0xFFFFFFFFu);
        const unsigned bs = __ballot_sync(0xffffffffu, (x & kRunStart) != 0 && x != 0xFFFFFFFFu);
        if ((bt >> lane) & 1) {
          const int slot = cnt + __popc(bt & ((1u << lane) - 1));
          const int run = runs + __popc(bs & ((2u << lane) - 1));
          lx[slot] = (unsigned long long)e | ((unsigned long long)run << 8);
        }
        cnt += __popc(bt);
        runs += __popc(bs);
      }
      __syncwarp();
      unsigned long long key = 0ull;
      uint2 ent = make_uint2(0u, 0u);
      uint32_t cc = 0;
      if (lane < cnt) {
        my_e = (int)(lx[lane] & 0xFF);
        my_run = (int)(lx[lane] >> 8);
        ent = rlist[my_e];
        cc = ent.x & kChunkMask;
      }
      // as many entries at a time as the warp has groups of lanes; entry i's score goes to lane i
      float e = 0.f;
      constexpr int kPer = 32 / kScoreLanes<D>;
      auto score = [&](int i0) {
        const int mine = i0 + lane / kScoreLanes<D>;
        const uint32_t ec = __shfl_sync(0xffffffffu, cc, mine & 31);     // (past the last entry: a chunk scored in vain)
        const float score = contract_score_group<kHalf, D>(r_q, means + ((int64_t)(slot0 + (int)ec) * p.Hkv + t.hk) * D);
        const float got = __shfl_sync(0xffffffffu, score, ((lane - i0) * kScoreLanes<D>) & 31);
        if (lane >= i0 && lane < i0 + kPer) e = got;
      };
      if constexpr (kShort) {
#pragma unroll 1
        for (int i0 = 0; i0 < cnt; i0 += kPer) score(i0);
      } else {
        for (int i0 = 0; i0 < cnt; i0 += kPer) score(i0);
      }
      if (lane < cnt) {
        key = ((unsigned long long)float_key(e) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(slot0 + (int)cc));
        if (stats != nullptr) {
          const float diff = fabsf(estimate(ent.y) - e);
          if (!(diff <= r_eps)) atomicAdd(&stats[2], 1);
          atomicMax(&stats[1], (int)fminf(diff / r_eps * 65536.f, 1.0e9f));
        }
      }
      int rank = 0, first = my_e;
      auto compare = [&](int t2) {
        const unsigned long long kt = __shfl_sync(0xffffffffu, key, t2);
        const int rt = __shfl_sync(0xffffffffu, my_run, t2), et = __shfl_sync(0xffffffffu, my_e, t2);
        if (lane < cnt && rt == my_run) {
          rank += kt > key;
          first = min(first, et);
        }
      };
      if constexpr (kShort) {
#pragma unroll 1
        for (int t2 = 0; t2 < cnt; ++t2) compare(t2);
      } else {
        for (int t2 = 0; t2 < cnt; ++t2) compare(t2);
      }
      __syncwarp();
      if (lane < cnt) rlist[first + rank].x = cc;          // a run occupies consecutive places; marks are cleared
      __syncwarp();
      if (stats != nullptr && lane == 0) atomicAdd(&stats[0], 1);
      continue;
    }
    lx[lane] = 0ull;
    lx[lane + 32] = 0ull;
    __syncwarp();
    int viol = 0, ratio = 0;
    for (int base = 0; base < r_total; base += 32) {
      const int idx = base + lane;
      unsigned long long key = 0ull;
      if (idx < r_total) {
        const int cc = r_mode == 2 ? idx : (int)rlist[idx].x;
        const float e = contract_score<kHalf, D>(r_q, means + ((int64_t)(slot0 + cc) * p.Hkv + t.hk) * D);
        key = ((unsigned long long)float_key(e) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)(slot0 + cc));
        if (r_mode == 1 && stats != nullptr) {
          const float diff = fabsf(estimate(rlist[idx].y) - e);
          if (!(diff <= r_eps)) viol = 1;
          ratio = (int)fminf(diff / r_eps * 65536.f, 1.0e9f);
        }
      }
      // the keys of this batch, in lane order, into the ordered list lx[0, r_keep)
      unsigned hits = __ballot_sync(0xffffffffu, key > lx[r_keep - 1]);
      while (hits) {
        const int l = __ffs(hits) - 1;
        hits &= hits - 1;
        const unsigned long long kk = __shfl_sync(0xffffffffu, key, l);
        const unsigned long long k0 = lane < r_keep ? lx[lane] : 0ull;
        const unsigned long long k1 = lane + 32 < r_keep ? lx[lane + 32] : 0ull;
        const int pos = __popc(__ballot_sync(0xffffffffu, k0 > kk)) + __popc(__ballot_sync(0xffffffffu, k1 > kk));
        if (pos < r_keep) {                                  // uniform; false when the list filled up meanwhile
          if (lane >= pos && lane + 1 < r_keep) lx[lane + 1] = k0;
          if (lane + 32 >= pos && lane + 33 < r_keep) lx[lane + 33] = k1;
          if (lane == 0) lx[pos] = kk;
        }
        __syncwarp();
      }
    }
    // the exact ranking replaces the chunk ids of the row's list
    for (int i = lane; i < hist; i += 32) {
      const unsigned long long key = i < r_keep ? lx[i] : 0ull;
      rlist[i].x = key ? (0xFFFFFFFFu - (uint32_t)(key & 0xFFFFFFFFull)) - (uint32_t)slot0 : 0xFFFFFFFFu;
    }
    __syncwarp();
    if (stats != nullptr) {
      viol = __any_sync(0xffffffffu, viol);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ratio = max(ratio, __shfl_xor_sync(0xffffffffu, ratio, o));
      if (lane == 0) {
        atomicAdd(&stats[r_mode == 2 ? 3 : 0], 1);
        if (r_mode == 1) atomicMax(&stats[1], ratio);
        if (viol) atomicAdd(&stats[2], 1);
      }
    }
  }
}

// The CTA that finishes last turns the counts of all into the offsets of the lists.  Executed by the whole CTA.
template <int kThreads>
__device__ __forceinline__ void finish_scan(const ListScan& scan, int32_t* __restrict__ ticket, int* scratch) {
  __threadfence();
  __syncthreads();                                            // (`scratch` is free from here on)
  if (threadIdx.x == 0) scratch[0] = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  const bool last = scratch[0] != 0;
  __syncthreads();
  if (last) {
    __threadfence();
    scan_lists<kThreads, 8>(scan, scratch);
  }
}

// ---------------------------------------------------------------------------
// rows with at most 32 candidates
//
// One tile of means, one network a row, so what counts is the latency of a tile of rows: 25 000 cycles of it were
// spent waiting for Q, on norms, on walks through lists in shared memory and at a barrier behind the warp with
// the most near-ties, 2400 in the network.  Here
//   warp 4     walks the row tiles of the CTA: requests Q and means and issues the MMA as soon as every row has its
//              norms and its estimates of the tile before in registers, while networks, decisions and stores go on
//   warps 0-3  a thread per row.  The sorted estimates stay in registers, and what they settle is decided there; a row with
//              near-ties goes through a list in shared memory.  Every warp counts for itself and warp 4 adds the
//              counts of a tile to the lists a tile later: no barrier of the CTA in the loop, a warp may be a tile
//              behind another.  (Added by every warp for itself, four requests for one, and some 7 ns each for the 128-byte
//              line of counters that all CTAs are at: 32768 x 32/8, 31 candidates, top-k 4 203-265 us, 161 this way;
//              head dim 64, top-k 8 195-251, 149.)
// Measured against the kernel below for these shapes, with the wait for the chunk means: 2 x 4096 tokens x 16 heads, 31
// candidates 44 -> 40 us, at head dim 256 105 -> 91; 32768 x 32/8, 7 candidates 179 -> 152; a decode token on 32 chunks 24 -> 17.
// (The few-lane score of near-ties alone, which the kernel below has too: 32768 x 32/8, 255 candidates 620 -> 573.)
// Networks over the estimates instead of integer keys, as there (kernel alone, us): 2 x 4096 x 16 heads 43.0 -> 40.9, at head dim 256
// 90.2 -> 86.9; 32768 x 32/8, 7 candidates 122.8 -> 108.5; 131072 x 32/8, 31 780 -> 685; 32768 x 16/4, 31 118.8 -> 104.5, head dim 64 86 -> 78.
// ---------------------------------------------------------------------------
constexpr int kOneThreads = 160;
constexpr int kOneMeans = 32;              // rows of the tile of means, columns of tensor memory

struct OneCtrl {
  uint64_t full;                           // per row tile: Q and means landed
  uint64_t read;                           // ... and have been read by everybody
  uint64_t mma_done;
  uint32_t tmem_slot;
  GateTile tile[2];
  int32_t mean_ssq[2][kGateRows / 32];     // largest squared norm of a mean, by the warps
  int32_t cnt[4][kGateRows / 32][kOneMeans];   // rows of a warp that selected a chunk; row tile n: place n & 3
  int64_t cnt_list[4];                     // at the end: the list of the first chunk of cnt[place], < 0: nothing to add
  unsigned long long exact[kGateRows / 32][64];
};

template <bool kHalf, int D, int kW>
__global__ void __launch_bounds__(kOneThreads, kGateMinCtas<kW>)
gate_one_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_m,
                int tokens_per_cta, int nt, int list_len, int, int, const __nv_bfloat16* __restrict__ q,
                const __nv_bfloat16* __restrict__ means, const int32_t* __restrict__ cu, int32_t* __restrict__ selected,
                int32_t* __restrict__ list_counts, int32_t* __restrict__ stats, int flags, const ListScan scan,
                int32_t* __restrict__ ticket) {
  extern __shared__ unsigned char gate_smem_raw[];
  constexpr int kNBlk = (D + 63) / 64;
  const int hist = p.hist;
  const int lstride = list_len | 1;
  unsigned char* sQ = reinterpret_cast<unsigned char*>(((uintptr_t)gate_smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sB = sQ + (size_t)kNBlk * kQBlockBytes;                 // kNBlk blocks [32][64]
  uint2* lists = reinterpret_cast<uint2*>(sB + (size_t)kNBlk * kOneMeans * 128);
  OneCtrl& c = *reinterpret_cast<OneCtrl*>(lists + (size_t)kGateRows * lstride);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_x = window_tiles(p, tokens_per_cta);
  const int n_tiles = tiles_x * p.Hkv * p.B;
  const int rows_box = tokens_per_cta * p.G;

  if (tid == 0) {
    mbar_init(smem_u32(&c.full), 1);
    mbar_init(smem_u32(&c.read), kGateRows);
    mbar_init(smem_u32(&c.mma_done), 1);
    fence_barrier_init();
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_m);
  }
  for (int i = tid; i < 4 * kGateRows; i += kOneThreads) reinterpret_cast<int32_t*>(c.cnt)[i] = 0;
  if (warp == 0) {
    tmem_alloc(smem_u32(&c.tmem_slot), (uint32_t)kOneMeans);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;

  // (With the wider networks, whose calls have a row tile a CTA at most (gate_one), every warp adds its own counts.)
  constexpr bool kDefer = kW == 8;
  // counts of a tile into those of the lists (warp 4); `list` of its first chunk, < 0: nothing to add
  auto add_counts = [&](int place, int64_t list) {
    if (list < 0 || list_counts == nullptr) return;
    int k = 0;
#pragma unroll
    for (int w = 0; w < kGateRows / 32; ++w) {
      k += c.cnt[place][w][lane];
      c.cnt[place][w][lane] = 0;
    }
    if (k > 0) atomicAdd(&list_counts[list + (int64_t)lane * p.Hkv], k);
  };
  if (warp == 4) {
    // row tile n of the CTA is tile blockIdx.x + n * gridDim.x of the grid, valid or not
    uint32_t n = 0;
    int64_t list1 = -1, list2 = -1;                    // of tiles n - 1, n - 2: their counts are not added yet
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x, ++n) {
      const GateTile t = gate_tile(p, cu, ti, tiles_x, tokens_per_cta);
      const bool work = t.valid && t.max_cand > 0;
      // Q, means and tensor memory are free once everybody has read the tile before (c.tile and c.mean_ssq have two
      // places: a thread that has read it is through with the tile before that)
      bool ok = n == 0 || mbar_wait(smem_u32(&c.read), (n - 1) & 1);
      if (!__all_sync(0xffffffffu, ok)) break;         // the rows' threads run into their own bounded waits
      if (lane == 0) {
        c.tile[n & 1] = t;
        const uint32_t bar = smem_u32(&c.full);
        if (work) {
          mbar_expect_tx(bar, (uint32_t)(kNBlk * (rows_box + kOneMeans) * 128));
#pragma unroll
          for (int blk = 0; blk < kNBlk; ++blk) {
            tma_load_3d(smem_u32(sQ + (size_t)blk * kQBlockBytes), &tmap_q, bar, blk * 64, t.hk * p.G, t.tok_lo - p.win_lo);
            tma_load_3d(smem_u32(sB + (size_t)blk * kOneMeans * 128), &tmap_m, bar, blk * 64, t.hk, t.b * p.mc);
          }
        } else {
          mbar_arrive(bar);
        }
      }
      // Who has read tile n - 1 has counted tile n - 2.  Its place is that of tile n + 2, which is requested behind this.
      if (kDefer) add_counts((n + 2) & 3, list2);
      list2 = list1;
      list1 = work ? (int64_t)t.b * p.mc * p.Hkv + t.hk : -1;
      __syncwarp();
      ok = mbar_wait(smem_u32(&c.full), n & 1);
      if (work && __all_sync(0xffffffffu, ok)) {
        if (lane == 0) {
          tc_fence_after();
          const uint32_t idesc = idesc_16_f32(kHalf, 128, kOneMeans, 0, 0);
          const uint32_t aQ = smem_u32(sQ), aB = smem_u32(sB);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            mma_ss(tmem, gate_desc(aQ + (ks >> 2) * kQBlockBytes + (ks & 3) * 32),
                   gate_desc(aB + (ks >> 2) * kOneMeans * 128 + (ks & 3) * 32), idesc, ks > 0);
          tc_commit(smem_u32(&c.mma_done));
        }
        __syncwarp();
      }
      if (!__all_sync(0xffffffffu, ok)) { ++n; break; }
    }
    if (kDefer && lane < 4)                            // (tile n - 1 is the last one requested)
      c.cnt_list[(n + lane) & 3] = lane == 3 ? list1 : lane == 2 ? list2 : -1;
  } else {
    const int row = tid;
    uint2* mylist = lists + (size_t)row * lstride;
    uint32_t n = 0, m = 0;                             // row tiles, tiles with candidates
    bool lost = false;                                 // a wait gave up: no copies or estimates any more, from this tile on
    for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x, ++n) {
      bool failed = lost || !mbar_wait(smem_u32(&c.full), n & 1);
      failed = lost = __any_sync(0xffffffffu, failed);
      const GateTile t = failed ? gate_tile(p, cu, ti, tiles_x, tokens_per_cta) : c.tile[n & 1];
      const int nrows = t.valid ? t.ntok * p.G : 0;
      const int slot0 = t.b * p.mc;
      const int tl = row / p.G, hl = row - tl * p.G;   // token and head of the row in the tile
      int32_t* dst = selected + (int64_t)(t.hk * p.G + hl) * p.Tq + (t.tok_lo - p.win_lo) + tl;
      if (!t.valid || t.max_cand <= 0) {               // nothing, or the first chunk of a sequence: nothing to select
        if (!failed) mbar_arrive(smem_u32(&c.read));
        if (row < nrows)
          for (int r = 0; r < hist; ++r) dst[(int64_t)r * p.sel_rs] = -1;
        continue;
      }
      const int ncand = row < nrows ? (t.tok_lo + tl - t.s0) / p.C : 0;     // chunks before the row's own chunk
      // squared norms: of the row, and of the means (four lanes a mean, eight means a warp)
      float q_ssq = 0.f;
      if (!failed) {
        q_ssq = row_ssq<kHalf, D>(sQ, row, kQBlockBytes);
        const int mrow = tid >> 2;
        float s = 0.f;
#pragma unroll
        for (int ch = 0; ch < D / 32; ++ch) {
          float f[8];
          unpack8<kHalf>(*reinterpret_cast<const uint4*>(sB + swz_piece(mrow, 4 * ch + (lane & 3), kOneMeans * 128)), f);
#pragma unroll
          for (int e = 0; e < 8; ++e) s = __fmaf_rn(f[e], f[e], s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        // floats >= 0 order like their bit patterns; +inf and NaN have the largest patterns
        int ssq = mrow < t.max_cand ? __float_as_int(s) & 0x7FFFFFFF : 0;
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) ssq = max(ssq, __shfl_xor_sync(0xffffffffu, ssq, o));
        if (lane == 0) c.mean_ssq[m & 1][warp] = ssq;
        if (!mbar_wait(smem_u32(&c.mma_done), m & 1)) failed = true;
      } else if (lane == 0) {
        c.mean_ssq[m & 1][warp] = 0x7F800000;          // no bound: the other warps' rows are ranked exactly too
      }
      tc_fence_after();
      uint32_t v[32];
      float f[32];
      __syncwarp();
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16), v);
      tmem_wait_ld();
      tc_fence_before();
      // Q, means and the estimates have been read.  (A thread whose wait gave up arrives no more, so that a phase is
      // never complete without somebody: the others' waits give up in turn, and all rank the rows of this CTA exactly.)
      if (!failed) mbar_arrive(smem_u32(&c.read));
#pragma unroll
      for (int i = 0; i < 32; ++i)                     // the estimates, position in the low bits, as in the kernel below
        f[i] = i < ncand ? __uint_as_float((v[i] & ~31u) | (uint32_t)(31 - i)) : -INFINITY;
      topk::top_of_32<kW>(f);
      // the norms of the other warps: complete once all threads have arrived on `read`
      if (!failed && !mbar_wait(smem_u32(&c.read), n & 1)) failed = true;
      int ssq_max = 0;
#pragma unroll
      for (int w = 0; w < kGateRows / 32; ++w) ssq_max = max(ssq_max, c.mean_ssq[m & 1][w]);
      ++m;

      // What the estimates settle.  Bit i: entry i is a candidate (real), can be among the n_keep best (surv), is closer to
      // entry i + 1 than twice the error (tie)
      const float eps2 = 2.f * (gate_kappa<D, true> * sqrtf(q_ssq) * sqrtf(__int_as_float(ssq_max)) + 7.9e-31f);
      const int n_keep = min(hist, ncand), n_real = min(ncand, list_len);
      const bool all = (flags & GATE_FORCE_RECHECK) != 0;
      int mode = 0, n_surv = 0;                        // as in recheck_mode
      uint32_t tied = 0, first = 0;
      if (ncand > 0) {
        uint32_t close = 0;
        bool holes = false;
        float theta = 0.f;
#pragma unroll
        for (int i = 0; i < kW; ++i) {
          if (i < n_real) holes |= !(f[i] > -INFINITY);
          if (i + 1 == n_keep) theta = f[i] - eps2;
          if (i + 1 < kW && i + 1 < n_real && (all || !(f[i] - f[i + 1 < kW ? i + 1 : i] > eps2)))
            close |= 1u << i;
        }
#pragma unroll
        for (int i = 0; i < kW; ++i) n_surv += i < n_real && f[i] >= theta;
        const bool amb = all || (close & ((1u << n_keep) - 1u)) != 0;       // n_keep < 32
        if ((flags & GATE_FORCE_EXACT) || failed || holes) {
          mode = 2;
        } else if (amb) {
          if ((n_surv == list_len && ncand > list_len) || !(eps2 < INFINITY) || n_surv < n_keep) {
            mode = 2;                                  // the near-ties may go on below the list, or eps is not finite
          } else {
            const uint32_t runs = n_surv > 0 ? close & ((1u << (n_surv - 1)) - 1u) : 0u;
            tied = runs | (runs << 1);
            first = runs & ~(runs << 1);
            if (all && tied == 0) tied = first = 1u;   // a single survivor, scored again on request
            mode = tied != 0 ? 3 : 0;                  // (at most 32 entries)
          }
        }
      }
      const __nv_bfloat16* qrow = q + (int64_t)(t.tok_lo + tl - p.win_lo) * p.sq_t + (int64_t)(t.hk * p.G + hl) * p.sq_h;
      if (__any_sync(0xffffffffu, mode != 0)) {
#pragma unroll
        for (int i = 0; i < kW; ++i)
          if (i < list_len)
            mylist[i] = make_uint2(f[i] > -INFINITY ? (31u - (__float_as_uint(f[i]) & 31u)) | ((tied >> i) & 1u ? kTied : 0u) |
                                                          ((first >> i) & 1u ? kRunStart : 0u)
                                                    : 0xFFFFFFFFu, __float_as_uint(f[i]));
        __syncwarp();
        rank_rows<kHalf, D, true, true>(p, GateLists{lists, lstride, list_len, c.exact[warp]}, t, qrow, row, mode, n_surv, n_keep, ncand,
                                  0.5f * eps2, means, stats);
        __syncwarp();
      }
      const bool count = list_counts != nullptr && !(kDefer && lost);
      if (row < nrows) {
#pragma unroll
        for (int r = 0; r < kW; ++r)
          if (r < hist) {
            const uint32_t x = mode != 0 ? mylist[r].x : f[r] > -INFINITY ? 31u - (__float_as_uint(f[r]) & 31u) : 0xFFFFFFFFu;
            const int cc = x == 0xFFFFFFFFu ? -1 : (int)(x & kChunkMask);
            dst[(int64_t)r * p.sel_rs] = cc >= 0 ? slot0 + cc : -1;
            if (cc >= 0 && count) atomicAdd(&c.cnt[n & 3][warp][cc], 1);
          }
        // Nobody is told when the counts of a tile that was not seen to land are complete.  (Those of the last two
        // requested tiles are added at the end, and without this warp's arrivals no more than one is requested.)
        if (kDefer && lost && list_counts != nullptr && ncand > 0)
          for (int r = 0; r < n_keep; ++r)
            atomicAdd(&list_counts[(int64_t)(slot0 + (int)(mylist[r].x & kChunkMask)) * p.Hkv + t.hk], 1);
      }
      lost = __any_sync(0xffffffffu, failed);
      __syncwarp();
      if (!kDefer && list_counts != nullptr) {
        const int k = c.cnt[n & 3][warp][lane];
        if (k > 0) atomicAdd(&list_counts[(int64_t)(slot0 + lane) * p.Hkv + t.hk], k);
        c.cnt[n & 3][warp][lane] = 0;
        __syncwarp();
      }
    }
  }

  __syncwarp();
  if (kDefer) __syncthreads();                         // everybody has counted
  if (kDefer && warp == 4)
    for (int i = 0; i < 4; ++i) add_counts(i, c.cnt_list[i]);
  if (ticket != nullptr) finish_scan<kOneThreads>(scan, ticket, reinterpret_cast<int*>(c.exact));
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, (uint32_t)kOneMeans);
}

// rows with more than 32 candidates, lists longer than 32, and what else gate_one() leaves
// kW: width of the compare-exchange network (8, 16 or 32 >= list_len), 0: lists longer than 32 (min-heap)
template <bool kHalf, int D, int kW>
__global__ void __launch_bounds__(kGateThreads, kGateMinCtas<kW>)
gate_topk_kernel(const Params p, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_m,
                 int tokens_per_cta, int nt, int list_len, int nbuf, int cnt_in_smem,
                 const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ means,
                 const int32_t* __restrict__ cu, int32_t* __restrict__ selected,
                 int32_t* __restrict__ list_counts, int32_t* __restrict__ stats, int flags, const ListScan scan,
                 int32_t* __restrict__ ticket) {
  extern __shared__ unsigned char gate_smem_raw[];
  constexpr int kNBlk = (D + 63) / 64;                 // 64-dim blocks of a row
  const int hist = p.hist;
  const int lstride = list_len | 1;                    // odd: the rows' lists start in different banks

  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)gate_smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sQ0 = smem;                                             // nbuf x kNBlk blocks [128][64]
  unsigned char* sB = sQ0 + (size_t)nbuf * kNBlk * kQBlockBytes;        // kNBlk blocks [nt][64]
  uint2* lists = reinterpret_cast<uint2*>(sB + (size_t)kNBlk * nt * 128);   // [128][lstride] {chunk, score bits}
  float* scratch = reinterpret_cast<float*>(lists + (size_t)kGateRows * lstride);   // [128][scratch_stride], absent when unused
  GateCtrl& c = *reinterpret_cast<GateCtrl*>(scratch + (has_scratch(p.mc, kW) ? kGateRows * scratch_stride(kW) : 0));
  int32_t* cnt_s = reinterpret_cast<int32_t*>(&c + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_x = window_tiles(p, tokens_per_cta);
  const int n_tiles = tiles_x * p.Hkv * p.B;
  const int rows_box = tokens_per_cta * p.G;           // rows one Q box brings

  if (tid == 0) {
    mbar_init(smem_u32(&c.q_full[0]), 1);
    mbar_init(smem_u32(&c.q_full[1]), 1);
    mbar_init(smem_u32(&c.b_full), 1);
    mbar_init(smem_u32(&c.mma_done), 1);
    c.mean_ssq_max = 0;
    fence_barrier_init();
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_m);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&c.tmem_slot), (uint32_t)nt);
    tmem_relinquish();
  }
  if (cnt_in_smem)
    for (int i = tid; i < p.mc; i += kGateThreads) cnt_s[i] = 0;       // every tile leaves them at zero again
  pdl_wait();
  pdl_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = c.tmem_slot;
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);          // this thread's lane, column 0

  // producer state (thread 0): Q tiles requested so far, tile index to look for the next one from
  int q_requested = 0, q_next_from = blockIdx.x;
  uint32_t b_phase = 0, mma_phase = 0;
  int n = 0;                                           // tiles with candidates processed so far
  // mean norms: the (sequence, kv head) the running maximum belongs to and the candidates it covers
  int norm_b = -1, norm_hk = -1, norm_covered = 0;

  auto request_q = [&](const GateTile& t, int buf) {
    const uint32_t bar = smem_u32(&c.q_full[buf]);
    mbar_expect_tx(bar, (uint32_t)(kNBlk * rows_box * 128));
#pragma unroll
    for (int blk = 0; blk < kNBlk; ++blk)
      tma_load_3d(smem_u32(sQ0 + ((size_t)buf * kNBlk + blk) * kQBlockBytes), &tmap_q, bar, blk * 64, t.hk * p.G,
                  t.tok_lo - p.win_lo);
  };
  auto request_b = [&](const GateTile& t, int c0) {
    const uint32_t bar = smem_u32(&c.b_full);
    mbar_expect_tx(bar, (uint32_t)(kNBlk * nt * 128));
#pragma unroll
    for (int blk = 0; blk < kNBlk; ++blk)
      tma_load_3d(smem_u32(sB + (size_t)blk * nt * 128), &tmap_m, bar, blk * 64, t.hk, t.b * p.mc + c0);
  };

  for (int ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
    const GateTile t = gate_tile(p, cu, ti, tiles_x, tokens_per_cta);
    if (!t.valid) continue;
    const int nrows = t.ntok * p.G;
    const int slot0 = t.b * p.mc;
    // selected[r][head][tok]: `ntok` consecutive ints per (rank, head)
    auto store_selected = [&](int i, int slot) {
      const int r = i / nrows, rem = i - r * nrows;
      const int hl = rem / t.ntok, tl = rem - hl * t.ntok;
      selected[(int64_t)r * p.sel_rs + (int64_t)(t.hk * p.G + hl) * p.Tq + (t.tok_lo - p.win_lo) + tl] = slot;
    };
    if (t.max_cand <= 0) {                             // first chunk of a sequence: nothing to select
      for (int i = tid; i < hist * nrows; i += kGateThreads) store_selected(i, -1);
      continue;
    }
    const int buf = nbuf == 2 ? (n & 1) : 0;
    const uint32_t q_phase = nbuf == 2 ? ((n >> 1) & 1) : (n & 1);
    unsigned char* sQ = sQ0 + (size_t)buf * kNBlk * kQBlockBytes;
    if (tid == 0) {
      if (q_requested == n) {                          // not prefetched (first tile, or a single buffer)
        request_q(t, buf);
        q_requested = n + 1;
        q_next_from = ti + gridDim.x;
      }
      request_b(t, 0);
      if (nbuf == 2 && q_requested == n + 1) {         // the next tile with candidates, into the other buffer
        for (; q_next_from < n_tiles; q_next_from += gridDim.x) {
          const GateTile nx = gate_tile(p, cu, q_next_from, tiles_x, tokens_per_cta);
          if (nx.valid && nx.max_cand > 0) {
            request_q(nx, buf ^ 1);
            q_requested = n + 2;
            q_next_from += gridDim.x;
            break;
          }
        }
      }
    }

    // Largest squared norm over the means this tile's rows can meet: kept per (sequence, kv head)
    // and extended when a tile reaches further than the ones before it (a CTA walks the tiles
    // of a sequence in order, so every mean is read once per CTA).
    if (t.b != norm_b || t.hk != norm_hk || t.max_cand > norm_covered) {
      const bool fresh = t.b != norm_b || t.hk != norm_hk;
      if (fresh) {                                   // every thread is past its last read of the old maximum
        if (tid == 0) c.mean_ssq_max = 0;
        __syncthreads();
      }
      int ssq_max = 0;
      for (int cc = (fresh ? 0 : norm_covered) + tid; cc < t.max_cand; cc += kGateThreads)
        // floats >= 0 order like their bit patterns; +inf and NaN have the largest patterns
        ssq_max = max(ssq_max, __float_as_int(global_ssq<kHalf, D>(means + ((int64_t)(slot0 + cc) * p.Hkv + t.hk) * D)) &
                                   0x7FFFFFFF);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ssq_max = max(ssq_max, __shfl_xor_sync(0xffffffffu, ssq_max, o));
      if (lane == 0 && ssq_max > 0) atomicMax(&c.mean_ssq_max, ssq_max);
      __syncthreads();
      norm_b = t.b;
      norm_hk = t.hk;
      norm_covered = t.max_cand;
    }

    // this thread's row
    const int row = tid;
    const int ncand = row < nrows ? (t.tok_lo + row / p.G - t.s0) / p.C : 0;     // chunks before the row's own chunk
    uint2* mylist = lists + (size_t)row * lstride;
    for (int i = 0; i < list_len; ++i) mylist[i] = make_uint2(0xFFFFFFFFu, kW > 0 ? 0xff800000u : 0u);   // chunk -1, -inf or key 0: empty place
    uint32_t tau = 0;                                  // smallest key kept, the heap's root; 0 while places are free
    float last = -INFINITY;                            // the same of a sorted list, its last place
    uint32_t* myscratch = reinterpret_cast<uint32_t*>(scratch + row * scratch_stride(kW));

    // A wait that gives up is remembered by the thread: its row is then ranked exactly, from Q rows
    // read with plain loads (see the recheck).
    bool failed = !mbar_wait(smem_u32(&c.q_full[buf]), q_phase);
    const float q_ssq = failed ? 0.f : row_ssq<kHalf, D>(sQ, row, kQBlockBytes);

    for (int c0 = 0; c0 < t.max_cand; c0 += nt) {
      const int ct = min(nt, t.max_cand - c0);
      if (!mbar_wait(smem_u32(&c.b_full), b_phase)) failed = true;
      b_phase ^= 1;
      if (tid == 0) {
        tc_fence_after();
        const uint32_t idesc = idesc_16_f32(kHalf, 128, nt, 0, 0);
        const uint32_t aQ = smem_u32(sQ), aB = smem_u32(sB);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          mma_ss(tmem, gate_desc(aQ + (ks >> 2) * kQBlockBytes + (ks & 3) * 32),
                 gate_desc(aB + (ks >> 2) * nt * 128 + (ks & 3) * 32), idesc, ks > 0);
        tc_commit(smem_u32(&c.mma_done));
      }
      if (!mbar_wait(smem_u32(&c.mma_done), mma_phase)) failed = true;
      mma_phase ^= 1;
      tc_fence_after();
      // ---- estimates of this row: keep the largest in the heap -------------------------------
      const int cend = min(ct, ncand - c0);                   // this row's candidates in the tile
      int wend = cend;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) wend = max(wend, __shfl_xor_sync(0xffffffffu, wend, o));
      for (int col = 0; col < wend; col += 32) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(trow + col, v);
        tmem_wait_ld();
        const int rem = cend - col;
        const uint32_t chunk0 = (uint32_t)(c0 + col);
        if constexpr (kW > 0) {
          // Estimates as they are, with their place in the five low bits; places past the row's candidates get -inf.  (Estimates
          // this close are near-ties, ranked again whatever their order here, and a row with one that is not finite is ranked over
          // all its candidates.)  Integer keys in the same order took four more instructions an estimate of a kernel that is bound by
          // integer and min/max instructions: 32768 x 32/8, 255 candidates, top-k 8 545 -> 508 us, 4 424 -> 388, 24 1313 -> 1267;
          // 65536 x 16/4, 127 candidates 356 -> 327; head dim 64, up to 63 57.7 -> 54.1; 256 508 -> 489.
          float f[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = __uint_as_float((v[i] & ~31u) | (uint32_t)(31 - i));
          if (!__all_sync(0xffffffffu, rem >= 32)) {
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = i < rem ? f[i] : -INFINITY;
          }
          float fmx = -INFINITY;
#pragma unroll
          for (int i = 0; i < 32; i += 2) fmx = max3(fmx, f[i], f[i + 1]);
          if (!__any_sync(0xffffffffu, fmx > last)) continue;           // nothing here enters any list of the warp
          topk::top_of_32<kW>(f);
          auto entry = [&](uint32_t bits) { return make_uint2(chunk0 + 31u - (bits & 31u), bits); };
          if (c0 == 0 && col == 0) {
            // first candidates of the row: the list is the head of the sorted ones
#pragma unroll
            for (int i = 0; i < kW; ++i)
              if (i < list_len && f[i] > -INFINITY) mylist[i] = entry(__float_as_uint(f[i]));
          } else {
            // s_t enters the list iff it beats the entry t places from the end (both are sorted)
            int j = 0;
#pragma unroll
            for (int t2 = 0; t2 < kW; ++t2)
              if (t2 < list_len) j += f[t2] > __uint_as_float(mylist[list_len - 1 - t2].y);
            if (j > 0) {
#pragma unroll
              for (int i = 0; i < kW; i += 4)
                *reinterpret_cast<float4*>(myscratch + i) = make_float4(f[i], f[i + 1], f[i + 2], f[i + 3]);
              // in-place merge from the bottom: the smaller of the two tails goes to `pos`; equal ones
              // keep the list's entry (an earlier chunk) above
              int i = list_len - j - 1, jj = j - 1;
              for (int pos = list_len - 1; jj >= 0; --pos) {
                const uint32_t sk = myscratch[jj];
                if (i >= 0 && __uint_as_float(mylist[i].y) < __uint_as_float(sk)) {
                  mylist[pos] = mylist[i];
                  --i;
                } else {
                  mylist[pos] = entry(sk);
                  --jj;
                }
              }
            }
          }
          last = __uint_as_float(mylist[list_len - 1].y);
        } else {
          // order-preserving keys; places past the row's candidates get key 0
          uint32_t vmax = 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v[i] = i < rem ? float_key(__uint_as_float(v[i])) : 0u;
            vmax = max(vmax, v[i]);
          }
          if (!__any_sync(0xffffffffu, vmax > tau)) continue;
          uint32_t hits = 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) hits |= v[i] > tau ? (1u << i) : 0u;
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<uint4*>(myscratch + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
          // every lane walks its own hits; tau rises as it goes
          while (hits) {
            const int i = __ffs(hits) - 1;
            hits &= hits - 1;
            const uint32_t key = myscratch[i];
            if (key > tau) {
              heap_replace_root(mylist, list_len, key, chunk0 + (uint32_t)i);
              tau = mylist[0].y;
            }
          }
        }
      }
      tc_fence_before();
      if (c0 + nt < t.max_cand) {
        __syncthreads();                                      // the means and their estimates are consumed
        if (tid == 0) request_b(t, c0 + nt);
      }
    }

    // ---- a heap is sorted now: largest key first (equal scores in any order: they are rechecked) ----
    if (kW == 0)
      for (int m = list_len - 1; m > 0; --m) {
        const uint2 last = mylist[m];
        mylist[m] = mylist[0];
        heap_replace_root(mylist, m, last.y, last.x);
      }

    // ---- recheck ------------------------------------------------------------------------------
    // eps of this row (see the head of this section); inf or NaN sends the row to the exact ranking
    const float eps = gate_kappa<D, (kW > 0)> * sqrtf(q_ssq) * sqrtf(__int_as_float(c.mean_ssq_max)) + 7.9e-31f;
    const int n_keep = min(hist, ncand);
    auto value = [&](int i) { return kW > 0 ? __uint_as_float(mylist[i].y) : key_float(mylist[i].y); };   // estimate of entry i
    // 0: list is exact; 3: order the runs of near-ties (marked in the list); 1: rank all survivors;
    // 2: rank all candidates
    int mode = 0, n_surv = 0;
    if (ncand > 0) {
      int n_real = 0;
      for (int i = 0; i < list_len; ++i) n_real += (int32_t)mylist[i].x >= 0;
      if ((flags & GATE_FORCE_EXACT) || failed || n_real < min(ncand, list_len)) {
        mode = 2;
      } else {
        const float eps2 = 2.f * eps;
        const bool all = (flags & GATE_FORCE_RECHECK) != 0;
        // settled by the estimates alone? (the common case: nothing else is computed for the row)
        bool amb = all;
        {
          float prev = value(0);
          for (int i = 0; i < n_keep && i + 1 < n_real; ++i) {
            const float next = value(i + 1);
            if (!(prev - next > eps2)) amb = true;
            prev = next;
          }
        }
        // survivors: the only candidates that can be among the n_keep best exact scores
        if (amb) {
          const float theta = value(n_keep - 1) - eps2;
          while (n_surv < n_real && value(n_surv) >= theta) ++n_surv;
        }
        if (!amb) {
          mode = 0;
        } else if ((n_surv == list_len && ncand > list_len) || !(eps2 < INFINITY) || n_surv < n_keep) {
          mode = 2;            // the near-ties may go on below the list, or eps is not finite
        } else {
          // Runs of neighbours closer than 2 eps: entries of different runs are certainly in the
          // order of their estimates, entries of one run are ordered by their exact scores.  The
          // members of a run are marked in the chunk word (kTied, kRunStart on its first member).
          int tied = 0;
          bool in_run = false;
          float prev = value(0);
          for (int i = 0; i + 1 < n_surv; ++i) {
            const float next = value(i + 1);
            if (all || !(prev - next > eps2)) {
              if (!in_run) { mylist[i].x |= kTied | kRunStart; ++tied; }
              mylist[i + 1].x |= kTied;
              ++tied;
              in_run = true;
            } else {
              in_run = false;
            }
            prev = next;
          }
          if (all && tied == 0) {                             // a single survivor, scored again on request
            mylist[0].x |= kTied | kRunStart;
            tied = 1;
          }
          if (tied > 32) {     // more near-ties than one round of the warp ranks: rank all survivors instead
            for (int i = 0; i < n_surv; ++i) mylist[i].x &= kChunkMask;
            mode = 1;
          } else if (tied > 0) {
            mode = 3;
          }
        }
      }
    }
    __syncwarp();                                             // the marks are visible to the warp
    const __nv_bfloat16* qrow = q + (int64_t)(t.tok_lo + row / p.G - p.win_lo) * p.sq_t + (int64_t)(t.hk * p.G + row % p.G) * p.sq_h;
    rank_rows<kHalf, D, false, (kW > 0)>(p, GateLists{lists, lstride, list_len, c.exact[warp]}, t, qrow, row, mode, n_surv, n_keep, ncand, eps, means,
                        stats);
    // selected[rank][head][token]: every thread stores the chunks of its own row (its list was
    // written by its own warp); neighbouring lanes are neighbouring heads, then tokens
    if (row < nrows) {
      const int tl = row / p.G, hl = row - tl * p.G;
      int32_t* dst = selected + (int64_t)(t.hk * p.G + hl) * p.Tq + (t.tok_lo - p.win_lo) + tl;
      for (int r = 0; r < hist; ++r) {
        const uint32_t x = mylist[r].x;
        const int cc = x == 0xFFFFFFFFu ? -1 : (int)(x & kChunkMask);
        dst[(int64_t)r * p.sel_rs] = cc >= 0 ? slot0 + cc : -1;
        if (cc >= 0 && list_counts != nullptr) {
          if (cnt_in_smem) atomicAdd(&cnt_s[cc], 1);
          else atomicAdd(&list_counts[(int64_t)(slot0 + cc) * p.Hkv + t.hk], 1);
        }
      }
    }
    __syncthreads();                                          // lists, scratch and the Q buffer are free again
    if (cnt_in_smem && list_counts != nullptr)
      for (int cc = tid; cc < t.max_cand; cc += kGateThreads) {        // flush and clear this thread's counters
        const int m = cnt_s[cc];
        if (m > 0) {
          atomicAdd(&list_counts[(int64_t)(slot0 + cc) * p.Hkv + t.hk], m);
          cnt_s[cc] = 0;
        }
      }
    ++n;
  }

  if (ticket != nullptr) finish_scan<kGateThreads>(scan, ticket, reinterpret_cast<int*>(c.exact));
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, (uint32_t)nt);
}

struct GateLaunch {
  int nt, list_len, nbuf, cnt_in_smem, ctas_per_sm;
  size_t smem;
};

// Width of the network for a list, 0: none.
inline int gate_network(int list_len) { return list_len <= 8 ? 8 : list_len <= 16 ? 16 : list_len <= 32 ? 32 : 0; }
// At most 32 candidates a row and a list of at most 8, or a network for the list and few row tiles.  The kernel for few
// candidates saves latency of a row tile; with the wider networks it has three CTAs or fewer and keeps a row's whole list in
// registers (spills), and once every SM has its tiles the other one is ahead.  Gating kernel, this / the other, head dim 128, 31 candidates:
//   top-k 12  one new token 8.4 / 10.5 us, 700 24.1 / 24.0, 1500 31 / 30; 32768 x 16/4 206 / 163
//   top-k 24  one new token 12.8 / 14.5 us, 64 24.4 / 24.4, 256 31.5 / 29.6; 32768 x 16/4 350 / 177
// at head dim 64 the lines cross at 200 row tiles (top-k 24: 700 tokens x 16/4 24.4 / 24.8), at 256 at 12 (top-k 12: 8 tokens x 32/8
// 21.2 / 22.6, 64 32.9 / 31.0; 32768 x 32/8 745 / 575, top-k 24 1113 / 660).  Lists of 8: 32768 x 16/4 117 / 127, one token 7.6 / 9.5.
inline bool gate_one(const Params& p) {
  if (p.mc - 1 > kOneMeans || p.hist + 1 > 32) return false;
  if (p.hist + 1 <= 8) return true;
  const int few = p.D == 64 || (p.D <= 128 && p.hist + 1 <= 16) ? 148 : 16;
  return (int64_t)window_tiles(p, kGateRows / p.G) * p.Hkv * p.B <= few;
}
// Candidate tile, Q buffers, list length and shared memory of a launch: the combination that puts
// the most CTAs on an SM (more warps hide the latency of the list updates), then the wider candidate
// tile, then two Q buffers.  smem == 0: nothing fits.
GateLaunch gate_launch_config(const Params& p) {
  GateLaunch best{};
  const int nblk = (p.D + 63) / 64;
  // hist + 1 places settle the cut; more only help rows with more than 32 candidates (a row with
  // fewer is ranked over all of them in one round of the exact path anyway)
  const int list_len = p.hist + 1 + (p.mc - 1 > 32 ? kListExtra : 0);
  const int cnt_in_smem = p.mc <= kCntSmemMax;
  if (gate_one(p))
    return GateLaunch{kOneMeans, list_len, 1, 0, 4,
                      1024 + (size_t)nblk * kQBlockBytes + (size_t)nblk * kOneMeans * 128 +
                          (size_t)kGateRows * (list_len | 1) * sizeof(uint2) + sizeof(OneCtrl)};
  const int w = gate_network(list_len);
  // No more CTAs than the register budget is set for: counted for a fourth, the kernels of the wider networks had tiles of
  // 32 candidates, and a round trip of TMA and MMA for each 32 of a row (32768 x 32/8, 255 candidates 577 -> 543 us
  // with 64).  (The min-heap's lists leave shared memory for three at most, whatever is counted here.)
  const int max_ctas = w == 8 ? kGateMinCtas<8> : w == 16 ? kGateMinCtas<16> : w == 32 ? kGateMinCtas<32> : kGateMinCtas<0>;
  int want = 32;
  while (want < p.mc - 1 && want < 256) want *= 2;            // a row has at most mc - 1 candidates
  for (int nt = want; nt >= 32; nt /= 2)
    for (int nbuf = 2; nbuf >= 1; --nbuf) {
      const size_t smem = 1024 + (size_t)nbuf * nblk * kQBlockBytes + (size_t)nblk * nt * 128 +
                          (size_t)kGateRows * (list_len | 1) * sizeof(uint2) +
                          (has_scratch(p.mc, w) ? (size_t)kGateRows * scratch_stride(w) * sizeof(float) : 0) + sizeof(GateCtrl) +
                          (cnt_in_smem ? (size_t)p.mc * sizeof(int32_t) : 0);
      if (smem > 227 * 1024) continue;
      int ctas = (int)((228 * 1024) / (smem + 1024));         // 1 KB per CTA is reserved by the system
      if (ctas > 512 / nt) ctas = 512 / nt;                   // tensor memory columns
      if (ctas > max_ctas) ctas = max_ctas;
      if (ctas < 1) continue;
      if (ctas > best.ctas_per_sm) best = GateLaunch{nt, list_len, nbuf, cnt_in_smem, ctas, smem};
    }
  return best;
}

}  // namespace

bool make_tile_map(CUtensorMap* m, bool fp16, int D, const __nv_bfloat16* base, int64_t T, int H, int64_t st,
                   int64_t sh, int box_heads, int box_rows);

bool gate_topk_fits(const Params& p) { return p.hist <= 0 || gate_launch_config(p).smem != 0; }

cudaError_t launch_gate_topk_stats(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* means,
                                   const int32_t* cu, int32_t* selected, int32_t* list_counts, int32_t* stats,
                                   int flags, cudaStream_t st, const ListScan* scan, int32_t* ticket, bool chained) {
  int tokens_per_cta = kGateRows / p.G;
  if (tokens_per_cta < 1) return cudaErrorInvalidConfiguration;
  const GateLaunch g = gate_launch_config(p);
  if (g.smem == 0) return cudaErrorInvalidConfiguration;
  CUtensorMap mq, mm;
  if (!make_tile_map(&mq, p.fp16 != 0, p.D, q, p.Tq, p.Hq, p.sq_t, p.sq_h, p.G, tokens_per_cta) ||
      !make_tile_map(&mm, p.fp16 != 0, p.D, means, p.slots, p.Hkv, (int64_t)p.Hkv * p.D, p.D, 1, g.nt))
    return cudaErrorNotSupported;
  typedef void (*Kernel)(Params, CUtensorMap, CUtensorMap, int, int, int, int, int, const __nv_bfloat16*,
                         const __nv_bfloat16*, const int32_t*, int32_t*, int32_t*, int32_t*, int, ListScan, int32_t*);
  Kernel kernel = nullptr;
  const int w = gate_network(g.list_len);
  const bool one = gate_one(p);
#define MOBA_GATE_W(HALF, DIM)                                                                       \
  kernel = one ? (w == 8 ? (Kernel)gate_one_kernel<HALF, DIM, 8> : w == 16 ? (Kernel)gate_one_kernel<HALF, DIM, 16>   \
                                                                   : (Kernel)gate_one_kernel<HALF, DIM, 32>)         \
         : w == 8 ? (Kernel)gate_topk_kernel<HALF, DIM, 8> : w == 16 ? (Kernel)gate_topk_kernel<HALF, DIM, 16> \
         : w == 32 ? (Kernel)gate_topk_kernel<HALF, DIM, 32> : (Kernel)gate_topk_kernel<HALF, DIM, 0>
  switch (p.D) {
    case 64:  if (p.fp16) MOBA_GATE_W(true, 64);  else MOBA_GATE_W(false, 64);  break;
    case 96:  if (p.fp16) MOBA_GATE_W(true, 96);  else MOBA_GATE_W(false, 96);  break;
    case 128: if (p.fp16) MOBA_GATE_W(true, 128); else MOBA_GATE_W(false, 128); break;
    case 256: if (p.fp16) MOBA_GATE_W(true, 256); else MOBA_GATE_W(false, 256); break;
    default: return cudaErrorInvalidValue;
  }
#undef MOBA_GATE_W
  int regs = 0;
  const cudaError_t e = prepare_kernel(kernel, g.smem, &regs, true);
  if (e != cudaSuccess) return e;
  const DeviceInfo dev = device_info();
  const int64_t n_tiles = (int64_t)window_tiles(p, tokens_per_cta) * p.Hkv * p.B;
  if (n_tiles >= ((int64_t)1 << 31)) return cudaErrorInvalidConfiguration;
  // persistent CTAs: as many as are resident at once, by shared memory (1 KB per CTA is reserved),
  // registers (allocated in units of 8 per thread) and tensor memory (512 columns per SM)
  int resident = (int)(dev.smem_per_sm / (g.smem + 1024));
  const int threads = one ? kOneThreads : kGateThreads;
  const int regs_per_cta = ((regs + 7) / 8 * 8) * threads;
  if (regs_per_cta > 0 && resident > dev.regs_per_sm / regs_per_cta) resident = dev.regs_per_sm / regs_per_cta;
  if (resident > 512 / g.nt) resident = 512 / g.nt;
  if (resident < 1) resident = 1;
  int64_t grid = (int64_t)dev.sms * resident;
  if (grid > n_tiles) grid = n_tiles;
  return launch_chained(chained, kernel, dim3((unsigned)grid), threads, g.smem, st, p, mq, mm, tokens_per_cta, g.nt,
                        g.list_len, g.nbuf, g.cnt_in_smem, q, means, cu, selected, list_counts, stats, flags,
                        scan ? *scan : ListScan{}, scan ? ticket : nullptr);
}

cudaError_t launch_gate_topk(const Params& p, const __nv_bfloat16* q, const __nv_bfloat16* means,
                             const int32_t* cu, int32_t* selected, int32_t* list_counts,
                             cudaStream_t st, const ListScan* scan, int32_t* ticket, bool chained) {
  return launch_gate_topk_stats(p, q, means, cu, selected, list_counts, nullptr, 0, st, scan, ticket, chained);
}

}  // namespace moba
