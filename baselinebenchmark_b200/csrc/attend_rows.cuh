// Pieces of the forward's dense-stage kernels on tcgen05 that more than one of them uses: tile sizes, instruction
// and shared-memory descriptors, the softmax step of a row in loops, and the epilogue of a row.
#pragma once

#include "common.cuh"
#include "short_items.cuh"
#include "sm100_ptx.cuh"

namespace moba {
namespace {

using namespace ptx;

constexpr int kTileM = 128;              // rows per MMA tile
constexpr int kBN = 128;                 // keys per K/V tile
constexpr int kHalfBytes = 128 * 64 * 2; // one [128][64] bf16 swizzled block
constexpr int kTileBytes = 2 * kHalfBytes;

template <bool kHalf> constexpr uint32_t kIdescQK = idesc_16_f32(kHalf, 128, kBN, 0, 0);
template <bool kHalf, int D> constexpr uint32_t kIdescPV = idesc_16_f32(kHalf, 128, D, 0, 1);

enum { ST_OK = 0, ST_PRODUCER = 1, ST_MMA = 2, ST_SOFTMAX = 3 };

// Pairs of score columns whose exponential is evaluated with the cubic on the
// FMA pipe instead of the special-function unit: kPolyPairs out of every 8.
// The special-function unit sustains 16 ex2 per clock and SM, which is exactly
// the rate two 128x128 MMAs per 1024 cycles would ask of it.
#ifndef MOBA_POLY_PAIRS
#define MOBA_POLY_PAIRS 2
#endif
constexpr int kPolyPairs = MOBA_POLY_PAIRS;

struct KernelArgs {
  const __nv_bfloat16* q;
  const int32_t* cu;
  const int32_t* list_counts;
  const int32_t* list_offsets;
  const int32_t* tile_prefix;
  const int32_t* row_list;
  __half* partial_out;                     // fp16 rows scaled by a power of two per row
  float2* partial_lse;                     // {natural-log LSE, 1 / scale}
  int32_t* work_counter;
  int32_t* status;
  int32_t wide_store;                      // partial_out is 32-byte aligned
};
struct ShortArgs {
  KernelArgs a;
  ItemQueue iq;
};

// The step of softmax_row (attend_tc5.cu) with the scores read twice and 32 columns at a time, in loops: for kernels whose items are one or two
// key tiles.  Unrolled, the step and the epilogue are some 50 KB of straight-line code that such an item
// runs through once, and fetching it took longer than executing it (4300 cycles a step and 4200 an
// epilogue, at a quarter of the issue slots); the loops are a few KB.  P of 32 columns never covers
// scores still to be read.  Same operations in the same order as there: the same bits.
template <bool kMasked, bool kHalf, int D, typename F>
__device__ __forceinline__ void softmax_row_rolled(uint32_t tS, uint32_t tO, int j, int key0, int lim, float sl2,
                                                   float& m_ref, float& l, F&& before_rescale) {
  float mx = -INFINITY;
  int rem = lim - key0;                    // visible columns left
#pragma unroll 1
  for (int ch = 0; ch < 4; ++ch, rem -= 32) {
    uint32_t v[32];
    tmem_ld32(tS + ch * 32, v);
    tmem_wait_ld();
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      if (kMasked) {
#pragma unroll
        for (int u = 0; u < 4; ++u) v[i + u] = i + u < rem ? v[i + u] : 0xff800000u;   // -inf
      }
      mx0 = max3(mx0, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      mx1 = max3(mx1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
    }
    mx = max3(mx, mx0, mx1);
  }
  const float m_new = fmaxf(m_ref, mx * sl2);
  const bool up = m_new > m_ref + 8.f;
  if (__any_sync(0xffffffffu, up)) {
    const float alpha = up ? ex2_approx(m_ref - m_new) : 1.f;
    if (j > 0) {
      before_rescale();
#pragma unroll 1
      for (int ch = 0; ch < D / 32; ++ch) {
        uint32_t o[32];
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
  rem = lim - key0;
#pragma unroll 1
  for (int ch = 0; ch < 4; ++ch, rem -= 32) {
    uint32_t v[32], pk[16];
    tmem_ld32(tS + ch * 32, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      uint32_t e0 = v[2 * i], e1 = v[2 * i + 1];
      if (kMasked) {
        e0 = 2 * i < rem ? e0 : 0xff800000u;
        e1 = 2 * i + 1 < rem ? e1 : 0xff800000u;
      }
      const uint64_t x = fma2(pack2(__uint_as_float(e0), __uint_as_float(e1)), scale2, negm2);
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

// Epilogue of a row in loops over 32 columns: the largest magnitude of the O row, whose first 64 dims are at column tO
// and the others at tHi, ...
template <int D>
__device__ __forceinline__ float amax_row_rolled(uint32_t tO, uint32_t tHi) {
  float a0 = 0.f, a1 = 0.f;
#pragma unroll 1
  for (int ch = 0; ch < D; ch += 32) {
    uint32_t v[32];
    tmem_ld32((ch < 64 ? tO : tHi - 64) + ch, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      a0 = max3(a0, fabsf(__uint_as_float(v[i])), fabsf(__uint_as_float(v[i + 1])));
      a1 = max3(a1, fabsf(__uint_as_float(v[i + 2])), fabsf(__uint_as_float(v[i + 3])));
    }
  }
  return fmaxf(a0, a1);
}
// ... and the row itself, scaled, as fp16 in 32-byte stores (`wide`; 16-byte ones otherwise) for the lanes with a row
// (`on`).  `drained` runs (warp-uniformly) when the last of O has been read.
template <int D, typename F>
__device__ __forceinline__ void store_row_rolled(uint32_t tO, uint32_t tHi, __half* dst, float mul, bool on, bool wide, F&& drained) {
#pragma unroll 1
  for (int ch = 0; ch < D; ch += 32) {
    uint32_t v[32];
    tmem_ld32((ch < 64 ? tO : tHi - 64) + ch, v);
    tmem_wait_ld();
    if (ch + 32 == D) drained();
    if (on) {
#pragma unroll
      for (int i = 0; i < 32; i += 16) {
        uint32_t pk[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint64_t x = mul2(pack2(__uint_as_float(v[i + 2 * u]), __uint_as_float(v[i + 2 * u + 1])), pack2(mul, mul));
          pk[u] = pack2_half(lo2(x), hi2(x));
        }
        if (wide) {
          store32(dst + ch + i, pk);
        } else {
          *reinterpret_cast<uint4*>(dst + ch + i) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          *reinterpret_cast<uint4*>(dst + ch + i + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
      }
    }
    __syncwarp();
  }
}

// Descriptor words.  Low word: start address >> 4 | (leading byte offset >> 4) << 16;
// high word (constant): stride byte offset 1024 >> 4 | version 1 << 14 | SWIZZLE_128B (2) << 29.
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr, uint32_t lbo_bytes) {
  return ((addr & 0x3FFFFu) >> 4) | ((lbo_bytes >> 4) << 16);
}
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint64_t desc64(uint32_t lo) { return ((uint64_t)kDescHi << 32) | lo; }

}  // namespace
}  // namespace moba
