// Compare-exchange networks over 32 floats held in registers (every index is a compile-time
// constant after unrolling): the W largest of them, in descending order.
//
//   1. bitonic sort inside groups of W values, even groups descending, odd groups ascending;
//   2. halving rounds: a descending group and its ascending neighbour are combined by taking
//      the element-wise maximum (a bitonic sequence that holds the W largest of the 2 W values)
//      which is then merged into a sorted group again, descending or ascending so that the next
//      round finds the same arrangement.
// Cost in compare-exchanges: W = 8: 156, W = 16: 208, W = 32: 240 (a full sort).
// A NaN is dropped, and the value it met may be there twice: a caller with one among its values has to rank them otherwise.
#pragma once

namespace moba {
namespace topk {

// after the call: hi = max, lo = min
__device__ __forceinline__ void ce(float& hi, float& lo) {
  const float a = fmaxf(hi, lo), b = fminf(hi, lo);
  hi = a;
  lo = b;
}

// Bitonic merge of the bitonic sequence v[base, base + W) into descending (kDesc) or ascending order.
template <int W, bool kDesc>
__device__ __forceinline__ void bitonic_merge(float (&v)[32], int base) {
#pragma unroll
  for (int j = W / 2; j > 0; j >>= 1)
#pragma unroll
    for (int i = 0; i < W; ++i)
      if ((i & j) == 0) {
        if (kDesc) ce(v[base + i], v[base + i + j]);
        else ce(v[base + i + j], v[base + i]);
      }
}

// Sorts v[base, base + W) (any order) descending or ascending.
template <int W, bool kDesc>
__device__ __forceinline__ void bitonic_sort(float (&v)[32], int base) {
  if constexpr (W > 1) {
    bitonic_sort<W / 2, true>(v, base);
    bitonic_sort<W / 2, false>(v, base + W / 2);
    bitonic_merge<W, kDesc>(v, base);
  }
}

// The W largest of the 32 values end up in v[0, W), largest first; the rest of v is unspecified.
template <int W>
__device__ __forceinline__ void top_of_32(float (&v)[32]) {
  static_assert(W == 8 || W == 16 || W == 32, "W is 8, 16 or 32");
  if constexpr (W == 32) {
    bitonic_sort<32, true>(v, 0);
  } else {
    // groups g = 0, 1, ...: even ones descending, odd ones ascending
#pragma unroll
    for (int g = 0; g < 32 / W; ++g) {
      if (g % 2 == 0) bitonic_sort<W, true>(v, g * W);
      else bitonic_sort<W, false>(v, g * W);
    }
    // halving rounds over the group pairs (0,1), (2,3), ...: the result of pair k goes to group k
#pragma unroll
    for (int groups = 32 / W; groups > 1; groups /= 2) {
#pragma unroll
      for (int k = 0; k < groups / 2; ++k) {
        const int a = 2 * k * W, b = (2 * k + 1) * W, dst = k * W;
#pragma unroll
        for (int i = 0; i < W; ++i) v[dst + i] = fmaxf(v[a + i], v[b + i]);
        if (k % 2 == 0) bitonic_merge<W, true>(v, dst);
        else bitonic_merge<W, false>(v, dst);
      }
    }
  }
}

}  // namespace topk
}  // namespace moba
