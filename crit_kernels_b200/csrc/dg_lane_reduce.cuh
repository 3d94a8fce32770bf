// Reduction of several values over a warp's lanes at once.
#pragma once
#include <cuda_runtime.h>

namespace dg {

// Lane reduction of V values per lane at once: the xor-shuffle tree 16, 8, 4, 2, 1 of every value, with the values
// split between the two partners at each level so that a level costs one shuffle per value pair instead of one per
// value. For each value the additions are those of the plain tree, pair by pair (a + b is commutative in IEEE
// arithmetic), so the bits are the plain tree's. After the last level value v's total sits in lane (v % 32),
// slot v / 32.
template <int V, int OFFSET, int NOUT>
struct LaneReduce {
  static constexpr int H = (V + 1) / 2;   // values kept per lane after this level
  __device__ __forceinline__ static void run(float (&val)[V], int lane, float (&out)[NOUT]) {
    if constexpr (V == 1) {
      float v = val[0];
#pragma unroll
      for (int o = OFFSET; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      out[0] = v;
    } else if constexpr (OFFSET == 0) {
      static_assert(V <= NOUT, "lane reduction output too small");
#pragma unroll
      for (int i = 0; i < V; ++i) out[i] = val[i];
    } else {
      // lanes with the OFFSET bit clear keep values [0, H) and send [H, V); the others keep [H, V) and send [0, H)
      const bool upper = (lane & OFFSET) != 0;
      float keep[H];
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const bool has_hi = H + i < V;
        const float lo = val[i], hi = has_hi ? val[H + i] : 0.0f;
        const float got = __shfl_xor_sync(0xffffffffu, upper ? lo : hi, OFFSET);
        // a value without a partner slot (odd V) is finished by the lower lanes; the upper lanes carry a zero there
        keep[i] = (upper ? hi : lo) + (has_hi || !upper ? got : 0.0f);
      }
      LaneReduce<H, OFFSET / 2, NOUT>::run(keep, lane, out);
    }
  }
};

// Which of the V values lane `lane` holds in output slot `slot` after LaneReduce<V, 16, .> (-1: none).
template <int V>
__device__ __forceinline__ int lane_value(int lane, int slot) {
  int size = V, real = V, base = 0;   // entries [0, real) of this lane's array are values base, base + 1, ...
  for (int o = 16; o > 0; o >>= 1) {
    if (size == 1) return (real == 1 && slot == 0 && (lane & (2 * o - 1)) == 0) ? base : -1;
    const int h = (size + 1) / 2;
    if (lane & o) {
      base += h;
      real = real > h ? real - h : 0;
    } else {
      real = real < h ? real : h;
    }
    size = h;
  }
  return slot < real ? base + slot : -1;
}

}  // namespace dg
