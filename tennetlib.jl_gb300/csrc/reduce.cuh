// Warp sums of several FP64 values per lane.
//
// A warp-wide FP64 add holds its SM sub-partition for 64 clocks, so the plain butterfly (5 adds
// per value, the same sum formed in every lane) costs 320 clocks per value.  Here the lanes of
// one half of a pair keep half of the values and hand over the others, so C values take
// C/2 + C/4 + ... + 1 adds and the remaining steps one each: 6 adds for 4 values instead of 20,
// 31 for 32 instead of 160.  Every value is added in the butterfly's order, so the sums are
// the same bits.
#pragma once

#include <cuda_runtime.h>

namespace tn {

// v[0..C): C a power of two up to 32.  Returns the sum of value warp_sum_index<C>(lane), which
// the lanes with warp_sum_owner<C>(lane) own (the others hold copies).
template <int C>
__device__ __forceinline__ double warp_sum_multi(double (&v)[C], int lane) {
    int c = C;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (c > 1) {
            const int h = c / 2;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const double keep = up ? v[h + i] : v[i];
                const double give = up ? v[i] : v[h + i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
            c = h;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return v[0];
}
template <int C>
__device__ __forceinline__ int warp_sum_index(int lane) {
    int idx = 0;
#pragma unroll
    for (int o = 16, h = C / 2; h > 0; o >>= 1, h >>= 1)
        if (lane & o) idx += h;
    return idx;
}
template <int C>
__device__ __forceinline__ bool warp_sum_owner(int lane) {
    return (lane & (32 / C - 1)) == 0;
}

}  // namespace tn
