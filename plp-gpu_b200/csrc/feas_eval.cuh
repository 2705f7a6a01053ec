// feas_eval.cuh -- lookups in a table of placed boxes held sorted by top z, by
// the top-z index where there is one, for the multi-warp decoder (decoder.cu).
#pragma once

#include "device_common.cuh"

namespace plpb {

__device__ __forceinline__ int lower_bound_top(const int* z2, int n, int z) {
    int lo = 0;
    while (n > 0) {
        const int half = n >> 1;
        if (z2[lo + half] < z) {
            lo += half + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    return lo;
}

// First box with top >= z from the top-z index zt (zt[z] = boxes with top
// < z), or by binary search when there is no index.
__device__ __forceinline__ int box_start(const unsigned short* zt, const int* z2, int nb, int z) {
    return zt ? (int)zt[z] : lower_bound_top(z2, nb, z);
}

}  // namespace plpb
