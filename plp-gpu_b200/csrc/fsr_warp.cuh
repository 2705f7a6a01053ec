// fsr_warp.cuh -- FSR stability score of one packing by one warp, over the
// packing's boxes held sorted by top z in shared memory. Shared by the
// extreme-point decoder (decoder.cu), the block engine (block.cu) and the
// standalone fsr_kernel.
#pragma once

#include <climits>

#include "device_common.cuh"

namespace plpb {

// Box tables sorted by top z, as the callers keep them.
struct WideBoxes {
    const int4* bx;               // {x, y, x2, y2}
    const int* bz;                // bottom z
    const int* z2;                // top z
    const unsigned short* bi;     // placement index
    __device__ __forceinline__ int4 xy(int p) const { return bx[p]; }
    __device__ __forceinline__ int bottom(int p) const { return bz[p]; }
    __device__ __forceinline__ int top(int p) const { return z2[p]; }
    __device__ __forceinline__ int index(int p) const { return bi[p]; }
};

// {x | x2 << 16, y | y2 << 16, z | z2 << 16, placement index}
struct PackedBoxes {
    const uint4* b;
    __device__ __forceinline__ int4 xy(int p) const {
        const uint2 v = *reinterpret_cast<const uint2*>(b + p);
        return make_int4((int)(v.x & 0xffffu), (int)(v.y & 0xffffu), (int)(v.x >> 16), (int)(v.y >> 16));
    }
    __device__ __forceinline__ int bottom(int p) const { return (int)(b[p].z & 0xffffu); }
    __device__ __forceinline__ int top(int p) const { return (int)(b[p].z >> 16); }
    __device__ __forceinline__ int index(int p) const { return (int)b[p].w; }
};

// First box with top >= z.
template <class Boxes>
__device__ __forceinline__ int first_top(const Boxes& B, int n, int z) {
    int lo = 0;
#pragma unroll 1
    while (n > 0) {
        const int half = n >> 1;
        if (B.top(lo + half) < z) {
            lo += half + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    return lo;
}

// Overlap area of two footprints {x, y, x2, y2}.
__device__ __forceinline__ int contact_area(const int4& b, const int4& c) {
    const int ox = min(b.z, c.z) - max(b.x, c.x), oy = min(b.w, c.w) - max(b.y, c.y);
    return ox > 0 && oy > 0 ? ox * oy : 0;
}

// ---------------------------------------------------------------------------
// FSR of the packing held in the box tables (warp). Load flows from each box
// k, taken in (z desc, placement index asc) order, to the boxes whose top is
// k's bottom, proportionally to the integer contact area. Levels are handled
// in descending z; inside a level the boxes k are taken in index order and
// the supports j are updated in parallel (each j by one lane), so every
// load[j] receives its additions in the reference order.
//
// The order needs no sort: a maximum over the bottoms below the last level
// gives the next one, and ballots over the bottoms by placement index give its
// boxes in order. A box's contact total is one reduction over the lanes of its
// supports. The chain of levels bounds it; with a bitonic sort, a pass for the
// totals and a search per level boundary one decode's score took 36 k cycles
// alone on an SM and 57 k among 18 others.
// ---------------------------------------------------------------------------
// zt (may be null): the top-z index zt[z] = number of boxes with top < z, so
// the boxes with top exactly z are [zt[z], zt[z + 1]) without a search.
// scratch: 14 bytes per box, 8-byte aligned.
template <int SPACE = 0, class Boxes>   // SPACE as for the MT helpers
static __device__ __noinline__ double fsr_score_warp(const Boxes B, int n, double mu, char* scratch, int lane,
                                                     double* fsr_out, const unsigned short* zt = nullptr) {
    if (n == 0) return 0.0;
    double* load = reinterpret_cast<double*>(scratch);                          // by sorted position
    int* zb = reinterpret_cast<int*>(scratch + 8 * n);                          // bottom by index
    unsigned short* pos = reinterpret_cast<unsigned short*>(scratch + 12 * n);  // index -> position
#pragma unroll 1
    for (int p = lane; p < n; p += 32) {
        const int4 b = B.xy(p);
        const int z = B.bottom(p), i = B.index(p);
        const long long vol = 1LL * (b.z - b.x) * (b.w - b.y) * (B.top(p) - z);
        load[p] = 50.0 * (double)vol / 1e6;
        zb[i] = z;
        pos[i] = (unsigned short)p;
    }
    __syncwarp();
    int zl = INT_MAX;
#pragma unroll 1
    for (;;) {
        int m = 0;
#pragma unroll 1
        for (int i = lane; i < n; i += 32) {
            const int z = zb[i];
            if (z < zl) m = max(m, z);
        }
        zl = __reduce_max_sync(FULL, m);
        if (zl <= 0) break;
        const int jlo = zt ? (int)zt[zl] : first_top(B, n, zl);
        const int jhi = zt ? (int)zt[zl + 1] : first_top(B, n, zl + 1);
#pragma unroll 1
        for (int jb = jlo; jb < jhi; jb += 32) {
            const int j = jb + lane;
            const bool in = j < jhi;
            const int4 c = in ? B.xy(j) : make_int4(0, 0, 0, 0);
            double lj = in ? load[j] : 0.0;
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += 32) {
                unsigned ks = __ballot_sync(FULL, i0 + lane < n && zb[i0 + lane] == zl);
#pragma unroll 1
                for (; ks; ks &= ks - 1) {
                    const int k = pos[i0 + __ffs(ks) - 1];
                    const int4 b = B.xy(k);
                    const int a = contact_area(b, c);   // 0 where !in
                    int total = a;
                    if (jhi - jlo > 32) {               // supports of more than one round
                        total = 0;
#pragma unroll 1
                        for (int q = jlo + lane; q < jhi; q += 32) total += contact_area(b, B.xy(q));
                    }
                    total = __reduce_add_sync(FULL, total);
                    if (a > 0) lj += load[k] * (double)a / (double)total;
                }
            }
            if (in) load[j] = lj;
        }
        __syncwarp();
    }
    int cnt = 0;
#pragma unroll 1
    for (int p = lane; p < n; p += 32) {
        const int4 b = B.xy(p);
        const long long vol = 1LL * (b.z - b.x) * (b.w - b.y) * (B.top(p) - B.bottom(p));
        const double m = 50.0 * (double)vol / 1e6;
        const double f = (mu / 0.3) * load[p] / m;
        if (fsr_out) fsr_out[B.index(p)] = f;
        cnt += f >= 1.0;
    }
    cnt = __reduce_add_sync(FULL, cnt);
    return (double)cnt / (double)n;
}

}  // namespace plpb
