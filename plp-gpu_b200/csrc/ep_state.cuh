// ep_state.cuh -- the packing state of one single-warp decoder: placed boxes
// sorted by top (PackedBoxes), the top-z index, and the live extreme points with
// their free extents; and the update a placement makes. Shared by the
// extreme-point decoder (decoder.cu, which describes the extents) and the
// block engine (block.cu).
#pragma once

#include "device_common.cuh"
#include "fsr_warp.cuh"

namespace plpb {

// First box with top >= z: from the top-z index, or by search without one.
__device__ __forceinline__ int top_start(const unsigned short* zt, const uint4* bx, int nb, int z) {
    return zt ? (int)zt[z] : first_top(PackedBoxes{bx}, nb, z);
}

// Smallest and largest edges over the instance's orientations (InstDesc) and
// the container.
struct EdgeRange {
    int w, d, h;      // smallest along x, y, z
    int Mw, Md, Mh;   // largest
    int L, W, H;
};

constexpr uint32_t PT_MARKED = 1u << 16;   // z extent word: a box meets the extents' cuboid

// A new box's corner coordinates (px .. px2 and so on) and the far ends of the
// smallest-edge cuboid at them. Sets of corners are eight-bit masks over
// c = (z2 << 2) | (y2 << 1) | x2.
struct CornerFrame {
    int x, y, z, x2, y2, z2;
    int xm, ym, zm, x2m, y2m, z2m;
    // The corners whose smallest-edge cuboid a placed box meets.
    __device__ __forceinline__ unsigned meets(const uint4& v) const {
        const int bx2 = (int)(v.x >> 16), by2 = (int)(v.y >> 16), bt = (int)(v.z >> 16);
        const int bx = (int)(v.x & 0xffffu), by = (int)(v.y & 0xffffu), bz = (int)(v.z & 0xffffu);
        // (reaching past the far corner implies reaching past the near one, and
        // beginning before the near end implies before the far one)
        return (x2 < bx2 ? 0xffu : x < bx2 ? 0x55u : 0u) & (y2 < by2 ? 0xffu : y < by2 ? 0x33u : 0u) &
               (z2 < bt ? 0xffu : z < bt ? 0x0fu : 0u) & (bx < xm ? 0xffu : bx < x2m ? 0xaau : 0u) &
               (by < ym ? 0xffu : by < y2m ? 0xccu : 0u) & (bz < zm ? 0xffu : bz < z2m ? 0xf0u : 0u);
    }
};

// Warp: places a w x d x h box at the point with key pkey: top-sorted box
// tables, top-z index, and the points K (arrays of `cap` entries: key,
// x | y << 16 extents, z extent | mark): the box is applied to every point,
// dead ones give up their slots, and the box's live corners come in.
__device__ __forceinline__ int place1(uint32_t pkey, int pw, int pd, int ph, uint32_t* K, int cap,
                                      unsigned short* free_slots, uint4* bx,
                                      unsigned short* zt, int Hz, int& nc, int& nb, int P, int C, uint32_t xmask,
                                      uint32_t ymask, int xb, int xyb, const EdgeRange& ME, int lane) {
    const int px = (int)(pkey & xmask), py = (int)((pkey >> xb) & ymask), pz = (int)(pkey >> xyb);
    const int px2 = px + pw, py2 = py + pd, pz2 = pz + ph;
    if (nb >= P) return ERR_BOX_CAP;
    // Box tables, one pass from the top: the corners of the new box that a
    // placed box makes dead, and the boxes whose top is above the new box's
    // move up one slot (each round reads before it writes, and writes only
    // slots it or an earlier round has read).
    const CornerFrame F{px, py, pz, px2, py2, pz2, px + ME.w, py + ME.d, pz + ME.h, px2 + ME.w, py2 + ME.d, pz2 + ME.h};
    unsigned dead = 1u;   // corner 0 = (px, py, pz): inside the new box
    if (F.x2m > ME.L) dead |= 0xaau;
    if (F.y2m > ME.W) dead |= 0xccu;
    if (F.z2m > ME.H) dead |= 0xf0u;
    int nabove = 0;
#pragma unroll 1
    for (int hi = nb; hi > 0; hi -= 32) {
        const int jj = hi - 1 - lane;
        const bool in = jj >= 0;
        const uint4 v = in ? bx[jj] : make_uint4(0, 0, 0, 0);   // the empty box lies before every corner
        dead |= F.meets(v);
        const bool up = in && (int)(v.z >> 16) > pz2;
        nabove += __popc(__ballot_sync(FULL, up));
        __syncwarp();
        if (up) bx[jj + 1] = v;
    }
    unsigned live = ~__reduce_or_sync(FULL, dead) & 0xffu;
    {
        const int ip = nb - nabove;   // after the boxes with equal tops
        __syncwarp();
        if (lane == 0) {
            bx[ip] = make_uint4((uint32_t)px | (uint32_t)px2 << 16, (uint32_t)py | (uint32_t)py2 << 16,
                                (uint32_t)pz | (uint32_t)pz2 << 16, (uint32_t)nb);
        }
    }
    if (zt) {
        // entries above the new top, two to a word (counts stay below 2^16), four words a lane in flight
        const int z0 = pz2 + 1;
        if ((z0 & 1) && lane == 0) zt[z0]++;
        uint32_t* zw = reinterpret_cast<uint32_t*>(zt);
#pragma unroll 1
        for (int w = ((z0 + 1) >> 1) + lane; w < Hz >> 1; w += 128) {
            uint32_t v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = w + 32 * u < Hz >> 1 ? zw[w + 32 * u] : 0u;
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (w + 32 * u < Hz >> 1) zw[w + 32 * u] = v[u] + 0x10001u;
        }
    }
    nb++;
    // Points in place. A corner that a point already lies on is not new.
    int nf = 0;            // slots freed
    unsigned dup = 0;      // corners this lane has met
#pragma unroll 1
    for (int cb = 0; cb < nc; cb += 32) {
        const int i = cb + lane;
        const bool in = i < nc;
        const uint32_t key = in ? K[i] : 0u, exy = in ? K[cap + i] : 0u, ezm = in ? K[2 * cap + i] : 0u;
        const int x = (int)(key & xmask), y = (int)((key >> xb) & ymask), z = (int)(key >> xyb);
        bool gone = in && exy == 0u;   // dead since a placement that freed more slots than it noted
        if (in && x < px2 && y < py2 && z < pz2) {   // else the box lies before the point
            int ex = (int)(exy & 0xffffu), ey = (int)(exy >> 16), ez = (int)(ezm & 0xffffu);
            const int dx = px - x, dy = py - y, dz = pz - z;
            const bool ix = dx < ME.w, iy = dy < ME.d, iz = dz < ME.h;
            if (iy && iz) ex = min(ex, dx);
            if (ix && iz) ey = min(ey, dy);
            if (ix && iy) ez = min(ez, dz);
            gone = ex < ME.w || ey < ME.d || ez < ME.h;
            const uint32_t mark = dx < ex && dy < ey && dz < ez ? PT_MARKED : ezm & PT_MARKED;
            K[cap + i] = gone ? 0u : (uint32_t)ex | ((uint32_t)ey << 16);
            K[2 * cap + i] = (uint32_t)ez | mark;
        }
        if ((x == px || x == px2) && (y == py || y == py2) && (z == pz || z == pz2))
            dup |= 1u << ((x == px2 ? 1 : 0) | (y == py2 ? 2 : 0) | (z == pz2 ? 4 : 0));
        const unsigned fr = __ballot_sync(FULL, gone);
        if (fr) {
            const int q = nf + __popc(fr & lanemask_lt());
            if (gone && q < 32) free_slots[q] = (unsigned short)i;
            nf += __popc(fr);
        }
    }
    // (Lanes past the end read key 0, the container's corner: never a live corner.)
    live &= ~__reduce_or_sync(FULL, dup);
    __syncwarp();   // box tables, top-z index, points and freed slots are final
    // New points take freed slots, or come after the end; the last point fills
    // a slot left over. Slots past the 32nd freed in one placement keep their
    // dead point (no extents), whose slot the next placement frees.
    nf = min(nf, 32);
    const int nl = __popc(live), nc0 = nc;
#pragma unroll 1
    for (int q = nf - 1; q >= nl; q--) {   // from the highest slot: the last point is alive or in it
        const int h = free_slots[q];
        nc--;
        if (h != nc && lane < 3) K[lane * cap + h] = K[lane * cap + nc];
        __syncwarp();
    }
    nc += max(nl - nf, 0);
    if (nc > C) return ERR_CAND_CAP;
    if (nl == 0) return ERR_NONE;
    // Extents of the new corners, all at once: 2^sh lanes to a corner, each
    // taking every 2^sh-th box above the new box's bottom (2.6 live corners and
    // some 20 boxes a placement: three rounds). With one corner after another,
    // the lanes over the boxes and three reductions each, this took 280
    // instructions a placement, 19 % of a decode.
    const int sh = nl <= 1 ? 5 : nl <= 2 ? 4 : nl <= 4 ? 3 : 2;
    const int g = lane >> sh, step = 1 << sh;
    unsigned mc = live;
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (k < g) mc &= mc - 1;
    const int c = __ffs(mc) - 1;           // the g-th live corner (-1: none)
    const int x = (c & 1) ? px2 : px, y = (c & 2) ? py2 : py, z = (c & 4) ? pz2 : pz;
    int ex = min(ME.L - x, ME.Mw), ey = min(ME.W - y, ME.Md), ez = min(ME.H - z, ME.Mh);
    const int j0 = top_start(zt, bx, nb, pz + 1) + (lane & (step - 1));
    bool beyond = false;   // some box reaches past the corner on every axis and ends no extent
#pragma unroll 1
    for (int j = j0; j < nb; j += step) {
        const uint4 v = bx[j];
        if ((int)(v.x >> 16) > x && (int)(v.y >> 16) > y && (int)(v.z >> 16) > z) {
            const int dx = (int)(v.x & 0xffffu) - x, dy = (int)(v.y & 0xffffu) - y, dz = (int)(v.z & 0xffffu) - z;
            const bool ix = dx < ME.w, iy = dy < ME.d, iz = dz < ME.h;
            if (iy && iz) ex = min(ex, dx);
            if (ix && iz) ey = min(ey, dy);
            if (ix && iy) ez = min(ez, dz);
            beyond = beyond || (dx < ex && dy < ey && dz < ez);
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int d = 1; d < step; d <<= 1) {
        ex = min(ex, __shfl_xor_sync(FULL, ex, d));
        ey = min(ey, __shfl_xor_sync(FULL, ey, d));
        ez = min(ez, __shfl_xor_sync(FULL, ez, d));
    }
    // whether a box meets the extents' cuboid: the final extents only shrank,
    // so only a lane that met one before needs to look again
    bool meets = false;
    if (beyond) {
#pragma unroll 1
        for (int j = j0; j < nb; j += step) {
            const uint4 v = bx[j];
            meets = meets || ((int)(v.x >> 16) > x && (int)(v.y >> 16) > y && (int)(v.z >> 16) > z &&
                              (int)(v.x & 0xffffu) < x + ex && (int)(v.y & 0xffffu) < y + ey &&
                              (int)(v.z & 0xffffu) < z + ez);
        }
    }
    const unsigned hit = __ballot_sync(FULL, meets);
    if (g < nl && (lane & (step - 1)) == 0) {
        // the g-th live corner takes the g-th freed slot, or one past the end
        const int slot = g < nf ? (int)free_slots[g] : nc0 + g - nf;
        const unsigned group = (step == 32 ? 0xffffffffu : (1u << step) - 1u) << lane;
        K[slot] = ((uint32_t)z << xyb) | ((uint32_t)y << xb) | (uint32_t)x;
        K[cap + slot] = (uint32_t)ex | ((uint32_t)ey << 16);
        K[2 * cap + slot] = (uint32_t)ez | (hit & group ? PT_MARKED : 0u);
    }
    __syncwarp();
    return ERR_NONE;
}

}  // namespace plpb
