// block.cu -- the block-building engine (blockproof/plp_block.cpp) as a
// persistent kernel: one warp per restart, every restart of every instance in
// one launch, like the extreme-point decoder.
//
// Reference semantics:
//   catalogue, shape precedence   blockproof/plp_block.cpp:29-47,237-262
//   block pass (plan, placement)  blockproof/plp_block.cpp:95-223
//   contact pick rules            blockproof/plp_block.cpp:55-84,188-200
//   run loop and selection        blockproof/plp_block.cpp:228-304
//   C1/C2/C3, EP update, FSR      gpu/plp_common.hpp (check_feasible_one,
//                                 sort_dedup_pt, compute_fsr)
//
// The catalogue and its orderings are computed on the host per instance (the
// shapes, each type's shapes in precedence order, the first fitting shape for
// every remaining count, the placement rank of every shape). Per sweep a warp
// builds the plan with the reference's RNG draws, sorts the plan's placement
// ranks with a bitonic sort in shared memory, and places the blocks: the live
// points whose extents let the block through are tested for support, then the
// pick (first feasible point, a uniform random one, or the best bottom/side
// contact) and the extreme-point update. A placed block is written out at once
// as its a x b x k item boxes in the reference's decomposition order; the pass
// is scored by FSR over them.
//
// Points, boxes and their update are the extreme-point decoder's (decoder.cu,
// ep_state.cuh): a point carries its free extents, every block contains the
// instance's smallest edges, so dead points are dropped; C3 is the exact integer
// form 2 s >= w d of the reference's FP64 ratio test. A shape that found no
// point is not tried again until a block is placed (it draws nothing), and
// after a placement the points before the shape's last first feasible one are
// left out, as in the decoder. Like the decoder it is bound by integer work per
// point and its dependent steps.
#include "device_common.cuh"
#include "engine.hpp"
#include "ep_state.cuh"
#include "fsr_warp.cuh"

#include <climits>

namespace plpb {

struct BlockArgs {
    const InstDesc* __restrict__ inst;
    const TypeOrs* __restrict__ types;
    const BlkShape* __restrict__ cat;
    const int* __restrict__ tab;
    const int2* __restrict__ work;
    int n_work;
    const int* n_work_dev;         // set: the work count, written by an earlier launch
    int* work_next;
    int* err_flag;
    int* abort;
    SlotHead* heads;
    unsigned long long* places;
    unsigned long long* scratch;
    int scratch_stride;            // words per decoder's row of scratch
    const uint32_t* __restrict__ mt_init;
    int P, C, N, T, Hz;   // blocks, live points, items, types (tile), top-z index
    const uint32_t* seed_tab;      // seeded MT states of seeds seed_lo .. seed_lo + seed_n - 1 (or null)
    long long seed_lo;
    int seed_n;
};

__host__ __device__ inline int pow2_at_least(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Shared memory of one decoder. The FSR of a pass's items overlays everything
// after the MT state: by then blocks, points and plan are done with.
struct BlkLayout {
    int off_box, off_pts, off_w, off_free, off_rem, off_types, off_plan, off_zt, bytes;
    int cap;                 // entries per array of the points
    int off_items, off_scr;  // FSR: PackedBoxes of the items; sort keys, then its scratch
};

__host__ __device__ inline BlkLayout blk_layout(int P, int C, int N, int T, int Hz) {
    BlkLayout l;
    const int n = N > 0 ? N : 1, t = T > 0 ? T : 1;
    int o = 624 * 4;                        // MT state
    o = (o + 15) & ~15;
    l.off_items = o;
    l.off_scr = o + 16 * n;
    int scr = 14 * n + 16;
    if (scr < 4 * pow2_at_least(n)) scr = 4 * pow2_at_least(n);
    const int fsr_end = l.off_scr + scr;
    l.off_box = o;  o += 16 * P;            // placed blocks sorted by top (PackedBoxes)
    l.cap = C + 8;
    l.off_pts = o;  o += 12 * l.cap;        // points {key, x | y extents, z extent | mark}
    l.off_w = o;    o += 8 * (C + 2);       // items of one block
    o = (o + 15) & ~15;
    l.off_free = o;   o += 64;              // slots a placement frees
    l.off_rem = o;    o += 4 * t;           // copies left per type
    l.off_types = o;  o += 4 * t;           // this sweep's type order
    l.off_plan = o;   o += 4 * pow2_at_least(n);  // plan ranks (bitonic width)
    if (o < fsr_end) o = fsr_end;
    o = (o + 15) & ~15;
    l.off_zt = o;     o += 2 * Hz;          // u16: boxes with top < z
    o = (o + 15) & ~15;
    l.bytes = o;
    return l;
}

int block_smem_bytes(int P, int C, int N, int T, int Hz) { return blk_layout(P, C, N, T, Hz).bytes; }

// Ascending bitonic sort of a[0, n) in shared memory by one warp; a holds
// room for the next power of two (padded with UINT_MAX).
static __device__ __noinline__ void warp_sort_u32(uint32_t* a, int n, int lane) {
    const int npad = pow2_at_least(n);
#pragma unroll 1
    for (int i = n + lane; i < npad; i += 32) a[i] = 0xffffffffu;
    __syncwarp();
#pragma unroll 1
    for (int k = 2; k <= npad; k <<= 1) {
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll 1
            for (int i = lane; i < npad; i += 32) {
                const int l = i ^ j;
                if (l > i) {
                    const uint32_t x = a[i], y = a[l];
                    const bool up = (i & k) == 0;
                    if ((x > y) == up) {
                        a[i] = y;
                        a[l] = x;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// Bottom support and flush side contact of a block at (x, y, z) against the
// placed boxes (blockproof/plp_block.cpp:68-84), 64-bit areas.
static __device__ __noinline__ void blk_contact(int x0, int y0, int z0, int bw, int bd, int bh, const uint4* bx,
                                            int nb, long long& bottom, long long& side) {
    const long long x = x0, y = y0, z = z0;
    long long bo = z == 0 ? (long long)bw * bd : 0, si = 0;
#pragma unroll 1
    for (int j = 0; j < nb; j++) {
        const int4 b = PackedBoxes{bx}.xy(j);
        const long long bz = PackedBoxes{bx}.bottom(j), bt = PackedBoxes{bx}.top(j);
        const long long ox = min(x + bw, (long long)b.z) - max(x, (long long)b.x);
        const long long oy = min(y + bd, (long long)b.w) - max(y, (long long)b.y);
        const long long oz = min(z + bh, bt) - max(z, bz);
        if (bt == z && ox > 0 && oy > 0) bo += ox * oy;
        if (oy > 0 && oz > 0 && (b.z == x || b.x == x + bw)) si += oy * oz;
        if (ox > 0 && oz > 0 && (b.w == y || b.y == y + bd)) si += ox * oz;
    }
    bottom = bo;
    side = si;
}

// The engine draws at five places of its loop; out of line, its code stays short.
struct MtDraw {
    unsigned long long v;
    MtPos p;
};
static __device__ __noinline__ MtDraw blk_random53(uint32_t* mt, MtPos p, int lane) {
    MtDraw d{0, p};
    d.v = mt_random53(mt, d.p, lane);
    return d;
}
static __device__ __noinline__ MtDraw blk_randrange(uint32_t* mt, MtPos p, int lane, int n) {
    MtDraw d{0, p};
    d.v = (unsigned long long)(long long)mt_randrange(mt, d.p, lane, n);
    return d;
}

__device__ __forceinline__ void block_body(const BlockArgs& a, unsigned char* base, int gdec) {
    const int lane = threadIdx.x & 31;
    const BlkLayout lay = blk_layout(a.P, a.C, a.N, a.T, a.Hz);
    uint32_t* mt = reinterpret_cast<uint32_t*>(base);
    uint4* bx = reinterpret_cast<uint4*>(base + lay.off_box);
    uint32_t* pts = reinterpret_cast<uint32_t*>(base + lay.off_pts);
    uint2* Wl = reinterpret_cast<uint2*>(base + lay.off_w);
    unsigned short* free_slots = reinterpret_cast<unsigned short*>(base + lay.off_free);
    int* rem = reinterpret_cast<int*>(base + lay.off_rem);
    int* tys = reinterpret_cast<int*>(base + lay.off_types);
    uint32_t* plan = reinterpret_cast<uint32_t*>(base + lay.off_plan);
    unsigned short* zt = a.Hz ? reinterpret_cast<unsigned short*>(base + lay.off_zt) : nullptr;

    const int n_work = a.n_work_dev ? *a.n_work_dev : a.n_work;
    const int n_dec = gridDim.x * (blockDim.x >> 5);   // decoders of the launch
    int item = -1;
#pragma unroll 1
    for (;;) {
        if (*reinterpret_cast<volatile int*>(a.abort)) return;
        if (item < 0) {   // the first item is the decoder's own number (see decoder1_body)
            item = gdec;
        } else {
            if (lane == 0) item = n_dec + atomicAdd(a.work_next, 1);
            item = __shfl_sync(FULL, item, 0);
        }
        if (item >= n_work) break;
        const int2 wk = a.work[item];
        const InstDesc I = a.inst[wk.x];
        const int restart = wk.y;
        const int slot = I.slot_base + restart;
        const int L = I.L, W = I.W, H = I.H;
        const uint32_t xmask = (1u << I.xb) - 1u, ymask = (1u << I.yb) - 1u;
        const int xb = I.xb, xyb = I.xb + I.yb;
        const bool randomized = I.eps > 0.0;
        const int* tab = a.tab;
        const BlkShape* cat = a.cat + I.cat_off;
        const TypeOrs* tors = a.types + I.type_off;
        unsigned long long* best_out = a.places + I.place_off + (long long)restart * I.place_stride;
        unsigned long long* pass_out =
            I.passes > 1 ? a.scratch + (long long)gdec * a.scratch_stride : best_out;
        MtPos mpos{MT_WORDS, 0u};
        const unsigned long long random_from = mt_threshold(1.0 - I.eps);
        auto draw53 = [&] {
            const MtDraw d = blk_random53(mt, mpos, lane);
            mpos = d.p;
            return d.v;
        };
        auto draw_below = [&](int n) {
            const MtDraw d = blk_randrange(mt, mpos, lane, n);
            mpos = d.p;
            return (int)d.v;
        };
        if (randomized) {   // else no draw is ever made
            const long long sd = I.seed + restart;
            if (a.seed_tab && sd >= a.seed_lo && sd - a.seed_lo < a.seed_n) {
                const uint4* src = reinterpret_cast<const uint4*>(a.seed_tab + (sd - a.seed_lo) * 624);
                uint4* dst = reinterpret_cast<uint4*>(mt);
#pragma unroll 1
                for (int i = lane; i < 156; i += 32) dst[i] = __ldg(src + i);
                __syncwarp();
            } else {
                mt_seed_warp(mt, (unsigned long long)(sd < 0 ? -sd : sd), a.mt_init, lane);
            }
        }
        const long long t0 = global_ns();
        int npass = 0;
        int err = ERR_NONE;
        bool have_acc = false, have_any = false;
        long long best_vol = 0;
        int best_n = 0;
        double best_score = 0.0;

#pragma unroll 1
        for (int pass = 0; pass < I.passes && err == ERR_NONE; pass++) {
            int nb = 0, nc = 1, n_items = 0;
            long long vol = 0;
            if (zt)
#pragma unroll 1
                for (int i = lane; i < a.Hz; i += 32) zt[i] = 0;
#pragma unroll 1
            for (int t = lane; t < I.n_types; t += 32) rem[t] = tab[I.bo_qty + t];
            if (lane == 0) {
                pts[0] = 0u;
                pts[lay.cap] = (uint32_t)min(L, I.xw) | ((uint32_t)min(W, I.xd) << 16);
                pts[2 * lay.cap] = (uint32_t)min(H, I.xh);
            }
            __syncwarp();
            const EdgeRange ER{I.mw, I.md, I.mh, I.xw, I.xd, I.xh, L, W, H};
            int last = -1;           // rank of the last shape tried
            bool stuck = false;      // it found no point, and nothing was placed since
            uint32_t from_key = 0;   // points at smaller keys hold no feasible place for it
#pragma unroll 1
            for (;;) {   // sweeps: plan, then placement (blockproof/plp_block.cpp:129-207)
                // types with copies left, by (volume desc, index)
                int nty = 0;
#pragma unroll 1
                for (int q0 = 0; q0 < I.n_types; q0 += 32) {
                    const int q = q0 + lane;
                    const int t = q < I.n_types ? tab[I.bo_order + q] : 0;
                    const bool ok = q < I.n_types && rem[t] > 0 && tors[t].n > 0;
                    const unsigned bal = __ballot_sync(FULL, ok);
                    if (ok) tys[nty + __popc(bal & lanemask_lt())] = t;
                    nty += __popc(bal);
                }
                __syncwarp();
                if (nty == 0) break;
                if (randomized && draw53() >= random_from) {   // shuffle the type order
#pragma unroll 1
                    for (int i = nty - 1; i > 0; i--) {
                        const int j = draw_below(i + 1);
                        if (j < 0) { err = ERR_RNG; break; }
                        if (lane == 0) {
                            const int tmp = tys[i];
                            tys[i] = tys[j];
                            tys[j] = tmp;
                        }
                        __syncwarp();
                    }
                    if (err != ERR_NONE) break;
                }
                // plan: per type, the largest fitting shapes (eps: one of the top-k)
                int nplan = 0;
#pragma unroll 1
                for (int q = 0; q < nty && err == ERR_NONE; q++) {
                    const int t = tys[q];
                    int r = rem[t];
                    const int l0 = tab[I.bo_list_off + t], ns = tab[I.bo_list_off + t + 1] - l0;
                    const int s0 = tab[I.bo_start_off + t], nst = tab[I.bo_start_off + t + 1] - s0;
#pragma unroll 1
                    while (r > 0 && ns > 0) {
                        // first shape with cnt <= r (the table covers r below the largest count)
                        const int start = r > nst ? 0 : tab[I.bo_start + s0 + r - 1];
                        if (start >= ns) break;
                        const int tk = min(I.blk_topk, ns - start);
                        int pick = 0;
                        if (randomized && draw53() >= random_from) {
                            pick = draw_below(tk);
                            if (pick < 0) { err = ERR_RNG; break; }
                        }
                        const BlkShape S = cat[tab[I.bo_list + l0 + start + pick]];
                        if (lane == 0) plan[nplan] = (uint32_t)S.rank;
                        nplan++;
                        r -= S.cnt;
                    }
                }
                if (err != ERR_NONE || nplan == 0) break;
                __syncwarp();
                warp_sort_u32(plan, nplan, lane);   // placement order
                bool any = false;
#pragma unroll 1
                for (int e = 0; e < nplan && err == ERR_NONE; e++) {
                    const int rank = (int)plan[e];
                    const bool again = rank == last;
                    if (again && stuck) continue;
                    const BlkShape S = cat[tab[I.bo_shape_of_rank + rank]];
                    if (rem[S.ti] < S.cnt) continue;   // planned before, stale
                    last = rank;
                    if (!again) from_key = 0;
                    // items {key, marked << 7}: the points whose extents let the block through
                    int nW = 0;
#pragma unroll 1
                    for (int cb = 0; cb < nc; cb += 32) {
                        const int i = cb + lane;
                        bool ok = false;
                        uint32_t key = 0, mark = 0;
                        if (i < nc) {
                            key = pts[i];
                            const uint32_t exy = pts[lay.cap + i], ezm = pts[2 * lay.cap + i];
                            ok = S.bw <= (int)(exy & 0xffffu) && S.bd <= (int)(exy >> 16) &&
                                 S.bh <= (int)(ezm & 0xffffu) && key >= from_key;
                            mark = (ezm & PT_MARKED) >> 9;
                        }
                        const unsigned bal = __ballot_sync(FULL, ok);
                        if (ok) Wl[nW + __popc(bal & lanemask_lt())] = make_uint2(key, mark);
                        nW += __popc(bal);
                    }
                    __syncwarp();
                    // feasible items: C3, then C1 of the marked ones; the first is the smallest key
                    uint32_t best_key = 0xffffffffu;
                    int count = 0;
                    const unsigned need = (unsigned)S.bw * S.bd;
#pragma unroll 1
                    for (int w0 = 0; w0 < nW; w0 += 32) {
                        const bool has = w0 + lane < nW;
                        const uint2 it = has ? Wl[w0 + lane] : make_uint2(0, 0);
                        const int x = (int)(it.x & xmask), y = (int)((it.x >> xb) & ymask), z = (int)(it.x >> xyb);
                        bool ok = has;
                        if (has && z > 0) {
                            const int je = top_start(zt, bx, nb, z + 1);
                            const int4 f = make_int4(x, y, x + S.bw, y + S.bd);
                            unsigned area = 0;   // below 2^31, like the footprint
#pragma unroll 1
                            for (int j = top_start(zt, bx, nb, z); j < je; j++)
                                area += (unsigned)contact_area(f, PackedBoxes{bx}.xy(j));
                            ok = 2u * area >= need;
                        }
                        __syncwarp();
#pragma unroll 1
                        for (unsigned bal = __ballot_sync(FULL, ok && (it.y & 0x80u)); bal; bal &= bal - 1) {
                            const int q = __ffs(bal) - 1;
                            const int qx = __shfl_sync(FULL, x, q), qy = __shfl_sync(FULL, y, q),
                                      qz = __shfl_sync(FULL, z, q);
                            bool hit = false;
#pragma unroll 1
                            for (int j = top_start(zt, bx, nb, qz + 1) + lane; j < nb; j += 32) {
                                const int4 b = PackedBoxes{bx}.xy(j);
                                hit = hit || (b.x < qx + S.bw && qx < b.z && b.y < qy + S.bd && qy < b.w &&
                                              PackedBoxes{bx}.bottom(j) < qz + S.bh);
                            }
                            __syncwarp();
                            if (__any_sync(FULL, hit) && lane == q) ok = false;
                        }
                        if (has) Wl[w0 + lane].y = ok ? 1u : 0u;
                        if (ok) best_key = min(best_key, it.x);
                        count += ok;
                    }
                    uint32_t pkey = __reduce_min_sync(FULL, best_key);
                    stuck = pkey == 0xffffffffu;
                    if (stuck) continue;   // this block stays out (for now): no draw
                    from_key = pkey;
                    __syncwarp();
                    if (randomized && draw53() >= random_from) {
                        const int idx = draw_below(__reduce_add_sync(FULL, count));
                        if (idx < 0) { err = ERR_RNG; break; }
                        // the feasible item with idx feasible ones at smaller keys
#pragma unroll 1
                        for (int w0 = 0; w0 < nW; w0 += 32) {
                            const uint2 it = w0 + lane < nW ? Wl[w0 + lane] : make_uint2(0, 0);
                            int k = idx;
#pragma unroll 4
                            for (int w = 0; w < nW; w++) {
                                const uint2 o = Wl[w];
                                if (o.x < it.x) k -= (int)o.y;
                            }
                            const unsigned hit = __ballot_sync(FULL, it.y && k == 0);
                            if (hit) {
                                pkey = __shfl_sync(FULL, it.x, __ffs(hit) - 1);
                                break;
                            }
                        }
                    } else if (I.blk_pick != 0) {
                        // best (primary, secondary) contact; the earliest point on ties
                        long long k0 = -1, k1 = -1;
                        uint32_t bk = 0xffffffffu;
#pragma unroll 1
                        for (int w = lane; w < nW; w += 32) {
                            const uint2 it = Wl[w];
                            if (it.y) {
                                long long sup, side;
                                blk_contact((int)(it.x & xmask), (int)((it.x >> xb) & ymask), (int)(it.x >> xyb), S.bw,
                                            S.bd, S.bh, bx, nb, sup, side);
                                const long long p0 = I.blk_pick == 1 ? sup : sup + side;
                                const long long p1 = I.blk_pick == 1 ? side : sup;
                                if (p0 > k0 || (p0 == k0 && (p1 > k1 || (p1 == k1 && it.x < bk)))) {
                                    k0 = p0; k1 = p1; bk = it.x;
                                }
                            }
                        }
#pragma unroll
                        for (int d = 16; d > 0; d >>= 1) {
                            const long long o0 = __shfl_xor_sync(FULL, k0, d);
                            const long long o1 = __shfl_xor_sync(FULL, k1, d);
                            const uint32_t ob = __shfl_xor_sync(FULL, bk, d);
                            if (o0 > k0 || (o0 == k0 && (o1 > k1 || (o1 == k1 && ob < bk)))) {
                                k0 = o0; k1 = o1; bk = ob;
                            }
                        }
                        pkey = bk;
                    }
                    const int px = (int)(pkey & xmask), py = (int)((pkey >> xb) & ymask), pz = (int)(pkey >> xyb);
                    if (n_items + S.cnt > I.place_stride) { err = ERR_BOX_CAP; break; }
                    // the block's item boxes, in the reference's (a, b, k) order
                    const TypeOrs& T = tors[S.ti];
                    const int iw = T.w[S.oi], id = T.d[S.oi], ih = T.h[S.oi];
#pragma unroll 1
                    for (int q = lane; q < S.cnt; q += 32) {
                        const int i = q / (S.b * S.k), j = (q / S.k) % S.b, t = q % S.k;
                        pass_out[n_items + q] = pack_place(px + i * iw, py + j * id, pz + t * ih, S.oi, S.ti);
                    }
                    n_items += S.cnt;
                    vol += (long long)S.cnt * iw * id * ih;
                    __syncwarp();
                    err = place1(pkey, S.bw, S.bd, S.bh, pts, lay.cap, free_slots, bx, zt, a.Hz, nc, nb, a.P, a.C,
                                 xmask, ymask, xb, xyb, ER, lane);
                    if (lane == 0) rem[S.ti] -= S.cnt;
                    __syncwarp();
                    any = true;
                }
                if (err != ERR_NONE || !any) break;
            }
            if (err != ERR_NONE) break;
            // FSR over the item boxes: top-sorted tables rebuilt from the pass's items
            {
                uint4* items = reinterpret_cast<uint4*>(base + lay.off_items);
                uint32_t* sk = reinterpret_cast<uint32_t*>(base + lay.off_scr);
                __syncwarp();
#pragma unroll 1
                for (int q = lane; q < n_items; q += 32) {
                    int x, y, z, oi, ty;
                    unpack_place(pass_out[q], x, y, z, oi, ty);
                    sk[q] = ((uint32_t)(z + tors[ty].h[oi]) << 16) | (uint32_t)q;
                }
                warp_sort_u32(sk, n_items, lane);
                // top-z index of the items, in place of the blocks'
                if (zt) {
#pragma unroll 1
                    for (int i = lane; i < a.Hz; i += 32) zt[i] = (unsigned short)n_items;
                    __syncwarp();
#pragma unroll 1
                    for (int p = lane; p < n_items; p += 32) {
                        // no item before p reaches the levels above the top of p - 1
                        const int t = (int)(sk[p] >> 16), t0 = p > 0 ? (int)(sk[p - 1] >> 16) : -1;
#pragma unroll 1
                        for (int h = t0 + 1; h <= t; h++) zt[h] = (unsigned short)p;
                    }
                }
#pragma unroll 1
                for (int p = lane; p < n_items; p += 32) {
                    const int q = (int)(sk[p] & 0xffffu);
                    int x, y, z, oi, ty;
                    unpack_place(pass_out[q], x, y, z, oi, ty);
                    items[p] = make_uint4((uint32_t)x | (uint32_t)(x + tors[ty].w[oi]) << 16,
                                          (uint32_t)y | (uint32_t)(y + tors[ty].d[oi]) << 16,
                                          (uint32_t)z | (uint32_t)(z + tors[ty].h[oi]) << 16, (uint32_t)q);
                }
                __syncwarp();
                const double score = fsr_score_warp(PackedBoxes{items}, n_items, I.mu,
                                                    reinterpret_cast<char*>(base + lay.off_scr), lane, nullptr, zt);
                const bool acc = !I.has_theta || score >= I.theta;
                bool take;
                if (acc) take = !have_acc || vol > best_vol || (vol == best_vol && n_items > best_n);
                else take = !have_acc && (!have_any || vol > best_vol || (vol == best_vol && n_items > best_n));
                if (take) {
                    best_vol = vol;
                    best_n = n_items;
                    best_score = score;
                    if (pass_out != best_out)
#pragma unroll 1
                        for (int i = lane; i < n_items; i += 32) best_out[i] = pass_out[i];
                }
                have_any = true;
                have_acc = have_acc || acc;
                npass = pass + 1;
                __syncwarp();
            }
            if (I.budget_ns >= 0 && __shfl_sync(FULL, global_ns() - t0, 0) >= I.budget_ns) break;
        }
        if (lane == 0) {
            if (err) atomicOr(a.err_flag, 1 << err);
            SlotHead h;
            h.n_boxes = err ? 0 : best_n;
            h.err = err;
            h.volume = err ? 0 : best_vol;
            h.score = err ? 0.0 : best_score;
            h.n_passes = npass;
            h.fallback = have_acc ? 0 : 1;
            a.heads[slot] = h;
        }
        __syncwarp();
    }
}

// One decoder per CTA is built for 14 resident ones (121 registers instead of
// 154). 512 batched instances x 64 restarts, campaign configuration, 128 blocks,
// 192 points: 2.9 ms (when the bound was chosen 3.40, with 3.68 uncapped, 3.48 for
// 16 and 3.59 for 18; 9.07 ms with every point evaluated against every box for
// every block).
template <int D, int M>
__global__ void __launch_bounds__(32 * D, D == 1 ? 14 : M) block_kernel(BlockArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int dec = threadIdx.x >> 5;
    const BlkLayout lay = blk_layout(a.P, a.C, a.N, a.T, a.Hz);
    block_body(a, smem_raw + (size_t)dec * lay.bytes, blockIdx.x * D + dec);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
#define PLP_BLOCK_CONFIGS(X) X(1, 1) X(2, 1) X(4, 1) X(8, 1)

using BlockFn = void (*)(BlockArgs);

static BlockFn block_fn(int D, int M) {
#define PLP_PICK(d, m) \
    if (D == d && M == m) return block_kernel<d, m>;
    PLP_BLOCK_CONFIGS(PLP_PICK)
#undef PLP_PICK
    return nullptr;
}

bool block_config_supported(int D, int M) { return block_fn(D, M) != nullptr; }

static int block_launch_smem(const DecodeLaunch& L) {
    return block_smem_bytes(L.P, L.C, L.N, L.T, L.Hz) * L.decoders_per_cta;
}

cudaError_t block_occupancy(int P, int C, int N, int T, int Hz, int D, int M, int* ctas_per_sm) {
    BlockFn fn = block_fn(D, M);
    if (!fn) return cudaErrorInvalidConfiguration;
    const int smem = block_smem_bytes(P, C, N, T, Hz) * D;
    return cached_occupancy(reinterpret_cast<const void*>(fn), 32 * D, smem, ctas_per_sm);
}

cudaError_t configure_block(const DecodeLaunch& L) {
    BlockFn fn = block_fn(L.decoders_per_cta, L.min_blocks);
    if (!fn) return cudaErrorInvalidConfiguration;
    return ensure_dyn_smem(reinterpret_cast<const void*>(fn), block_launch_smem(L));
}

cudaError_t enqueue_block(const DecodeLaunch& L, cudaStream_t st) {
    BlockFn fn = block_fn(L.decoders_per_cta, L.min_blocks);
    if (!fn) return cudaErrorInvalidConfiguration;
    if (!L.zeroed) {
        cudaError_t e = cudaMemsetAsync(L.work_next, 0, sizeof(int), st);
        if (e != cudaSuccess) return e;
        e = cudaMemsetAsync(L.abort, 0, sizeof(int), st);
        if (e != cudaSuccess) return e;
    }
    BlockArgs a;
    a.inst = L.inst;
    a.types = L.types;
    a.cat = L.bcat;
    a.tab = L.btab;
    a.work = L.work;
    a.n_work = L.n_work;
    a.n_work_dev = L.n_work_dev;
    a.work_next = L.work_next;
    a.err_flag = L.err_flag;
    a.abort = L.abort;
    a.heads = L.heads;
    a.places = L.places;
    a.scratch = L.scratch;
    a.scratch_stride = L.scratch_stride;
    a.mt_init = L.mt_init;
    a.P = L.P;
    a.C = L.C;
    a.N = L.N;
    a.T = L.T;
    a.Hz = L.Hz;
    a.seed_tab = L.seed_tab;
    a.seed_lo = L.seed_lo;
    a.seed_n = L.seed_n;
    fn<<<L.ctas, 32 * L.decoders_per_cta, block_launch_smem(L), st>>>(a);
    return cudaGetLastError();
}

}  // namespace plpb
