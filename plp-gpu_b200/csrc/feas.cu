// feas.cu -- one-step feasibility kernel (kernel a) and the C-ABI entry
// points that replace the reference's per-step backend:
//   FeasibilityBackend::check_all   gpu/plp_common.hpp:326-332
//   CudaBackend::check_all          gpu/plp_gpu.cu:443-495 (one launch per step)
//
// A CTA takes 32 candidates, one per lane, and splits the placed boxes over its
// sixteen warps: every warp walks its share of the boxes (staged in shared
// memory, read as broadcasts), and the warps' blocked sets and contact areas
// are combined at the end. bits[ci * n_ors + oi] follow the reference's
// candidate-major order.
#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "capi_internal.hpp"
#include "device_common.cuh"
#include "engine.hpp"

namespace plpb {

// C1/C2/C3 of one candidate, gpu/plp_common.hpp:297-321 (C2, then C3 with the
// FP64 ratio (double)s / (double)(w*d) < 0.5, then C1):
//  * C3 (z > 0) sums the same integer overlap areas over the boxes whose top is
//    exactly z, the only ones the reference adds;
//  * C1 counts the boxes whose top is above z: one with top <= z fails the
//    reference's `z < b.z2` term.
// Sums and unions do not depend on the order of the boxes, so they need no sort.
//
// The kernel is bound by integer compares, and at the sizes of a decode (some
// 230 points, 50 boxes) by its dependent steps. Splitting the boxes over the
// warps gives 32 candidates a CTA instead of 256, so 4096 points use 128 SMs
// instead of 16, and no list is ranked by top first. 4096 points x 6
// orientations x 512 boxes: 7.3 us a call instead of 52 (10.1 with 8 warps);
// 230 x 6 x 48: 3.7 us instead of 12.8; 20000 x 6 x 2000: 37 instead of 316.
constexpr int FEAS_WARPS = 16;
constexpr int FEAS_BLOCK = 32 * FEAS_WARPS;

__global__ void __launch_bounds__(FEAS_BLOCK) feas_kernel(
    const int* __restrict__ cand, int n_cand, const int* __restrict__ ors, int n_ors,
    const int* __restrict__ fast6, int n_fast, int L, int W, int H, unsigned char* __restrict__ bits) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long s_area[FEAS_WARPS][6][32];
    __shared__ unsigned s_alive[FEAS_WARPS][32];
    int4* bxy = reinterpret_cast<int4*>(smem_raw);              // {x, y, x2, y2}
    int2* bzz = reinterpret_cast<int2*>(smem_raw + 16 * (size_t)n_fast);   // {z, z2}
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ci = blockIdx.x * 32 + lane;
    const bool in = ci < n_cand;
    const int x = in ? cand[3 * ci] : 0, y = in ? cand[3 * ci + 1] : 0, z = in ? cand[3 * ci + 2] : 0;
    for (int i = threadIdx.x; i < n_fast; i += FEAS_BLOCK) {
        const int* b = fast6 + 6 * i;
        bxy[i] = make_int4(b[0], b[1], b[3], b[4]);
        bzz[i] = make_int2(b[2], b[5]);
    }
    __syncthreads();
    for (int o0 = 0; o0 < n_ors; o0 += 6) {
        const int no = min(6, n_ors - o0);
        int ow[6], od[6], oh[6], wmax = INT_MIN, dmax = INT_MIN, hmax = INT_MIN;
        unsigned alive = 0;
#pragma unroll
        for (int o = 0; o < 6; o++) {
            ow[o] = o < no ? ors[3 * (o0 + o)] : 0;
            od[o] = o < no ? ors[3 * (o0 + o) + 1] : 0;
            oh[o] = o < no ? ors[3 * (o0 + o) + 2] : 0;
            if (in && o < no && !(x + ow[o] > L || y + od[o] > W || z + oh[o] > H)) {
                alive |= 1u << o;   // C2
                wmax = max(wmax, x + ow[o]);
                dmax = max(dmax, y + od[o]);
                hmax = max(hmax, z + oh[o]);
            }
        }
        long long s[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 2
        for (int j = warp; j < n_fast; j += FEAS_WARPS) {
            const int4 b = bxy[j];
            const int2 bz = bzz[j];
            // near: past the point on x and y, and before the far end of some
            // orientation that is left
            if (x < b.z && y < b.w && b.x < wmax && b.y < dmax) {
                if (bz.y > z) {
                    if (bz.x < hmax) {
#pragma unroll
                        for (int o = 0; o < 6; o++)
                            if (b.x < x + ow[o] && b.y < y + od[o] && bz.x < z + oh[o]) alive &= ~(1u << o);   // C1
                    }
                } else if (bz.y == z && z > 0) {
                    const int x0 = max(x, b.x), y0 = max(y, b.y);
#pragma unroll
                    for (int o = 0; o < 6; o++) {
                        // a positive difference of two ints fits an unsigned one
                        const int x1 = min(x + ow[o], b.z), y1 = min(y + od[o], b.w);
                        if (x1 > x0 && y1 > y0)
                            s[o] += (long long)((unsigned long long)((unsigned)x1 - (unsigned)x0) *
                                                ((unsigned)y1 - (unsigned)y0));
                    }
                }
            }
        }
        s_alive[warp][lane] = alive;
#pragma unroll
        for (int o = 0; o < 6; o++) s_area[warp][o][lane] = s[o];
        __syncthreads();
        // warp o finishes orientation o for the CTA's candidates
        if (warp < no && in) {
            unsigned m = s_alive[0][lane];
            long long t = s_area[0][warp][lane];
#pragma unroll
            for (int k = 1; k < FEAS_WARPS; k++) {
                m &= s_alive[k][lane];
                t += s_area[k][warp][lane];
            }
            bool ok = (m >> warp) & 1u;
            const int* q = ors + 3 * (o0 + warp);
            if (ok && z > 0 && (double)t / (double)(q[0] * q[1]) < 0.5) ok = false;   // C3
            bits[(long long)ci * n_ors + o0 + warp] = ok ? 1 : 0;
        }
        __syncthreads();   // before the next six orientations reuse the tables
    }
}

cudaError_t launch_feas(const int* cand, int n_cand, const int* ors, int n_ors, const int* fast6,
                        int n_fast, int L, int W, int H, unsigned char* bits, cudaStream_t st) {
    if (n_cand <= 0 || n_ors <= 0) return cudaSuccess;
    const int smem = 24 * n_fast;
    cudaError_t e = smem > 20 * 1024 ? ensure_dyn_smem(reinterpret_cast<const void*>(feas_kernel), smem) : cudaSuccess;
    if (e != cudaSuccess) return e;
    feas_kernel<<<(n_cand + 31) / 32, FEAS_BLOCK, smem, st>>>(cand, n_cand, ors, n_ors, fast6, n_fast, L, W, H, bits);
    return cudaGetLastError();
}

// largest placed-box list a call takes; 24 bytes of shared memory each
constexpr int FEAS_MAX_FAST = (227 * 1024) / 48;

// ---------------------------------------------------------------------------
// per-thread context of the host-buffer entry point and the plain path
// ---------------------------------------------------------------------------
struct StepCtx {
    cudaStream_t stream = nullptr;
    int device = -1;
    char* h_stage = nullptr;   // pinned: [cand | ors | fast] in, bits out
    char* d_stage = nullptr;
    size_t cap = 0;
    ~StepCtx() {
        if (h_stage) cudaFreeHost(h_stage);
        if (d_stage) cudaFree(d_stage);
        if (stream) cudaStreamDestroy(stream);
    }
    cudaError_t ensure(size_t need) {
        cudaError_t e = cudaSuccess;
        if (!stream) {
            e = cudaGetDevice(&device);
            if (e != cudaSuccess) return e;
            e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
            if (e != cudaSuccess) return e;
        }
        if (need <= cap) return cudaSuccess;
        size_t nc = cap ? cap : 1 << 16;
        while (nc < need) nc *= 2;
        if (h_stage) cudaFreeHost(h_stage);
        if (d_stage) cudaFree(d_stage);
        h_stage = nullptr;
        d_stage = nullptr;
        cap = 0;
        e = cudaMallocHost(&h_stage, nc);
        if (e != cudaSuccess) return e;
        e = cudaMalloc(&d_stage, nc);
        if (e != cudaSuccess) return e;
        cap = nc;
        return cudaSuccess;
    }
};

static StepCtx& step_ctx() {
    thread_local StepCtx ctx;
    return ctx;
}

static size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

// Inputs up to this size are read by the kernel straight from the pinned
// staging buffer, and the bits written there: at the sizes of a decode (a few
// KB) the two copies cost more than the kernel's reads over PCIe. One decode on
// the plain path (a 10-type instance; copies, the earlier kernel and a score
// with allocations of its own against this): 2.76 -> 1.83 ms.
constexpr size_t STEP_DIRECT = 64 << 10;

// One step on the thread's stream: inputs staged, launch, bits back,
// synchronise. Returns the smallest feasible pair index (or INT_MAX) through
// first (when non-null).
static int step_check(const int32_t* cand, int n_cand, const int32_t* ors, int n_ors,
                      const int32_t* fast6, int n_fast, int L, int W, int H, uint8_t* bits_out,
                      int* first) {
    StepCtx& c = step_ctx();
    const size_t o_cand = 0;
    const size_t o_ors = align16(o_cand + 12 * (size_t)n_cand);
    const size_t o_fast = align16(o_ors + 12 * (size_t)n_ors);
    const size_t o_bits = align16(o_fast + 24 * (size_t)n_fast);
    const size_t nbits = (size_t)n_cand * n_ors;
    const size_t total = o_bits + nbits;
    cudaError_t e = c.ensure(total);
    if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all: allocation", e);
    std::memcpy(c.h_stage + o_cand, cand, 12 * (size_t)n_cand);
    std::memcpy(c.h_stage + o_ors, ors, 12 * (size_t)n_ors);
    if (n_fast) std::memcpy(c.h_stage + o_fast, fast6, 24 * (size_t)n_fast);
    const bool direct = total <= STEP_DIRECT;
    char* base = direct ? c.h_stage : c.d_stage;
    if (!direct) {
        e = cudaMemcpyAsync(c.d_stage, c.h_stage, o_bits, cudaMemcpyHostToDevice, c.stream);
        if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all: copy in", e);
    }
    e = launch_feas(reinterpret_cast<const int*>(base + o_cand), n_cand, reinterpret_cast<const int*>(base + o_ors),
                    n_ors, reinterpret_cast<const int*>(base + o_fast), n_fast, L, W, H,
                    reinterpret_cast<unsigned char*>(base + o_bits), c.stream);
    if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all: launch", e);
    if (!direct) {
        e = cudaMemcpyAsync(c.h_stage + o_bits, c.d_stage + o_bits, nbits, cudaMemcpyDeviceToHost, c.stream);
        if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all: copy out", e);
    }
    e = cudaStreamSynchronize(c.stream);
    if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all: sync", e);
    const char* bits = c.h_stage + o_bits;
    if (bits_out) std::memcpy(bits_out, bits, nbits);
    if (first) {
        const void* p = std::memchr(bits, 1, nbits);
        *first = p ? (int)(static_cast<const char*>(p) - bits) : INT_MAX;
    }
    return PLP_OK;
}

// The pass's score on the thread's stream, rows and score in the pinned
// staging buffer (no allocation, no copy of its own).
static int step_fsr(const std::vector<Placement>& p, double mu, double* score) {
    const int n = (int)p.size();
    int cap = 32;
    while (cap < n) cap += 32;
    if (fsr_smem_per_warp(cap) * 4 > 227 * 1024) return device_fsr_score(p, mu, score);
    StepCtx& c = step_ctx();
    const size_t o_rows = 64;   // [offsets | score] before the rows
    cudaError_t e = c.ensure(o_rows + 28 * (size_t)std::max(n, 1));
    if (e != cudaSuccess) return set_cuda_error("plp_run_plain: allocation", e);
    int* off = reinterpret_cast<int*>(c.h_stage);
    double* out = reinterpret_cast<double*>(c.h_stage + 16);
    off[0] = 0;
    off[1] = n;
    int* rows = reinterpret_cast<int*>(c.h_stage + o_rows);
    for (int i = 0; i < n; i++) {
        const Placement& q = p[i];
        const int r[7] = {q.type, q.x, q.y, q.z, q.w, q.d, q.h};
        std::memcpy(rows + 7 * i, r, sizeof r);
    }
    e = launch_fsr(rows, off, 1, cap, mu, out, nullptr, c.stream);
    if (e != cudaSuccess) return set_cuda_error("plp_run_plain: score launch", e);
    e = cudaStreamSynchronize(c.stream);
    if (e != cudaSuccess) return set_cuda_error("plp_run_plain: score", e);
    *score = *out;
    return PLP_OK;
}

static int check_feas_args(int n_cand, int n_ors, int n_fast, int L, int W, int H,
                           const void* cand, const void* ors, const void* fast, const void* out) {
    if (n_cand < 0 || n_ors < 0 || n_fast < 0)
        return set_error(PLP_E_INVALID, "plp_feas_check_all: negative size");
    if ((n_cand && !cand) || (n_ors && !ors) || (n_fast && !fast) || (n_cand && n_ors && !out))
        return set_error(PLP_E_INVALID, "plp_feas_check_all: null buffer");
    if (n_fast > FEAS_MAX_FAST)
        return set_error(PLP_E_CAPACITY, "plp_feas_check_all: more than " +
                                             std::to_string(FEAS_MAX_FAST) + " placed boxes");
    (void)L; (void)W; (void)H;
    return PLP_OK;
}

}  // namespace plpb

using namespace plpb;

extern "C" int plp_feas_check_all(const int32_t* cand_xyz, int32_t n_cand, const int32_t* ors_wdh,
                                  int32_t n_ors, const int32_t* fast6, int32_t n_fast, int32_t L,
                                  int32_t W, int32_t H, uint8_t* bits_out) {
    int s = check_feas_args(n_cand, n_ors, n_fast, L, W, H, cand_xyz, ors_wdh, fast6, bits_out);
    if (s != PLP_OK) return s;
    if ((long long)n_cand * n_ors == 0) return PLP_OK;
    return step_check(cand_xyz, n_cand, ors_wdh, n_ors, fast6, n_fast, L, W, H, bits_out, nullptr);
}

extern "C" int plp_feas_check_all_dev(const int32_t* d_cand_xyz, int32_t n_cand,
                                      const int32_t* d_ors_wdh, int32_t n_ors,
                                      const int32_t* d_fast6, int32_t n_fast, int32_t L, int32_t W,
                                      int32_t H, uint8_t* d_bits_out, void* stream) {
    int s = check_feas_args(n_cand, n_ors, n_fast, L, W, H, d_cand_xyz, d_ors_wdh, d_fast6,
                            d_bits_out);
    if (s != PLP_OK) return s;
    cudaError_t e = launch_feas(d_cand_xyz, n_cand, d_ors_wdh, n_ors, d_fast6, n_fast, L, W, H,
                                d_bits_out, reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return set_cuda_error("plp_feas_check_all_dev: launch", e);
    return PLP_OK;
}

namespace plpb {

// ---------------------------------------------------------------------------
// plain path: the reference's host decode loop (gpu/plp_common.hpp:404-456)
// with one feasibility launch per item step, and the device FSR per pass.
// ---------------------------------------------------------------------------
int run_plain(const Instance& inst, const plp_run_opts& o, std::vector<RunSummary>& summ,
              std::vector<std::vector<Placement>>& placements) {
    const std::vector<int> seq = item_sequence(inst, o.order);
    std::vector<std::vector<Dims>> ors;
    for (const auto& t : inst.types) ors.push_back(orientations(t));
    const bool has_theta = !std::isnan(o.theta);
    const bool randomized = !(o.first_fit || o.eps == 0.0);
    summ.assign(o.restarts, RunSummary{});
    placements.assign(o.restarts, {});
    std::vector<int32_t> cand, fast, orsf;
    std::vector<uint8_t> bits;
    for (int r = 0; r < o.restarts; r++) {
        const long long seed = o.seed + r;
        PyRng rng((uint64_t)(seed < 0 ? -seed : seed));
        const double t0 = now_seconds();
        bool have_acc = false, have_any = false;
        long long best_vol = 0;
        int best_n = 0;
        double best_score = 0;
        std::vector<Placement> best, cur;
        int k = 0;
        for (;;) {
            cur.clear();
            cand.assign({0, 0, 0});
            fast.clear();
            long long vol = 0;
            for (int t : seq) {
                const auto& ot = ors[t];
                if (ot.empty()) continue;
                orsf.clear();
                for (const auto& d : ot) orsf.insert(orsf.end(), d.begin(), d.end());
                const int nc = (int)cand.size() / 3, no = (int)ot.size();
                bits.resize((size_t)nc * no);
                int first = INT_MAX;
                int s = step_check(cand.data(), nc, orsf.data(), no, fast.data(),
                                   (int)fast.size() / 6, inst.L, inst.W, inst.H, bits.data(), &first);
                if (s != PLP_OK) return s;
                if (first == INT_MAX) continue;
                int pick = first;
                if (randomized && rng.random() >= 1.0 - o.eps) {
                    int cnt = 0;
                    for (size_t p = (size_t)first; p < bits.size(); p++) cnt += bits[p];
                    int idx = rng.randrange(cnt);
                    for (size_t p = (size_t)first; p < bits.size(); p++)
                        if (bits[p] && idx-- == 0) { pick = (int)p; break; }
                }
                const int ci = pick / no, oi = pick % no;
                const int x = cand[3 * ci], y = cand[3 * ci + 1], z = cand[3 * ci + 2];
                const int w = ot[oi][0], d = ot[oi][1], h = ot[oi][2];
                cur.push_back({t, x, y, z, w, d, h});
                vol += 1LL * w * d * h;
                fast.insert(fast.end(), {x, y, z, x + w, y + d, z + h});
                // extreme points: drop those strictly inside, add 8 corners,
                // keep sorted by (z, y, x) and unique
                std::vector<std::array<int, 3>> pts;
                pts.reserve(nc + 8);
                for (int i = 0; i < nc; i++) {
                    const int px = cand[3 * i], py = cand[3 * i + 1], pz = cand[3 * i + 2];
                    if (x < px && px < x + w && y < py && py < y + d && z < pz && pz < z + h) continue;
                    pts.push_back({pz, py, px});
                }
                for (int c = 0; c < 8; c++)
                    pts.push_back({z + ((c & 4) ? h : 0), y + ((c & 2) ? d : 0), x + ((c & 1) ? w : 0)});
                std::sort(pts.begin(), pts.end());
                pts.erase(std::unique(pts.begin(), pts.end()), pts.end());
                cand.clear();
                for (const auto& p : pts) cand.insert(cand.end(), {p[2], p[1], p[0]});
            }
            k++;
            double score = 0;
            int s = step_fsr(cur, o.mu, &score);
            if (s != PLP_OK) return s;
            const int n = (int)cur.size();
            const bool acc = !has_theta || score >= o.theta;
            bool take;
            if (acc) take = !have_acc || vol > best_vol || (vol == best_vol && n > best_n);
            else take = !have_acc && (!have_any || vol > best_vol || (vol == best_vol && n > best_n));
            if (take) {
                best_vol = vol;
                best_n = n;
                best_score = score;
                best = cur;
            }
            have_any = true;
            have_acc = have_acc || acc;
            const bool done = o.time_limit_s < 0
                                  ? k >= o.passes
                                  : now_seconds() - t0 >= o.time_limit_s || (o.passes > 0 && k >= o.passes);
            if (done) break;
        }
        RunSummary& S = summ[r];
        S.n_boxes = best_n;
        S.volume = best_vol;
        S.score = best_score;
        S.fallback = !have_acc;
        S.n_passes = k;
        S.seed = seed;
        S.time_s = now_seconds() - t0;
        placements[r] = std::move(best);
    }
    return PLP_OK;
}

}  // namespace plpb
