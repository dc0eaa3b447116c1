// sgm_device.cuh -- device code of the SGM stage (reference: sgm.cu:5-135, filter_cost.cu:3-70):
// the path recurrences, the opposite-path pair block, and the pixel-range combine with the
// winner-take-all.  Included by sgm.cu (the stand-alone kernels) and persist.cu (the batched
// form's persistent kernel).
#pragma once

#include <climits>

#include "pm_device.cuh"

namespace pm {
namespace {

// Path r of the reference order (L->R, R->L, T->B, B->T, then TL->BR, BR->TL, TR->BL, BL->TR);
// pair p = paths (2p, 2p+1) runs along direction pair_dir(p) = the direction of path 2p.
__host__ __device__ inline void pair_dir(int p, int& dx, int& dy) {
    dx = p == 1 ? 0 : 1;
    dy = p == 0 ? 0 : 1;
    if (p == 3) dx = -1;
}

constexpr int PF = 8;      // prefetch distance in pixel steps

struct Chain {
    int x, y, n;
};

// Blocks of NW scanlines of several path pairs in one launch: entry i covers blocks [start[i], start[i + 1]).
struct PairSet {
    int n, pair[4], start[5];
};

__host__ __device__ inline int num_chains(int dx, int dy, int W, int H) {
    return dy == 0 ? H : (dx == 0 ? W : W + H - 1);
}

// The pairs of `mask` (bit p: pair p), those with the longest scanlines first, the vertical one of a wide image
// last (at 752x480x128 FP16 this order takes 388 us, the pairs' own 407 and their reverse 440).
inline PairSet make_pair_set(unsigned mask, int W, int H, int nw) {
    PairSet s{};
    const int wide[4] = {0, 2, 3, 1}, tall[4] = {1, 2, 3, 0};
    for (int i = 0; i < 4; ++i) {
        const int p = W >= H ? wide[i] : tall[i];
        if (!((mask >> p) & 1u)) continue;
        int dx, dy;
        pair_dir(p, dx, dy);
        s.pair[s.n] = p;
        s.start[s.n + 1] = s.start[s.n] + (num_chains(dx, dy, W, H) + nw - 1) / nw;
        ++s.n;
    }
    return s;
}
// Fewer than twelve scanlines per SM: one per block, else four neighbouring ones.
inline bool few_chains(unsigned mask, int W, int H, int sms) {
    const PairSet s = make_pair_set(mask, W, H, 1);
    return s.start[s.n] < sms * 12;
}
// The pair of block bx; bx becomes the block's index within it.
__device__ __forceinline__ int pair_of_block(const PairSet& s, int& bx) {
    int pair = s.pair[0], first = 0;
#pragma unroll
    for (int i = 1; i < 4; ++i)
        if (i < s.n && bx >= s.start[i]) {
            pair = s.pair[i];
            first = s.start[i];
        }
    bx -= first;
    return pair;
}

// Start pixel of chain c: pixels whose predecessor (x-dx, y-dy) lies outside the image.
__device__ __forceinline__ Chain chain_start(int c, int dx, int dy, int W, int H) {
    int x, y;
    if (dy == 0) { x = dx > 0 ? 0 : W - 1; y = c; }
    else if (dx == 0) { x = c; y = dy > 0 ? 0 : H - 1; }
    else if (c < W) { x = c; y = dy > 0 ? 0 : H - 1; }
    else { x = dx > 0 ? 0 : W - 1; y = dy > 0 ? (c - W + 1) : (c - W); }
    const int nx = dx > 0 ? W - x : (dx < 0 ? x + 1 : INT_MAX);
    const int ny = dy > 0 ? H - y : (dy < 0 ? y + 1 : INT_MAX);
    return {x, y, nx < ny ? nx : ny};
}

__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// value of plane d (warp-uniform) from the lane that owns it
template <int PPL> __device__ __forceinline__ float plane_value(const float (&s)[PPL], int d) {
    const int j = d % PPL;
    float v = s[0];
#pragma unroll
    for (int t = 1; t < PPL; ++t) v = (j == t) ? s[t] : v;
    return __shfl_sync(kFull, v, d / PPL);
}

// This lane's entries of the plane-order table, through shared memory.  Read straight from the
// kernel parameters with a lane-dependent index they become indexed constant-cache loads, which
// serialise per distinct address and which the compiler re-issues inside the pixel loop.
template <int PPL>
__device__ __forceinline__ void lane_order(const PlaneOrder& o, int lane, uint32_t& incl, uint16_t (&rk)[PPL]) {
    __shared__ uint32_t s_incl[32];
    __shared__ uint16_t s_rank[kMaxPlanes];
    for (int i = threadIdx.x; i < kMaxPlanes; i += blockDim.x) s_rank[i] = o.rank[i];
    if (threadIdx.x < 32) s_incl[threadIdx.x] = o.incl[threadIdx.x];
    __syncthreads();
    incl = s_incl[lane];
#pragma unroll
    for (int j = 0; j < PPL; ++j) rk[j] = s_rank[lane * PPL + j];
}

// |x| < FLOAT_EPS evaluated in double, as the reference's float-against-double compares
// (filter_cost.cu:37, stereo_mapper.cpp:651): RN_float(1e-5) = 9.99999974737875e-06 lies below
// 1e-5 and the next float above it, so (double)x < 1e-5 holds exactly when x <= that float.
constexpr float kFloatEpsBelow = 9.99999974737875e-06f;
__device__ __forceinline__ bool below_eps(float x) { return x <= kFloatEpsBelow; }
__device__ __forceinline__ bool within_eps(float x) { return x <= kFloatEpsBelow && x >= -kFloatEpsBelow; }

// Winner-take-all with the reference tree's tie-break, then the three rejection rules and
// the parabola subpixel refinement (filter_cost.cu:22-52), plus the optional uniqueness test.
template <int PPL>
__device__ __forceinline__ void wta_filter(const float (&s)[PPL], uint32_t incl, const uint16_t (&rk)[PPL],
                                           int lane, int D, const FilterParams& fp, float& depth_out,
                                           int& idx_out, int& cls_out) {
    float lmin = inf_f();
#pragma unroll
    for (int j = 0; j < PPL; ++j)
        if ((incl >> j) & 1u) lmin = fminf(lmin, s[j]);
    const float mn = warp_min_f32(lmin);
    unsigned lr = 0xffffffffu;
    int lj = 0;
#pragma unroll
    for (int j = 0; j < PPL; ++j)
        if (((incl >> j) & 1u) && s[j] == mn && rk[j] < lr) { lr = rk[j]; lj = j; }
    const unsigned r = __reduce_min_sync(kFull, lr);
    const unsigned ball = __ballot_sync(kFull, lr == r);
    const int idx = __shfl_sync(kFull, lane * PPL + lj, __ffs(ball) - 1);

    float depth;
    int cls = kWtaDepth;
    if (within_eps(mn)) {
        depth = kDepInf;                                   // non-overlap (:37-38)
        cls = kWtaNoOverlap;
    } else if (idx == 0 || idx == D - 1) {
        depth = 0.0f;                                      // border plane (:39-40)
        cls = kWtaBorder;
    } else {
        const float pre = plane_value(s, idx - 1), post = plane_value(s, idx + 1);
        if (__fadd_rn(pre, post) < __fmul_rn(__fmul_rn(2.0f, mn), fp.var_scale)) {
            depth = 0.0f;                                  // flat minimum (:41-42)
            cls = kWtaFlat;
        } else {
            bool reject = false;
            if (fp.uniq > 0.0f && fp.uniq < 1.0f) {
                float l2 = inf_f();
#pragma unroll
                for (int j = 0; j < PPL; ++j) {
                    const int d = lane * PPL + j;
                    if (((incl >> j) & 1u) && (d < idx - 1 || d > idx + 1)) l2 = fminf(l2, s[j]);
                }
                const float second = warp_min_f32(l2);
                reject = mn > __fmul_rn(fp.uniq, second);
            }
            if (reject) {
                depth = 0.0f;
                cls = kWtaAmbiguous;
            } else {                                       // parabola (:45-51)
                const float a2 = __fadd_rn(__fsub_rn(pre, __fmul_rn(2.0f, mn)), post);
                const float b = __fadd_rn(-pre, post);
                const float sub = __fsub_rn((float)idx, __fdiv_rn(b, __fmul_rn(2.0f, a2)));
                depth = rcp_rn(__fmaf_rn(sub, fp.drho, fp.rho0));
            }
        }
    }
    depth_out = depth;
    idx_out = idx;
    cls_out = cls;
}

// The debug winner-take-all of outputFusionCPU's CASE 0 and CASE 1 (stereo_mapper.cpp:636-660,
// 680-704): planes scanned in order from a minimum of 100000, the first strictly smaller value
// wins (so ties go to the lower plane); |min| < FLOAT_EPS gives 10000, the first and last plane
// give 0, otherwise the depth of the plane itself, 1 / (rho0 + d * drho), without subpixel
// refinement.  When no plane is below 100000 the reference leaves its index unset; plane 0 (and
// so 0) is reported here.
template <int PPL>
__device__ __forceinline__ void case_argmin(const float (&s)[PPL], int lane, int D, const FilterParams& fp,
                                            float& out, int& idx_out) {
    float m = 100000.0f;
    unsigned mi = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < PPL; ++j)
        if (s[j] < m) { m = s[j]; mi = (unsigned)(lane * PPL + j); }
    const float mn = warp_min_f32(m);
    const unsigned r = __reduce_min_sync(kFull, m == mn ? mi : 0xffffffffu);
    const int idx = r < (unsigned)D ? (int)r : 0;
    float v;
    if (below_eps(mn)) v = kCaseInf;
    else if (idx == 0 || idx == D - 1) v = 0.0f;
    else v = rcp_rn(__fmaf_rn((float)idx, fp.drho, fp.rho0));
    out = v;
    idx_out = idx;
}

template <bool HALF> struct CostElem;
template <> struct CostElem<false> { using T = float; };
template <> struct CostElem<true> { using T = __half; };

// Ring stage of a warp: for each of its two chains the 32 lanes' cost slices of one step.
template <int PPL, bool HALF> struct Ring {
    static constexpr int CB = PPL * (int)sizeof(typename CostElem<HALF>::T);
    static constexpr int CHAIN_B = 32 * CB;
    static constexpr int STAGE_B = 2 * CHAIN_B;
};

template <int PPL, bool HALF, bool CG = false>
__device__ __forceinline__ void load_slice(float (&cv)[PPL], const unsigned char* p) {
    if constexpr (HALF) {
        const __half2* hp = reinterpret_cast<const __half2*>(p);
#pragma unroll
        for (int j = 0; j < PPL / 2; ++j) {
            const float2 v = __half22float2(CG ? __ldcg(hp + j) : hp[j]);
            cv[2 * j] = v.x;
            cv[2 * j + 1] = v.y;
        }
    } else {
        load_planes<PPL, CG>(cv, reinterpret_cast<const float*>(p));
    }
}

// Adds v to p[0..PPL) in global memory with vector float reductions (no result returned).
template <int PPL> __device__ __forceinline__ void red_planes(float* p, const float (&v)[PPL]) {
    if constexpr (PPL % 4 == 0) {
#pragma unroll
        for (int j = 0; j < PPL; j += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + j), "f"(v[j]), "f"(v[j + 1]),
                         "f"(v[j + 2]), "f"(v[j + 3])
                         : "memory");
    } else if constexpr (PPL % 2 == 0) {
#pragma unroll
        for (int j = 0; j < PPL; j += 2)
            asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p + j), "f"(v[j]), "f"(v[j + 1]) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < PPL; ++j) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p + j), "f"(v[j]) : "memory");
    }
}

// The FP16 form's pair volumes: the lane's planes rounded to FP16 (round to nearest) and stored,
// or added to what is stored with packed FP16 reductions (the sum rounded to FP16, no flush).
template <int PPL> __device__ __forceinline__ void pack_h(uint32_t (&w)[PPL / 2], const float (&v)[PPL]) {
    static_assert(PPL % 2 == 0, "FP16 pair volumes need an even number of planes per lane");
#pragma unroll
    for (int j = 0; j < PPL / 2; ++j) {
        const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
        w[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
}
template <int PPL> __device__ __forceinline__ void store_planes_h(__half* p, const float (&v)[PPL]) {
    uint32_t w[PPL / 2];
    pack_h<PPL>(w, v);
    if constexpr (PPL == 8) {
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if constexpr (PPL == 4) {
        *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
        for (int j = 0; j < PPL / 2; ++j) reinterpret_cast<uint32_t*>(p)[j] = w[j];
    }
}
template <int PPL> __device__ __forceinline__ void red_planes_h(__half* p, const float (&v)[PPL]) {
    uint32_t w[PPL / 2];
    pack_h<PPL>(w, v);
    if constexpr (PPL == 8) {
        asm volatile("red.global.add.noftz.v4.f16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(w[0]), "r"(w[1]),
                     "r"(w[2]), "r"(w[3])
                     : "memory");
    } else if constexpr (PPL == 4) {
        asm volatile("red.global.add.noftz.v2.f16x2 [%0], {%1, %2};" ::"l"(p), "r"(w[0]), "r"(w[1]) : "memory");
    } else {
#pragma unroll
        for (int j = 0; j < PPL / 2; ++j)
            asm volatile("red.global.add.noftz.f16x2 [%0], %1;" ::"l"(p + 2 * j), "r"(w[j]) : "memory");
    }
}
// The meeting pixel of an odd chain in an FP16 pair volume: both paths' values rounded to FP16
// and added in FP16, as the reduction does for the other pixels.
template <int PPL> __device__ __forceinline__ void add_h(float (&o)[PPL], const float (&a)[PPL], const float (&b)[PPL]) {
#pragma unroll
    for (int j = 0; j < PPL; ++j) o[j] = __half2float(__hadd(__float2half_rn(a[j]), __float2half_rn(b[j])));
}

// Recurrence state of one path along one scanline, and the adaptive-penalty flags of the 32
// steps of the current batch (bit i: step k0 + i has a reference-image gradient below tau).
template <int PPL> struct PathState {
    float L[PPL];
    float below, above;   // the neighbour lanes' planes next to this lane's first and last (+inf at the ends)
    float mprev;
    unsigned qmask;
};

// a + b for the planes of a lane, two at a time on the packed FP32x2 pipe (each element rounds
// as the scalar add does).
template <int PPL>
__device__ __forceinline__ void add_planes(float (&o)[PPL], const float (&a)[PPL], const float (&b)[PPL]) {
#pragma unroll
    for (int j = 0; j + 1 < PPL; j += 2) {
        const float2 r = __fadd2_rn(make_float2(a[j], a[j + 1]), make_float2(b[j], b[j + 1]));
        o[j] = r.x;
        o[j + 1] = r.y;
    }
    if constexpr (PPL % 2) o[PPL - 1] = __fadd_rn(a[PPL - 1], b[PPL - 1]);
}
template <int PPL> __device__ __forceinline__ void add_planes(float (&o)[PPL], const float (&a)[PPL], float b) {
#pragma unroll
    for (int j = 0; j + 1 < PPL; j += 2) {
        const float2 r = __fadd2_rn(make_float2(a[j], a[j + 1]), make_float2(b, b));
        o[j] = r.x;
        o[j + 1] = r.y;
    }
    if constexpr (PPL % 2) o[PPL - 1] = __fadd_rn(a[PPL - 1], b);
}

// The planes of a lane that take part in the reduction tree of sgm.cu:24-31 (bit j: plane j), for 32 * ppl planes:
// the tree halves down to ppl classes of planes modulo ppl, which are the same for every lane, and then drops some
// of them where ppl is no power of two.  A constant of the kernel, so a dropped plane costs nothing (masks read per
// lane cost a test and a select per plane: the stage at 1280x720x192 3277 -> 3240 us, 333x251x96 148 -> 145).
constexpr unsigned tree_mask(int ppl) {
    unsigned slot[8] = {};
    for (int d = 0; d < ppl; ++d) slot[d] = 1u << d;
    for (int i = ppl >> 1; i > 0; i >>= 1)
        for (int d = 0; d < i; ++d)
            if (d + i < ppl) {
                slot[d] |= slot[d + i];
                slot[d + i] = 0;
            }
    return slot[0];
}

// Smallest of the lane's planes that take part in the minimum (all of them when FULL).
template <int PPL, bool FULL> __device__ __forceinline__ float lane_min(const float (&v)[PPL]) {
    constexpr unsigned MASK = FULL ? (1u << PPL) - 1u : tree_mask(PPL);
    static_assert(MASK & 1u, "plane 0 always takes part");
    float m = v[0], one = 0.0f;
    bool have = false;   // the odd one of two planes for a three-input minimum (all constants)
#pragma unroll
    for (int j = 1; j < PPL; ++j) {
        if (!((MASK >> j) & 1u)) continue;
        if (have) m = min3f(m, one, v[j]);
        one = v[j];
        have = !have;
    }
    return have ? fminf(m, one) : m;
}

// Whether the pixel has a plane that was never measured (cost < 0): the path treats its cost as 0
// and outputs COST_INF = 0 there (sgm.cu:33-38, 67-71, 101-104).
template <int PPL, bool FULL> __device__ __forceinline__ bool pixel_invalid(const float (&cv)[PPL]) {
    return __any_sync(kFull, lane_min<PPL, FULL>(cv) < 0.0f);
}

// A pixel's costs as the path takes them (0 on an invalid pixel); returns whether the pixel is invalid.
template <int PPL, bool FULL>
__device__ __forceinline__ bool path_costs(float (&cz)[PPL], const float (&cv)[PPL]) {
    const bool inv = pixel_invalid<PPL, FULL>(cv);
#pragma unroll
    for (int j = 0; j < PPL; ++j) cz[j] = inv ? 0.0f : cv[j];
    return inv;
}

// What the next step needs of a path's new values from the other lanes: started as soon as the values are there,
// so that their latency passes behind the other end's step, the stores and the next costs.  Up to four planes per
// lane (kAhead): with more, and with records, the registers for it cost more warps than it gives (1280x720x192 FP16
// 1764 -> 1789 us), and there the neighbour lanes' planes are fetched, and the costs read, where a step begins.
template <int PPL, bool ROUTE> constexpr bool kAhead = PPL <= 4 && !ROUTE;
template <int PPL>
__device__ __forceinline__ void path_neighbours(PathState<PPL>& s, int lane) {
    s.below = __shfl_up_sync(kFull, s.L[PPL - 1], 1);
    s.above = __shfl_down_sync(kFull, s.L[0], 1);
    if (lane == 0) s.below = inf_f();
    if (lane == 31) s.above = inf_f();
}
template <int PPL, bool FULL, bool ROUTE>
__device__ __forceinline__ void path_exchange(PathState<PPL>& s, int lane) {
    if constexpr (kAhead<PPL, ROUTE>) path_neighbours<PPL>(s, lane);
    s.mprev = warp_min_f32(lane_min<PPL, FULL>(s.L));
}

// First pixel of a path: L = C, or 0 on an invalid pixel (sgm.cu:21-43).
template <int PPL, bool FULL, bool ROUTE>
__device__ __forceinline__ void path_first(PathState<PPL>& s, const float (&cz)[PPL], int lane,
                                           float (&o)[PPL]) {
#pragma unroll
    for (int j = 0; j < PPL; ++j) s.L[j] = o[j] = cz[j];
    path_exchange<PPL, FULL, ROUTE>(s, lane);
}

// The differentiation form's record of one step: which term of the minimum each plane took, as three
// ballots per plane j of a lane (word 3j: the same plane's; 3j + 1: a neighbour's; 3j + 2: the lower
// neighbour is not above the upper one; earlier words take precedence), and the lowest plane that
// holds the predecessor's minimum (word 3 * PPL).  Plain comparisons: two bits per plane would hold
// the choice, but their encoding takes more instructions than the third ballot.
template <int PPL> struct Route {
    static constexpr int WORDS = (3 * PPL + 1 + 3) / 4 * 4;   // whole 16-byte pieces
    uint32_t w[WORDS];
};
// Where a pass with records puts them: path r's record of a pixel is record r * N + pixel; and the invalid
// flag of every pixel (written by pair 0).  8 * N < 2^32.  Path r's values go to volume
// (slots >> 4 * r) & 15 of vol: the two paths of a pair meet in one volume, as in the product, or have
// one each.
struct RouteOut {
    uint32_t* codes;
    uint8_t* invalid;
    float* vol;
    unsigned slots;
};
template <int PPL> __device__ __forceinline__ void store_route(uint32_t* p, const Route<PPL>& r) {
#pragma unroll
    for (int i = 0; i < Route<PPL>::WORDS; i += 4)
        *reinterpret_cast<uint4*>(p + i) = make_uint4(r.w[i], r.w[i + 1], r.w[i + 2], r.w[i + 3]);
}

// One pixel step of a path (sgm.cu:57-108): L(p, d) = C(p, d) + min(L(p-r, d), L(p-r, d+-1) + P1,
// min_k L(p-r, k) + P2) - min_k L(p-r, k), P1/P2 scaled by q1/q2 when the flag q says the
// reference image's path gradient is below tau; a plane never measured makes the pixel invalid:
// its cost counts as 0 (cz) and the path's output there is COST_INF = 0.  o receives the output.
// ROUTE: rt receives the step's record; equal terms resolve to the same plane, then to a neighbour (the
// lower one first), then to the minimum; and an invalid pixel's output is the path's value, as a NaN must show in the
// sum there too (the loss leaves the pixel out).
template <int PPL, bool FULL, bool ROUTE = false>
__device__ __forceinline__ void path_step(const SgmLaunch& a, PathState<PPL>& s, const float (&cz)[PPL], bool inv,
                                          bool q, float p1q, float p2q, int lane, float (&o)[PPL],
                                          Route<PPL>* rt = nullptr) {
    const float P1 = q ? p1q : a.p1, P2 = q ? p2q : a.p2;
    const float mP2 = __fadd_rn(s.mprev, P2);
    if constexpr (!kAhead<PPL, ROUTE>) path_neighbours<PPL>(s, lane);
    const float lm = s.below, lp = s.above;
    // min(L[d], minL + P2, L[d-1] + P1, L[d+1] + P1) (sgm.cu:85-92); min(a+P1, b+P1) is
    // min(a, b) + P1 exactly because rounding is monotonic
    float nb[PPL], vv[PPL];
#pragma unroll
    for (int j = 0; j < PPL; ++j) nb[j] = fminf(j == 0 ? lm : s.L[j - 1], j == PPL - 1 ? lp : s.L[j + 1]);
    add_planes<PPL>(nb, nb, P1);
#pragma unroll
    for (int j = 0; j < PPL; ++j) vv[j] = min3f(s.L[j], mP2, nb[j]);
    if constexpr (ROUTE) {
        unsigned at = ~0u;
#pragma unroll
        for (int j = PPL - 1; j >= 0; --j) {
            rt->w[3 * j] = __ballot_sync(kFull, s.L[j] == vv[j]);
            rt->w[3 * j + 1] = __ballot_sync(kFull, nb[j] == vv[j]);
            rt->w[3 * j + 2] = __ballot_sync(kFull, (j == 0 ? lm : s.L[j - 1]) <= (j == PPL - 1 ? lp : s.L[j + 1]));
            at = s.L[j] == s.mprev ? (unsigned)(lane * PPL + j) : at;
        }
        rt->w[3 * PPL] = __reduce_min_sync(kFull, at);
#pragma unroll
        for (int i = 3 * PPL + 1; i < Route<PPL>::WORDS; ++i) rt->w[i] = 0u;
    }
    add_planes<PPL>(vv, cz, vv);               // C + val
    add_planes<PPL>(s.L, vv, -s.mprev);        // - minL (:98); the negation is exact
#pragma unroll
    for (int j = 0; j < PPL; ++j) o[j] = !ROUTE && inv ? 0.0f : s.L[j];
    path_exchange<PPL, FULL, ROUTE>(s, lane);
}

// Reference intensity of step k of a chain starting at pixel p0 (0 past its end).
__device__ __forceinline__ float chain_ref(const float* __restrict__ ref, int p0, int step, int k, int n, int npix) {
    return k < n && PM_IN_BOUNDS(p0 + k * step, npix, kSitePairRef) ? __ldg(ref + (unsigned)(p0 + k * step)) : 0.0f;
}

// The flags |I(k) - I(k-1)| < tau of the 32 steps k0 .. k0+31 of one chain as a ballot (bit i:
// step k0 + i).  Lane i holds I(k0 + i) in `cur` (read one batch ahead into `nxt`, which is
// then refilled with I(k0 + 64 + i)); `last` carries I(k0 - 1).
__device__ __forceinline__ unsigned penalty_flags(float& cur, float& nxt, const float* __restrict__ ref, int p0,
                                                  int step, int k0, int n, int lane, float tau, float& last, int npix) {
    const float I = cur;
    cur = nxt;
    nxt = chain_ref(ref, p0, step, k0 + 64 + lane, n, npix);
    float prev = __shfl_up_sync(kFull, I, 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(kFull, I, 31);
    return __ballot_sync(kFull, fabsf(__fsub_rn(I, prev)) < tau);
}

// A pair of opposite paths along the same scanlines: warp c takes scanline c of direction
// (dx, dy) and walks it from both ends at once into the pair's volume part[slot / 2]: while the
// two ends have not met, each stores its pixel's path values; after they have, each adds its
// values to what the other end stored there; at the meeting pixel of an odd chain the two are
// added in registers.  The two recurrences are independent, so each warp keeps two dependency
// chains in flight.  The cost slices of both ends are streamed PF steps ahead with cp.async into
// a per-warp shared ring; the reference pixels are read 32 steps at a time (one per lane, a batch
// ahead) and turned into one ballot of penalty flags.  The loop is split at the meeting point,
// so the store and the reduction phases run without a per-step branch.  HOUT: FP16 pair volume.
// One block of NW warps: scanlines bx*NW .. bx*NW + NW-1; `ring` holds NW * PF * STAGE_B bytes.
// ROUTE: the steps' records go to *ro (paths slot and slot + 1).
template <int PPL, bool HALF, int NW, bool FULL, bool HOUT, bool ROUTE = false>
__device__ __forceinline__ void sgm_pair_block(const SgmLaunch& a, int dx, int dy, int slot, int bx,
                                               unsigned char* ring, const RouteOut* ro = nullptr) {
    using CT = typename CostElem<HALF>::T;
    using OT = typename CostElem<HOUT>::T;
    using RG = Ring<PPL, HALF>;
    constexpr int CB = RG::CB, CHAIN_B = RG::CHAIN_B, STAGE_B = RG::STAGE_B;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = a.W, H = a.H, D = a.D;
    const int c = bx * NW + warp;
    if (c >= num_chains(dx, dy, W, H)) return;        // warp-uniform; no block barriers below
    const Chain ch = chain_start(c, dx, dy, W, H);
    const int n = ch.n;
    // pixel indices (W * H < 2^31), and running addresses of the slices read and written.  ROUTE: the
    // addresses are formed from the pixels, which takes an instruction more per slice and leaves the
    // registers that the records need.
    const int step = dy * W + dx;
    const int pf0 = ch.y * W + ch.x;                    // forward start
    const int pb0 = pf0 + (n - 1) * step;               // backward start (the forward end)
    int pf = pf0, pb = pb0;                             // the current step's pixels

    unsigned char* const wbase = ring + (size_t)warp * PF * STAGE_B;
    const CT* const cost = reinterpret_cast<const CT*>(a.cost) + lane * PPL;
    OT* out = static_cast<OT*>(a.part[slot >> 1]) + lane * PPL;
    [[maybe_unused]] OT* out2 = out;   // ROUTE: the second path's volume
    if constexpr (ROUTE) {
        const size_t nv = (size_t)W * H * D;
        out = reinterpret_cast<OT*>(ro->vol) + ((ro->slots >> (4 * slot)) & 15u) * nv + lane * PPL;
        out2 = reinterpret_cast<OT*>(ro->vol) + ((ro->slots >> (4 * slot + 4)) & 15u) * nv + lane * PPL;
    }
    const bool one = !ROUTE || out == out2;
    auto at = [&](int pix) { return (size_t)(unsigned)pix * (unsigned)D; };
    const long gstep = (long)step * D;
    [[maybe_unused]] const CT* const cf0 = cost + at(pf0);
    [[maybe_unused]] const CT* const cb0 = cost + at(pb0);
    OT* qf = ROUTE ? out : out + at(pf0);
    OT* qb = ROUTE ? out2 : out + at(pb0);
    const int npix = W * H;
    [[maybe_unused]] const long long nvox = (long long)npix * D;
    auto put = [&](int pix, OT* run, const float (&v)[PPL]) {   // run: the address, or ROUTE: the volume
        OT* const q = ROUTE ? run + at(pix) : run;
        if (!PM_RANGE_IN_BOUNDS((long long)pix * D + lane * PPL, PPL, nvox, kSitePairOut)) return;
        if constexpr (HOUT) store_planes_h<PPL>(q, v);
        else store_planes<PPL>(q, v);
    };
    auto add = [&](int pix, OT* run, const float (&v)[PPL]) {
        OT* const q = ROUTE ? run + at(pix) : run;
        if (!PM_RANGE_IN_BOUNDS((long long)pix * D + lane * PPL, PPL, nvox, kSitePairOut)) return;
        if constexpr (HOUT) red_planes_h<PPL>(q, v);
        else red_planes<PPL>(q, v);
    };
    auto meet = [](float (&o)[PPL], const float (&b)[PPL]) {   // o = o + b at the meeting pixel
        if constexpr (HOUT) {
            add_h<PPL>(o, o, b);
        } else {
#pragma unroll
            for (int j = 0; j < PPL; ++j) o[j] = __fadd_rn(o[j], b[j]);
        }
    };

    auto issue = [&](unsigned char* sb, int k) {   // the slices of step k's two pixels
        [[maybe_unused]] const int f = pf0 + k * step, b = pb0 - k * step;
        if (PM_RANGE_IN_BOUNDS((long long)f * D + lane * PPL, PPL, nvox, kSitePairLoad))
            cp_async_bytes<CB>(sb + lane * CB, ROUTE ? cost + at(f) : cf0 + (long)k * gstep);
        if (PM_RANGE_IN_BOUNDS((long long)b * D + lane * PPL, PPL, nvox, kSitePairLoad))
            cp_async_bytes<CB>(sb + CHAIN_B + lane * CB, ROUTE ? cost + at(b) : cb0 - (long)k * gstep);
    };
#pragma unroll 1
    for (int k = 0; k < PF; ++k) {
        if (k < n) issue(wbase + k * STAGE_B, k);
        cp_async_commit();
    }

    const float p1q = __fmul_rn(a.p1, a.q1), p2q = __fmul_rn(a.p2, a.q2);
    PathState<PPL> fs, bs;
    float lastf = 0.0f, lastb = 0.0f;
    // intensities of steps lane and 32 + lane of both chains; then the flags of steps 0..31
    float If = chain_ref(a.ref, pf0, step, lane, n, npix), Ifn = chain_ref(a.ref, pf0, step, 32 + lane, n, npix);
    float Ib = chain_ref(a.ref, pb0, -step, lane, n, npix), Ibn = chain_ref(a.ref, pb0, -step, 32 + lane, n, npix);
    fs.qmask = penalty_flags(If, Ifn, a.ref, pf0, step, 0, n, lane, a.tau, lastf, npix);
    bs.qmask = penalty_flags(Ib, Ibn, a.ref, pb0, -step, 0, n, lane, a.tau, lastb, npix);

    // ROUTE: the invalid flags of the current batch of 32 steps, stored together
    [[maybe_unused]] unsigned rinv = 0;
    [[maybe_unused]] auto flush_invalid = [&](int k) {
        const int kk = (k & ~31) + lane, f = pf - (k - kk) * step;
        if (kk <= k && PM_IN_BOUNDS(f, npix, kSiteDiffRoute)) ro->invalid[f] = (uint8_t)((rinv >> lane) & 1u);
    };
    [[maybe_unused]] auto put_route = [&](int path, int pix, const Route<PPL>& r) {
        if (lane == 0 && PM_IN_BOUNDS(pix, npix, kSiteDiffRoute))
            store_route<PPL>(ro->codes + (size_t)((unsigned)path * (unsigned)npix + (unsigned)pix) * Route<PPL>::WORDS, r);
    };

    // the costs of the coming step, read and tested one step ahead (kAhead)
    constexpr bool AHEAD = kAhead<PPL, ROUTE>;
    float czf[PPL], czb[PPL];
    bool invf, invb;
    auto slices = [&](const unsigned char* sb, float (&cf)[PPL], float (&cb)[PPL]) {
        load_slice<PPL, HALF>(cf, sb + lane * CB);
        load_slice<PPL, HALF>(cb, sb + CHAIN_B + lane * CB);
    };

    // step 0: the first pixel of both paths
    cp_async_wait<PF - 2>();
    {
        float cf[PPL], cb[PPL], of[PPL], ob[PPL];
        [[maybe_unused]] float nf[PPL], nb[PPL];
        slices(wbase, cf, cb);
        if constexpr (AHEAD) slices(wbase + STAGE_B, nf, nb);   // (past a scanline of one pixel: not used)
        invf = path_costs<PPL, FULL>(czf, cf);
        path_costs<PPL, FULL>(czb, cb);
        if constexpr (ROUTE) rinv = invf ? 1u : 0u;
        path_first<PPL, FULL, ROUTE>(fs, czf, lane, of);
        path_first<PPL, FULL, ROUTE>(bs, czb, lane, ob);
        if constexpr (ROUTE) {
            if (n == 1 && slot == 0) flush_invalid(0);
        }
        if (n == 1 && one) {
            meet(of, ob);
            put(pf, qf, of);
        } else {
            put(pf, qf, of);
            put(pb, qb, ob);
        }
        if (PF < n) issue(wbase, PF);
        cp_async_commit();
        if constexpr (AHEAD) {
            invf = path_costs<PPL, FULL>(czf, nf);
            invb = path_costs<PPL, FULL>(czb, nb);
        }
    }
    static_assert(PF > 2, "the ring holds the step after next");
    int st = 1;

    // steps 1 .. n-1: the first visits (stores), the meeting pixel of an odd chain, then the
    // second visits (reductions)
    auto body = [&](int k, float (&of)[PPL], float (&ob)[PPL]) {
        pf += step;
        pb -= step;
        if constexpr (!ROUTE) {
            qf += gstep;
            qb -= gstep;
        }
        if ((k & 31) == 0) {
            fs.qmask = penalty_flags(If, Ifn, a.ref, pf0, step, k, n, lane, a.tau, lastf, npix);
            bs.qmask = penalty_flags(Ib, Ibn, a.ref, pb0, -step, k, n, lane, a.tau, lastb, npix);
        }
        cp_async_wait<AHEAD ? PF - 2 : PF - 1>();
        const int nst = st + 1 == PF ? 0 : st + 1;
        float nf[PPL], nb[PPL];
        slices(wbase + (AHEAD ? nst : st) * STAGE_B, nf, nb);
        if constexpr (!AHEAD) {
            invf = path_costs<PPL, FULL>(czf, nf);
            invb = path_costs<PPL, FULL>(czb, nb);
        }
        const int bit = k & 31;
        if constexpr (ROUTE) {
            Route<PPL> r;
            path_step<PPL, FULL, true>(a, fs, czf, invf, (fs.qmask >> bit) & 1u, p1q, p2q, lane, of, &r);
            put_route(slot, pf, r);
            if (slot == 0) {
                rinv = (bit == 0 ? 0u : rinv) | (invf ? 1u << bit : 0u);
                if (bit == 31 || k == n - 1) flush_invalid(k);
            }
            path_step<PPL, FULL, true>(a, bs, czb, invb, (bs.qmask >> bit) & 1u, p1q, p2q, lane, ob, &r);
            put_route(slot + 1, pb, r);
        } else {
            path_step<PPL, FULL>(a, fs, czf, invf, (fs.qmask >> bit) & 1u, p1q, p2q, lane, of);
            path_step<PPL, FULL>(a, bs, czb, invb, (bs.qmask >> bit) & 1u, p1q, p2q, lane, ob);
        }
        // refill this step's stage (its costs are in registers) with step k + PF
        if (k + PF < n) issue(wbase + st * STAGE_B, k + PF);
        cp_async_commit();
        if constexpr (AHEAD) {
            invf = path_costs<PPL, FULL>(czf, nf);
            invb = path_costs<PPL, FULL>(czb, nb);
        }
        st = nst;
    };
    const int half = n >> 1;   // steps k < half are first visits of both ends
#pragma unroll 1
    for (int k = 1; k < half; ++k) {
        float of[PPL], ob[PPL];
        body(k, of, ob);
        put(pf, qf, of);
        put(pb, qb, ob);
    }
    int k = half > 1 ? half : 1;
    if ((n & 1) && n > 1 && one) {   // both ends on the middle pixel (k == half)
        float of[PPL], ob[PPL];
        body(k, of, ob);
        meet(of, ob);
        put(pf, qf, of);
        ++k;
    }
#pragma unroll 1
    for (; k < n; ++k) {   // second visits: the first ones were this warp's own stores
        float of[PPL], ob[PPL];
        body(k, of, ob);
        if (one) {
            add(pf, qf, of);
            add(pb, qb, ob);
        } else {
            put(pf, qf, of);
            put(pb, qb, ob);
        }
    }
    cp_async_wait<0>();
}

// The depth of pixel (x, y) in the caller's map.
__device__ __forceinline__ void depth_out(const SgmLaunch& a, int x, int y, float depth) {
    if (PM_IN_BOUNDS(x, a.W, kSiteDepthOut) && PM_IN_BOUNDS(y, a.H, kSiteDepthOut))
        pitched(a.depth2, a.depth2_pitch, x, y) = depth;
}

// Sum of the NP pair volumes (each P_2p + P_2p+1) in the order (P0 + P1) + (P2 + P3)
// [+ ((P4 + P5) + (P6 + P7))], then the winner-take-all filter (MODE kCombineFilter), the debug
// argmin (kCombineArgmin) or only a store of the sum (kCombineStore).  One warp per pixel: the
// calling warp takes pixels first, first + nw, ... below npix; the next pixel's slices are loaded
// before the current one is reduced.  Every thread of the block calls it (the plane-order table
// goes through shared memory).  CG: read the pair volumes and offsets through L2 only (written
// earlier in the same launch by other blocks).
template <int PPL, int MODE, int NP, bool HIN, bool CG>
__device__ __forceinline__ void combine_pixels(const SgmLaunch& a, long first, long nw, long npix) {
    const int lane = threadIdx.x & 31;
    const int D = a.D;
    uint32_t incl;
    uint16_t rk[PPL];
    lane_order<PPL>(a.order, lane, incl, rk);
    // raw 32-bit words of the lane's slice of each pair volume (FP16 pairs: two planes per word);
    // the FP16 volumes are half the bytes per pixel, so PD pixels are kept in flight instead of one
    constexpr int WPP = HIN ? PPL / 2 : PPL;
    constexpr int PD = HIN ? 3 : 1;
    [[maybe_unused]] const long long nvox = (long long)a.W * a.H * D;
    auto loadw = [&](long pix, uint32_t (&w)[NP][WPP], float& off) {
        const size_t e = (size_t)pix * D + lane * PPL;
        if (!PM_RANGE_IN_BOUNDS(e, PPL, nvox, kSiteCombineLoad)) {
#pragma unroll
            for (int g = 0; g < NP; ++g)
#pragma unroll
                for (int j = 0; j < WPP; ++j) w[g][j] = 0u;
            off = 0.0f;
            return;
        }
#pragma unroll
        for (int g = 0; g < NP; ++g) {
            const uint32_t* src = HIN ? reinterpret_cast<const uint32_t*>(static_cast<const __half*>(a.part[g]) + e)
                                      : reinterpret_cast<const uint32_t*>(static_cast<const float*>(a.part[g]) + e);
            if constexpr (WPP % 4 == 0) {
#pragma unroll
                for (int j = 0; j < WPP; j += 4) {
                    const uint4 t = CG ? __ldcg(reinterpret_cast<const uint4*>(src + j)) : *reinterpret_cast<const uint4*>(src + j);
                    w[g][j] = t.x; w[g][j + 1] = t.y; w[g][j + 2] = t.z; w[g][j + 3] = t.w;
                }
            } else if constexpr (WPP % 2 == 0) {
#pragma unroll
                for (int j = 0; j < WPP; j += 2) {
                    const uint2 t = CG ? __ldcg(reinterpret_cast<const uint2*>(src + j)) : *reinterpret_cast<const uint2*>(src + j);
                    w[g][j] = t.x; w[g][j + 1] = t.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < WPP; ++j) w[g][j] = CG ? __ldcg(src + j) : src[j];
            }
        }
        off = a.offset ? (CG ? __ldcg(a.offset + pix) : __ldg(a.offset + pix)) : 0.0f;
    };
    auto unpack = [](const uint32_t (&w)[WPP], float (&v)[PPL]) {
#pragma unroll
        for (int j = 0; j < WPP; ++j) {
            if constexpr (HIN) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                v[2 * j] = f.x;
                v[2 * j + 1] = f.y;
            } else {
                v[j] = __uint_as_float(w[j]);
            }
        }
    };
    uint32_t ring[PD + 1][NP][WPP];
    float offr[PD + 1];
    // up to four planes per lane, the pixel of the warp's step t sits in ring slot t % (PD + 1) and
    // the pixel loop is unrolled by PD + 1, so that every slot index is a constant and the ring
    // rotates without register moves
    const bool contiguous = a.depth_pitch == (size_t)a.W * sizeof(float);
    auto process = [&](long pix, const uint32_t (&w)[NP][WPP], float off) {
        float cur[NP][PPL];
#pragma unroll
        for (int g = 0; g < NP; ++g) unpack(w[g], cur[g]);
        float o[PPL];   // (P0 + P1) + (P2 + P3), two planes per packed add
        if constexpr (NP == 4) {
            float s01[PPL], s23[PPL];
            add_planes<PPL>(s01, cur[0], cur[1]);
            add_planes<PPL>(s23, cur[2], cur[3]);
            add_planes<PPL>(o, s01, s23);
        } else {
            add_planes<PPL>(o, cur[0], cur[1]);
        }
        if (a.offset) {   // every path carries the FP16 volume's per-pixel shift once
            add_planes<PPL>(o, o, __fmul_rn((float)(2 * NP), off));
        }

        if (a.total && PM_RANGE_IN_BOUNDS((size_t)pix * D + lane * PPL, PPL, nvox, kSiteCombineOut))
            store_planes<PPL>(a.total + (size_t)pix * D + lane * PPL, o);
        if constexpr (MODE != kCombineStore) {
            float depth;
            int idx;
            int cls = 0;
            if constexpr (MODE == kCombineFilter) wta_filter<PPL>(o, incl, rk, lane, D, a.fp, depth, idx, cls);
            else case_argmin<PPL>(o, lane, D, a.fp, depth, idx);
            if (lane == 0 && PM_IN_BOUNDS(pix, (long long)a.W * a.H, kSiteCombineOut)) {
                float* dp = a.depth + pix;
                if (!contiguous) {   // W * H < 2^32: 32-bit division
                    const unsigned up = (unsigned)pix, uw = (unsigned)a.W;
                    const unsigned y = up / uw, x = up - y * uw;
                    dp = reinterpret_cast<float*>(reinterpret_cast<char*>(a.depth) + (size_t)y * a.depth_pitch) + x;
                }
                *dp = depth;
                if (a.depth2) {
                    const unsigned up = (unsigned)pix, uw = (unsigned)a.W, y = up / uw;
                    depth_out(a, (int)(up - y * uw), (int)y, depth);
                }
                if (a.index) a.index[pix] = idx;
                if (a.wta_class) a.wta_class[pix] = (uint8_t)cls;
            }
        }
    };
#pragma unroll
    for (int i = 0; i < PD; ++i)
        if (first + i * nw < npix) loadw(first + i * nw, ring[i], offr[i]);
    if constexpr (PPL <= 4) {
        for (long pix = first; pix < npix;) {
#pragma unroll
            for (int u = 0; u <= PD; ++u) {   // slot u holds pix; slot (u + PD) % (PD + 1) takes pix + PD * nw
                if (pix >= npix) break;
                const int ld = (u + PD) % (PD + 1);
                if (pix + PD * nw < npix) loadw(pix + PD * nw, ring[ld], offr[ld]);
                process(pix, ring[u], offr[u]);
                pix += nw;
            }
        }
    } else {   // more planes per lane: one copy of the body, the ring shifted by register moves
        for (long pix = first; pix < npix; pix += nw) {
            if (pix + PD * nw < npix) loadw(pix + PD * nw, ring[PD], offr[PD]);
            process(pix, ring[0], offr[0]);
#pragma unroll
            for (int i = 0; i < PD; ++i) {
                offr[i] = offr[i + 1];
#pragma unroll
                for (int g = 0; g < NP; ++g)
#pragma unroll
                    for (int j = 0; j < WPP; ++j) ring[i][g][j] = ring[i + 1][g][j];
            }
        }
    }
}

// ---- four pixels per warp ----------------------------------------------------------------
// The same sum and winner-take-all with eight lanes per pixel: lane g of a pixel's eight holds planes
// 32 c + 4 g .. 4 g + 3 of every 32-plane chunk c (FP16 volumes: 64 c + 8 g .. 8 g + 7), so a chunk of
// a pixel is one contiguous 128-byte run of 16-byte loads.  One warp per pixel spends about a hundred
// instructions per pixel on the reductions, the tests and the parabola, whatever the number of planes;
// here a warp spends them on four pixels.  The values of the planes beside the minimum go through
// shared memory.  Needs 16-byte aligned volumes.
constexpr int GP = 4;        // pixels per warp
constexpr int GL = 32 / GP;  // lanes per pixel

__device__ __forceinline__ float group_min(float v) {
#pragma unroll
    for (int o = 1; o < GL; o <<= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
    return v;
}
__device__ __forceinline__ unsigned group_min(unsigned v) {
#pragma unroll
    for (int o = 1; o < GL; o <<= 1) v = min(v, __shfl_xor_sync(kFull, v, o));
    return v;
}

// Shared memory of a block of NWARP warps: the planes' tie-break ranks (0xffffffff for planes that take
// no part), the plane of each rank, and the warps' sums.
template <int NCH, int NWARP> struct GroupSmem {
    static constexpr int D = 32 * NCH, PITCH = D + 4;   // 16-byte rows, the pixels' on different banks
    __align__(16) unsigned rank[D];
    uint16_t plane[D];
    __align__(16) float sums[NWARP][GP][PITCH];
};

// NP pair volumes (NP = 1: vol is the sum itself, or HIN: the FP16 cost volume, whose offset counts once).
// The calling warp takes pixel groups first, first + nw, ... below ngroups.  FULL: every plane takes part.
template <int NCH, int MODE, int NP, bool HIN, bool FULL, int NWARP>
__device__ __forceinline__ void combine_groups(const SgmLaunch& a, const void* const (&vol)[NP],
                                               GroupSmem<NCH, NWARP>& sm, long first, long nw, long ngroups) {
    constexpr int D = 32 * NCH, NV = 4 * NCH;   // planes, and planes per lane
    constexpr int VEC = HIN ? 8 : 4;            // planes per 16-byte load
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane % GL, q = lane / GL;     // lane of the pixel, pixel of the group
    for (int d = threadIdx.x; d < D; d += NWARP * 32) {
        if constexpr (MODE == kCombineArgmin) {
            sm.rank[d] = (unsigned)d;           // planes in order
            sm.plane[d] = (uint16_t)d;
        } else {
            const int ppl = D / 32;
            const bool in = (a.order.incl[d / ppl] >> (d % ppl)) & 1u;
            const unsigned r = a.order.rank[d];
            sm.rank[d] = in ? r : 0xffffffffu;
            if (in) sm.plane[r] = (uint16_t)d;
        }
    }
    __syncthreads();
    const long npix = (long)a.W * a.H;
    // plane of the lane's value j
    auto plane = [&](int j) { return (j / VEC) * (GL * VEC) + g * VEC + j % VEC; };
    float(&row)[GroupSmem<NCH, NWARP>::PITCH] = sm.sums[warp][q];
    const bool contiguous = a.depth_pitch == (size_t)a.W * sizeof(float);
    for (long grp = first; grp < ngroups; grp += nw) {
        const long pix = grp * GP + q;
        const bool live = pix < npix;
        long lp = live ? pix : npix - 1;
        if (!PM_RANGE_IN_BOUNDS(lp * D, D, (long long)npix * D, kSiteCombineLoad)) lp = 0;   // the warp stays together
        float s[NV];
        const float off = HIN ? __ldg(a.offset + lp) : 0.0f;
#pragma unroll
        for (int c = 0; c < NV; c += VEC) {
            const size_t e = (size_t)lp * D + (c / VEC) * (GL * VEC) + g * VEC;
            float v[NP][VEC];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                if constexpr (HIN) {
                    const uint4 t = __ldg(reinterpret_cast<const uint4*>(static_cast<const __half*>(vol[p]) + e));
                    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                        v[p][2 * i] = f.x;
                        v[p][2 * i + 1] = f.y;
                    }
                } else {
                    const float4 t = *reinterpret_cast<const float4*>(static_cast<const float*>(vol[p]) + e);
                    v[p][0] = t.x; v[p][1] = t.y; v[p][2] = t.z; v[p][3] = t.w;
                }
            }
            float o[VEC];
            if constexpr (NP == 4) {
                float s01[VEC], s23[VEC];
                add_planes<VEC>(s01, v[0], v[1]);
                add_planes<VEC>(s23, v[2], v[3]);
                add_planes<VEC>(o, s01, s23);
            } else if constexpr (NP == 2) {
                add_planes<VEC>(o, v[0], v[1]);
            } else {
#pragma unroll
                for (int i = 0; i < VEC; ++i) o[i] = v[0][i];
            }
            if constexpr (HIN) add_planes<VEC>(o, o, NP == 1 ? off : __fmul_rn((float)(2 * NP), off));
#pragma unroll
            for (int i = 0; i < VEC; ++i) s[c + i] = o[i];
        }
        if (a.total && live)
#pragma unroll
            for (int c = 0; c < NV; c += 4)
                if (PM_RANGE_IN_BOUNDS(pix * D + plane(c), 4, (long long)npix * D, kSiteCombineSum))
                    *reinterpret_cast<float4*>(a.total + (size_t)pix * D + plane(c)) = make_float4(s[c], s[c + 1], s[c + 2], s[c + 3]);

        float depth;
        int idx, cls = kWtaDepth;
        // minimum over the planes that take part, then the lowest rank among its holders
        float m = inf_f();
#pragma unroll
        for (int c = 0; c < NV; c += 4) {
            const uint4 r = FULL || MODE == kCombineArgmin ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4*>(sm.rank + plane(c));
            const unsigned rk[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) m = FULL || MODE == kCombineArgmin || rk[i] != 0xffffffffu ? fminf(m, s[c + i]) : m;
        }
        if constexpr (MODE == kCombineArgmin) m = fminf(m, 100000.0f);
        const float mn = group_min(m);
        unsigned best = 0xffffffffu;
#pragma unroll
        for (int c = 0; c < NV; c += 4) {
            const uint4 r = *reinterpret_cast<const uint4*>(sm.rank + plane(c));
            const unsigned rk[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) best = s[c + i] == mn && rk[i] < best ? rk[i] : best;
        }
        best = group_min(best);
        if constexpr (MODE == kCombineArgmin) {
            // no plane below 100000: plane 0 (a value equal to 100000 is not below it)
            idx = mn < 100000.0f && best < (unsigned)D ? (int)best : 0;
            if (below_eps(mn)) depth = kCaseInf;
            else if (idx == 0 || idx == D - 1) depth = 0.0f;
            else depth = rcp_rn(__fmaf_rn((float)idx, a.fp.drho, a.fp.rho0));
        } else {
            idx = best < (unsigned)D ? (int)sm.plane[best] : 0;
#pragma unroll
            for (int c = 0; c < NV; c += 4) *reinterpret_cast<float4*>(&row[plane(c)]) = make_float4(s[c], s[c + 1], s[c + 2], s[c + 3]);
            __syncwarp();
            const float pre = row[idx > 0 ? idx - 1 : 0], post = row[idx < D - 1 ? idx + 1 : D - 1];
            float second = inf_f();
            const bool uniq = a.fp.uniq > 0.0f && a.fp.uniq < 1.0f;
            if (uniq) {   // kernel-uniform
#pragma unroll
                for (int c = 0; c < NV; c += 4) {
                    const uint4 r = FULL ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4*>(sm.rank + plane(c));
                    const unsigned rk[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool far = (unsigned)(plane(c) + i - idx + 1) > 2u;   // d < idx - 1 or d > idx + 1
                        second = far && (FULL || rk[i] != 0xffffffffu) ? fminf(second, s[c + i]) : second;
                    }
                }
                second = group_min(second);
            }
            __syncwarp();   // the row is read before the next group's sums are written
            if (within_eps(mn)) {
                depth = kDepInf;                                   // non-overlap (filter_cost.cu:37-38)
                cls = kWtaNoOverlap;
            } else if (idx == 0 || idx == D - 1) {
                depth = 0.0f;                                      // border plane (:39-40)
                cls = kWtaBorder;
            } else if (__fadd_rn(pre, post) < __fmul_rn(__fmul_rn(2.0f, mn), a.fp.var_scale)) {
                depth = 0.0f;                                      // flat minimum (:41-42)
                cls = kWtaFlat;
            } else if (uniq && mn > __fmul_rn(a.fp.uniq, second)) {
                depth = 0.0f;
                cls = kWtaAmbiguous;
            } else {                                               // parabola (:45-51)
                const float a2 = __fadd_rn(__fsub_rn(pre, __fmul_rn(2.0f, mn)), post);
                const float b = __fadd_rn(-pre, post);
                const float sub = __fsub_rn((float)idx, __fdiv_rn(b, __fmul_rn(2.0f, a2)));
                depth = rcp_rn(__fmaf_rn(sub, a.fp.drho, a.fp.rho0));
            }
        }
        if (g == 0 && live && PM_IN_BOUNDS(pix, (long long)npix, kSiteCombineOut)) {
            float* dp = a.depth + pix;
            if (!contiguous) {   // W * H < 2^32: 32-bit division
                const unsigned up = (unsigned)pix, uw = (unsigned)a.W;
                const unsigned y = up / uw, x = up - y * uw;
                dp = reinterpret_cast<float*>(reinterpret_cast<char*>(a.depth) + (size_t)y * a.depth_pitch) + x;
            }
            *dp = depth;
            if (a.depth2) {
                const unsigned up = (unsigned)pix, uw = (unsigned)a.W, y = up / uw;
                depth_out(a, (int)(up - y * uw), (int)y, depth);
            }
            if (a.index) a.index[pix] = idx;
            if (a.wta_class) a.wta_class[pix] = (uint8_t)cls;
        }
    }
}

}  // namespace
}  // namespace pm
