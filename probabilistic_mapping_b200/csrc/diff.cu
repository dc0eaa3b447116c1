// diff.cu -- the differentiation form: a differentiable depth loss over the motion-stereo path and
// its hand-written adjoint.
//
// Forward:  C = corrected 3x3 absolute-difference cost averaged over the valid sources (the cost
//           kernel of cost.cu, exact bilinear, FP32); 8 SGM paths (sgm.cu:57-108), the opposite ones
//           summed into one volume per pair; S = sum of the pairs;
//           rho_hat = sum_d softmax(-S/T)_d rho_d; loss = mean over valid pixels with rho_gt > 0 of
//           |rho_hat - rho_gt|; and the adjoint dS of the sum by the soft-argmin Jacobian.
// Backward: each path is walked in reverse along its scanlines and the adjoint is routed through the
//           minima the forward took, which it left as records: to the same plane, the nearer
//           neighbour plane (+P1) or the path minimum (+P2), and minus the path minimum's plane for
//           the subtracted minimum;
//           dC then flows through the absolute differences (their sign), into the source
//           intensities by the bilinear weights and into the 6-DoF pose of every source through
//           the spatial derivative of the bilinear sample and the projection, as the left se(3)
//           perturbation P_s -> exp([omega]) P_s + upsilon (omega first).
// One warp per scanline for the paths (lane l holds planes [l*PPL, (l+1)*PPL)); tiles of positions for the
// cost adjoint, with atomics into the intensity gradient and per-CTA reductions of the pose gradient.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "pm_stereo.h"
#include "sgm_device.cuh"

namespace pm {
namespace {

__device__ inline float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// ---- forward paths ------------------------------------------------------------------------
// The product's pair recurrences (sgm_pair_block), which also leave the records that the adjoint
// routes by: 3 to 4 bits per voxel and path, where the path states themselves would take 32.  Bound by memory like the
// product's: two reads of the costs, a store and a reduction per pair (two stores where each path has its own
// volume), 16 to 20 bytes per voxel and pair, and 1 for the records.  All eight paths at 640x480x128:
// 0.60 ms (one path after the other, each adding to the sum and storing its states: 5.0 ms).
constexpr int kPairWarps = 1;   // scanlines per block: small blocks spread an image's scanlines over the SMs

template <int PPL>
__global__ void __launch_bounds__(32 * kPairWarps, PPL <= 4 ? 23 : 1) diff_fwd_kernel(const SgmLaunch a, const RouteOut ro, const PairSet ps) {
    extern __shared__ __align__(16) unsigned char ring[];
    int bx = blockIdx.x, dx, dy;
    const int pair = pair_of_block(ps, bx);
    pair_dir(pair, dx, dy);
    sgm_pair_block<PPL, false, kPairWarps, true, false, true>(a, dx, dy, 2 * pair, bx, ring, &ro);
}

// ---- adjoint of the paths -----------------------------------------------------------------
struct AdjArgs {
    const float* gS;             // V adjoint of the sum
    const uint32_t* codes;       // records of the forward (RouteOut)
    float* vol;                  // volumes of V: the adjoint of the costs through a pair's two paths ...
    unsigned slots;              // ... goes to volume (slots >> 2 * pair) & 3
    unsigned acc;                // bit p: pair p's is added to what its volume holds
    int W, H, D;
};

// One adjoint recurrence along a scanline: lambda = gS + mu; the planes' lambda go to the
// predecessor's planes that the forward's minima took (the same, the lower or the upper one), and the
// plane of the predecessor's minimum receives the lambda that took the minimum, less all of them for
// the subtracted minimum: together the negative sum over the planes that did not take it.  A lambda that took it and
// is not finite leaves a NaN there, as in the two sums.
template <int PPL>
__device__ __forceinline__ void adjoint_step(const float (&g)[PPL], float (&mu)[PPL],
                                             const uint32_t (&w)[Route<PPL>::WORDS], int lane, float (&lam)[PPL]) {
    const unsigned bit = 1u << lane;
    add_planes<PPL>(lam, g, mu);
    float lo[PPL], hi[PPL], direct = 0.0f;   // to the lower and the upper plane
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
        const unsigned same = w[3 * j], side = w[3 * j + 1], lower = w[3 * j + 2];
        mu[j] = (same & bit) ? lam[j] : 0.0f;
        lo[j] = (~same & side & lower & bit) ? lam[j] : 0.0f;
        hi[j] = (~same & side & ~lower & bit) ? lam[j] : 0.0f;
        direct = __fmaf_rn(lam[j], ((same | side) & bit) ? 1.0f : 0.0f, direct);   // NaN where a lam is not finite
    }
    float fromU = __shfl_down_sync(kFull, lo[0], 1);        // lane + 1's first plane -> my last
    float fromL = __shfl_up_sync(kFull, hi[PPL - 1], 1);    // lane - 1's last plane -> my first
    if (lane == 31) fromU = 0.0f;
    if (lane == 0) fromL = 0.0f;
    const float rest = warp_sum(direct);
#pragma unroll
    for (int j = 0; j < PPL; ++j) {
        float v = mu[j] + (j + 1 < PPL ? lo[j + 1 < PPL ? j + 1 : j] : fromU);
        v += j > 0 ? hi[j > 0 ? j - 1 : j] : fromL;
        mu[j] = (unsigned)(lane * PPL + j) == w[3 * PPL] ? v - rest : v;
    }
}

// A pair's adjoints: path 2p's from the far end of the scanline, path 2p + 1's from its start, both
// by one warp, as sgm_pair_block walks the forward: two independent recurrences in flight, gS and the
// records streamed PF steps ahead, the first visit of a pixel stores and the second adds.  Bound by
// memory: two reads of gS, a store and a reduction, 20 bytes per voxel and pair (0.57 ms for all eight paths at
// 640x480x128, 5.5 TB/s; path by path from the stored states 6.4 ms).
template <int PPL, int NW>
__device__ __forceinline__ void adjoint_pair_block(const AdjArgs& a, int pair, int bx, unsigned char* ring) {
    constexpr int SLICE_B = 128 * PPL, REC_B = 4 * Route<PPL>::WORDS;
    constexpr int CHAIN_B = SLICE_B + REC_B, STAGE_B = 2 * CHAIN_B;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = a.W, H = a.H, D = a.D;
    int dx, dy;
    pair_dir(pair, dx, dy);
    const int c = bx * NW + warp;
    if (c >= num_chains(dx, dy, W, H)) return;   // warp-uniform; no block barriers below
    const Chain ch = chain_start(c, dx, dy, W, H);
    const int n = ch.n;
    const int step = dy * W + dx;
    const int pf0 = ch.y * W + ch.x, pb0 = pf0 + (n - 1) * step;
    const int npix = W * H;
    const long long nvox = (long long)npix * D;
    float* const out = a.vol + ((a.slots >> (2 * pair)) & 3u) * (size_t)nvox + lane * PPL;
    const bool acc = (a.acc >> pair) & 1u;
    unsigned char* const wbase = ring + (size_t)warp * PF * STAGE_B;

    // walker 0: path 2p's adjoint, pixel pb0 - k * step; walker 1: path 2p + 1's, pixel pf0 + k * step
    auto pixel = [&](int walker, int k) { return walker ? pf0 + k * step : pb0 - k * step; };
    auto record = [&](int walker, int pix) { return (unsigned)(2 * pair + walker) * (unsigned)npix + (unsigned)pix; };
    auto issue = [&](unsigned char* sb, int k) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int pix = pixel(v, k);
            if (!PM_IN_BOUNDS(pix, npix, kSiteDiffGrad)) continue;
            unsigned char* const s = sb + v * CHAIN_B;
            cp_async_bytes<4 * PPL>(s + lane * 4 * PPL, a.gS + lane * PPL + (size_t)(unsigned)pix * (unsigned)D);
            if (lane < REC_B / 16)
                cp_async_16(s + SLICE_B + 16 * lane, a.codes + (size_t)record(v, pix) * (REC_B / 4) + 4 * lane);
        }
    };
#pragma unroll 1
    for (int k = 0; k < PF; ++k) {
        if (k < n) issue(wbase + k * STAGE_B, k);
        cp_async_commit();
    }
    float mu0[PPL], mu1[PPL];
#pragma unroll
    for (int j = 0; j < PPL; ++j) mu0[j] = mu1[j] = 0.0f;
    int st = 0;

    auto body = [&](int k, float (&l0)[PPL], float (&l1)[PPL]) {
        cp_async_wait<PF - 1>();
        __syncwarp();   // the records are copied by a few lanes and read by all
        unsigned char* const sb = wbase + st * STAGE_B;
        float g[PPL];
        uint32_t w[REC_B / 4];
        auto load = [&](const unsigned char* s) {
            load_planes<PPL>(g, reinterpret_cast<const float*>(s + lane * 4 * PPL));
#pragma unroll
            for (int i = 0; i < REC_B / 16; ++i) {
                const uint4 t = *reinterpret_cast<const uint4*>(s + SLICE_B + 16 * i);
                w[4 * i] = t.x; w[4 * i + 1] = t.y; w[4 * i + 2] = t.z; w[4 * i + 3] = t.w;
            }
        };
        load(sb);
        adjoint_step<PPL>(g, mu0, w, lane, l0);
        load(sb + CHAIN_B);
        adjoint_step<PPL>(g, mu1, w, lane, l1);
        __syncwarp();   // every lane has read the stage that is refilled
        if (k + PF < n) issue(sb, k + PF);
        cp_async_commit();
        st = (st + 1 == PF) ? 0 : st + 1;
    };
    auto put = [&](int pix, const float (&v)[PPL], bool add) {
        float* const q = out + (size_t)(unsigned)pix * (unsigned)D;
        if (!PM_RANGE_IN_BOUNDS((long long)pix * D + lane * PPL, PPL, nvox, kSiteDiffGrad)) return;
        if (add) red_planes<PPL>(q, v);
        else store_planes<PPL>(q, v);
    };
    const int half = n >> 1;
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        float l0[PPL], l1[PPL];
        body(k, l0, l1);
        const int p0 = pixel(0, k), p1 = pixel(1, k);
        if (p0 == p1) {   // the middle of an odd scanline
            add_planes<PPL>(l0, l0, l1);
            put(p0, l0, acc);
        } else {
            put(p0, l0, acc || k >= half);
            put(p1, l1, acc || k >= half);
        }
    }
    cp_async_wait<0>();
}

template <int PPL>
__global__ void __launch_bounds__(32 * kPairWarps) diff_adj_kernel(const AdjArgs a, const PairSet ps) {
    extern __shared__ __align__(16) unsigned char ring[];
    int bx = blockIdx.x;
    const int pair = pair_of_block(ps, bx);
    adjoint_pair_block<PPL, kPairWarps>(a, pair, bx, ring);
}

// a = (a + b) + c over volumes of 4 * n4 floats
__global__ void __launch_bounds__(256) fold_kernel(float4* __restrict__ a, const float4* __restrict__ b,
                                                   const float4* __restrict__ c, size_t n4) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        float4 x = a[i];
        const float4 y = b[i], z = c[i];
        x.x = (x.x + y.x) + z.x;
        x.y = (x.y + y.y) + z.y;
        x.z = (x.z + y.z) + z.z;
        x.w = (x.w + y.w) + z.w;
        a[i] = x;
    }
}

// ---- soft-argmin --------------------------------------------------------------------------
struct SoftArgs {
    const float* vol;         // NV volumes, whose sum in their order is the SGM sum
    const float* rho_gt;
    const uint8_t* invalid;
    float* rho_hat;           // optional
    float* gS;                // adjoint of the sum, without the 1 / count of the loss's mean
    double* sums;             // loss sum, count, and the number of finished blocks (cleared before the launch)
    double* loss;             // their quotient, written by the last block (optional)
    int N, D;
    float rho0, drho, T;
};

// The sum of the volumes, the soft-argmin over it, the loss's terms and its adjoint, one warp per pixel.  The
// paths are added in their order, so that the loss's signs do not depend on the layout of the volumes.  Bound by
// memory: NV reads and a write per voxel (0.20 ms at 640x480x128 with 7 volumes: 6.2 TB/s).  Six blocks per SM where
// the volumes' planes leave the registers for it, and several waves of them: 268 -> 201 us against four that the
// compiler's choice let in and a grid of six per SM, 320x240x64 with 3 volumes 31.9 -> 25.1.  The loss is summed in
// double precision per warp, block and grid.
template <int PPL, int NV>
__global__ void __launch_bounds__(256, PPL <= 4 ? 6 : 1) soft_kernel(const SoftArgs a) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long nw = (long)gridDim.x * 8;
    double loss = 0.0;
    int count = 0;
    for (long p = (long)blockIdx.x * 8 + warp; p < a.N; p += nw) {
        if (!PM_IN_BOUNDS(p, a.N, kSiteDiffGrad)) continue;
        float v[NV][PPL], s[PPL];
#pragma unroll
        for (int i = 0; i < NV; ++i) load_planes<PPL>(v[i], a.vol + ((size_t)i * a.N + p) * a.D + lane * PPL);
        add_planes<PPL>(s, v[0], v[1]);
#pragma unroll
        for (int i = 2; i < NV; ++i) add_planes<PPL>(s, s, v[i]);
        float lmin = s[0];
#pragma unroll
        for (int j = 1; j < PPL; ++j) lmin = fminf(lmin, s[j]);
        const float smin = warp_min_f32(lmin);
        float w[PPL], z = 0.0f, r = 0.0f;
#pragma unroll
        for (int j = 0; j < PPL; ++j) {
            w[j] = expf(-(s[j] - smin) / a.T);
            z += w[j];
            r += w[j] * (a.rho0 + (float)(lane * PPL + j) * a.drho);
        }
        z = warp_sum(z);
        r = warp_sum(r);
        const float rh = r / z, gt = a.rho_gt[p];
        const bool in = !a.invalid[p] && gt > 0.0f;
        const float diff = rh - gt;
        if (lane == 0 && a.rho_hat) a.rho_hat[p] = in ? rh : 0.0f;
        if (in) {
            loss += (double)fabsf(diff);
            ++count;
        }
        const float g = !in ? 0.0f : diff > 0.0f ? 1.0f : (diff < 0.0f ? -1.0f : 0.0f);
        const float k = g * (-1.0f / a.T) / z;
        float o[PPL];
#pragma unroll
        for (int j = 0; j < PPL; ++j) o[j] = k * w[j] * ((a.rho0 + (float)(lane * PPL + j) * a.drho) - rh);
        store_planes<PPL>(a.gS + (size_t)p * a.D + lane * PPL, o);
    }
    __shared__ double sl[8];
    __shared__ int sc[8];
    if (lane == 0) {
        sl[warp] = loss;
        sc[warp] = count;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i) {
            loss += sl[i];
            count += sc[i];
        }
        if (count) {
            atomicAdd(a.sums, loss);
            atomicAdd(a.sums + 1, (double)count);
        }
        if (a.loss) {
            __threadfence();
            if (atomicAdd(reinterpret_cast<unsigned*>(a.sums + 2), 1u) == gridDim.x - 1) {
                __threadfence();
                const volatile double* sums = a.sums;
                *a.loss = sums[1] > 0.0 ? sums[0] / sums[1] : 0.0;
            }
        }
    }
}

constexpr int kMaxDiffSources = 4;

struct CostBwdArgs {
    const float* ref;
    const float4* quads;      // S slots: the cost kernel's source quads
    const float* gC[4];       // nv volumes whose sum is the costs' adjoint but for the 1 / count
    int nv;
    const double* count;      // pixels in the loss
    const uint8_t* invalid;
    float hom[kMaxDiffSources][12];
    float fx, fy, cx, cy;
    int W, H, D, S;
    float rho0, drho;
    float* gI;                // S x N
    double* gP;               // S x 6
};

// Adjoint of the corrected 3x3 cost.  The sample at position q, source s and plane d serves the nine
// pixels p around q, each term compares it with the same reference value ref(q), so the sign of
// ref(q) - val(q) is common to the nine and the adjoint of the sample is
//   -sign(ref(q) - val(q)) * sum over the 3x3 pixels p around q, measured by s at d, of gC(p, d) / (9 n(p, d)),
// n(p, d) the sources that measure p at d: ONE sample, one scatter into the image and one pose term per
// (q, s, d) instead of nine (and instead of the 18 more samples per (p, s, d) that a voxel's own validity
// takes).  A CTA owns 28 x R positions q and 16 planes; a warp owns a plane pair and walks the rows:
//   * lane l stands on column x0 - 2 + l.  A first pass over the R + 4 rows turns the validity of the
//     samples into one ballot per row and plane, from which "all nine samples valid" is a few
//     bit operations, and n a bit count over the sources;
//   * the tile's gC (with its ring of one pixel) sits in shared memory, read in 64-byte plane runs and
//     already divided by 9 n; the 3x3 sums are two shuffles per row and a rolling sum of three rows;
//   * a sample's lower two taps wait in registers for the next row, whose upper taps fall on the same
//     texels when the warp hardly turns the image, so that a sample costs two reductions, not four;
//   * the pose terms stay in registers over a tile's rows, then one double atomic per CTA and component.
// The samples repeat the cost kernel's operations (homography FMAs, reciprocal, exact bilinear), so that
// the signs are the forward's.  Bound by issue (about 100 instructions per sample and plane pair); with one
// thread per voxel, 27 samples per source and nine scatters it was bound by its atomics: 29.5 -> 0.81 ms at
// 640x480x128 with 3 sources, 5.14 -> 0.096 ms at 320x240x64 with 2.
constexpr int BQX = 28;                  // positions per row of a tile
constexpr int BWARPS = 8;                // plane pairs per CTA
constexpr int BPL = 2 * BWARPS;          // planes per CTA
constexpr int BSP = BPL + 2;             // pitch of a pixel's planes in shared memory

// Pending lower taps of the previous row: texel idx and its right neighbour.
struct Pending {
    unsigned idx;
    float l, r;
};

// Adds v to element idx + k of an image of npix pixels: the address p + idx, which a sample's two taps share, plus k.
__device__ __forceinline__ void red_add(float* p, unsigned idx, unsigned k, [[maybe_unused]] long long npix, float v) {
    if (v != 0.0f && PM_IN_BOUNDS((long long)idx + k, npix, kSiteDiffGrad)) atomicAdd(p + idx + k, v);
}

template <int R> __global__ void __launch_bounds__(32 * BWARPS) cost_bwd_kernel(const CostBwdArgs A) {
    constexpr int PX = BQX + 2, PY = R + 2;   // pixels p of the tile
    __shared__ __align__(16) float hs[PX * PY * BSP];
    __shared__ float refs[R * 32];
    __shared__ unsigned ok1[BWARPS][R + 4][2];                      // validity of the samples, one source
    __shared__ unsigned ok9[BWARPS][kMaxDiffSources][PY][2];        // all nine samples of a pixel valid
    __shared__ float ps[BWARPS][6 * kMaxDiffSources];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = A.W, H = A.H, D = A.D;
    const int x0 = blockIdx.x * BQX - 1, y0 = blockIdx.z * R - 1, d0 = blockIdx.y * BPL;   // first position q
    const int x = x0 - 2 + lane;

    for (int e = tid; e < PX * PY * (BPL / 4); e += 32 * BWARPS) {
        const int p = e >> 2, k = (e & 3) * 4;
        const int py = p / PX, px = p - py * PX;
        const int gx = x0 - 1 + px, gy = y0 - 1 + py;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (gx >= 0 && gy >= 0 && gx < W && gy < H) {
            const size_t pix = (size_t)gy * W + gx;
            if (!A.invalid[pix] && PM_RANGE_IN_BOUNDS(pix * D + d0 + k, 4, (long long)W * H * D, kSiteDiffGrad))
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= A.nv) break;
                    const float4 t = *reinterpret_cast<const float4*>(A.gC[i] + pix * D + d0 + k);
                    v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
                }
        }
        *reinterpret_cast<float2*>(hs + p * BSP + k) = make_float2(v.x, v.y);
        *reinterpret_cast<float2*>(hs + p * BSP + k + 2) = make_float2(v.z, v.w);
    }
    for (int e = tid; e < R * 32; e += 32 * BWARPS) {
        const int gx = x0 - 2 + (e & 31), gy = y0 + (e >> 5);
        refs[e] = gx >= 0 && gy >= 0 && gx < W && gy < H ? A.ref[(size_t)gy * W + gx] : 0.0f;
    }

    const int da = d0 + 2 * warp;
    const float2 rho = make_float2(__fmaf_rn((float)da, A.drho, A.rho0), __fmaf_rn((float)(da + 1), A.drho, A.rho0));
    const float fxl = (float)x;
    const unsigned Wb = __float_as_uint((float)(W - 1)), Hb = __float_as_uint((float)(H - 1));
    // warp of (x, y) at the plane pair: denominator, its reciprocal and the coordinates
    auto warp_pos = [&](const float* h, int y, float2& w, float2& r, float2& u, float2& v) {
        const float fy = (float)y;
        const float hx = __fmaf_rn(h[0], fxl, __fmaf_rn(h[1], fy, h[2]));
        const float hy = __fmaf_rn(h[3], fxl, __fmaf_rn(h[4], fy, h[5]));
        const float hz = __fmaf_rn(h[6], fxl, __fmaf_rn(h[7], fy, h[8]));
        w = __ffma2_rn(make_float2(h[11], h[11]), rho, make_float2(hz, hz));
        r = rcp_warp2(w);
        u = __fmul2_rn(__ffma2_rn(make_float2(h[9], h[9]), rho, make_float2(hx, hx)), r);
        v = __fmul2_rn(__ffma2_rn(make_float2(h[10], h[10]), rho, make_float2(hy, hy)), r);
    };

    for (int s = 0; s < A.S; ++s) {
        for (int r = 0; r < R + 4; ++r) {
            float2 w, rc, u, v;
            warp_pos(A.hom[s], y0 - 2 + r, w, rc, u, v);
            // + 0 turns -0 into +0; negative values and NaN have bit patterns above the bound's
            const float2 z = make_float2(0.0f, 0.0f);
            u = __fadd2_rn(u, z);
            v = __fadd2_rn(v, z);
            const unsigned b0 = __ballot_sync(kFull, w.x >= 0.0f && __float_as_uint(u.x) <= Wb && __float_as_uint(v.x) <= Hb);
            const unsigned b1 = __ballot_sync(kFull, w.y >= 0.0f && __float_as_uint(u.y) <= Wb && __float_as_uint(v.y) <= Hb);
            if (lane == 0) {
                ok1[warp][r][0] = b0;
                ok1[warp][r][1] = b1;
            }
        }
        __syncwarp();
        if (lane < PY)
            for (int j = 0; j < 2; ++j) {
                const unsigned m = ok1[warp][lane][j] & ok1[warp][lane + 1][j] & ok1[warp][lane + 2][j];
                ok9[warp][s][lane][j] = m & (m << 1) & (m >> 1);
            }
        __syncwarp();
    }
    __syncthreads();   // the tile's gC is staged

    // gC / (9 n) and the 1 / count of the loss's mean, in place (a warp's own planes)
    const float scale = A.count[0] > 0.0 ? 1.0f / (float)A.count[0] : 0.0f;
    float inv[kMaxDiffSources + 1];
    inv[0] = 0.0f;
#pragma unroll
    for (int n = 1; n <= kMaxDiffSources; ++n) inv[n] = scale / (9.0f * (float)n);
    const bool in_p = lane >= 1 && lane <= PX;
    float2* const hp = reinterpret_cast<float2*>(hs + (in_p ? lane - 1 : 0) * BSP + 2 * warp);
    constexpr int HROW = PX * BSP / 2;   // float2 per row of pixels
    if (in_p)
        for (int r = 0; r < PY; ++r) {
            int n0 = 0, n1 = 0;
            for (int s = 0; s < A.S; ++s) {
                n0 += (ok9[warp][s][r][0] >> lane) & 1u;
                n1 += (ok9[warp][s][r][1] >> lane) & 1u;
            }
            float i0 = 0.0f, i1 = 0.0f;
#pragma unroll
            for (int n = 1; n <= kMaxDiffSources; ++n) {
                i0 = n0 == n ? inv[n] : i0;
                i1 = n1 == n ? inv[n] : i1;
            }
            const float2 g = hp[r * HROW];
            hp[r * HROW] = make_float2(__fmul_rn(g.x, i0), __fmul_rn(g.y, i1));
        }
    __syncwarp();

    const bool in_q = lane >= 2 && lane < 2 + BQX;
    const float fW1 = (float)(W - 1), fH1 = (float)(H - 1);
    const float rfx = 1.0f / A.fx, rfy = 1.0f / A.fy;
    for (int s = 0; s < A.S; ++s) {
        const float4* const quads = A.quads + s * quad_stride((size_t)W * H);
        float* const gi = A.gI + (size_t)s * W * H;
        float gp[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        Pending pend[2] = {{0u, 0.0f, 0.0f}, {0u, 0.0f, 0.0f}};
        const long long npix = (long long)W * H;
        auto flush = [&](const Pending& q) {
            red_add(gi, q.idx, 0, npix, q.l);
            red_add(gi, q.idx, 1, npix, q.r);
        };
        float2 ha = make_float2(0.0f, 0.0f), hb = ha;   // row sums of the two rows above
        for (int r = 0; r < PY; ++r) {
            float2 g = make_float2(0.0f, 0.0f);
            if (in_p) {
                const float2 t = hp[r * HROW];
                g.x = (ok9[warp][s][r][0] >> lane) & 1u ? t.x : 0.0f;
                g.y = (ok9[warp][s][r][1] >> lane) & 1u ? t.y : 0.0f;
            }
            const float2 gl = make_float2(__shfl_up_sync(kFull, g.x, 1), __shfl_up_sync(kFull, g.y, 1));
            const float2 gr = make_float2(__shfl_down_sync(kFull, g.x, 1), __shfl_down_sync(kFull, g.y, 1));
            const float2 hc = __fadd2_rn(__fadd2_rn(gl, g), gr);
            float2 B = __fadd2_rn(__fadd2_rn(ha, hb), hc);
            ha = hb;
            hb = hc;
            if (r < 2) continue;
            if (!in_q) B = make_float2(0.0f, 0.0f);
            if (!__any_sync(kFull, B.x != 0.0f || B.y != 0.0f)) continue;
            float2 w, rc, u, v;
            warp_pos(A.hom[s], y0 + r - 2, w, rc, u, v);
            const float ref = refs[(r - 2) * 32 + lane];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float bj = j ? B.y : B.x;
                if (bj == 0.0f) continue;   // then some pixel around q is measured, and q's sample is valid
                const float uj = j ? u.y : u.x, vj = j ? v.y : v.x, rj = j ? rc.y : rc.x;
                float fu, fv;
                int iu, iv;
                floor_split(uj, fu, iu);
                floor_split(vj, fv, iv);
                const float a = __fsub_rn(uj, fu), b = __fsub_rn(vj, fv);
                const unsigned idx = (unsigned)iv * (unsigned)W + (unsigned)iu;
                if (!PM_IN_BOUNDS(idx, (long long)W * H, kSiteDiffGrad)) continue;
                const float4 t = __ldg(quads + idx);   // I(x,y), I(x,y+1), I(x+1,y), I(x+1,y+1)
                const float dx0 = __fsub_rn(t.z, t.x), dx1 = __fsub_rn(t.w, t.y);
                const float top = __fmaf_rn(a, dx0, t.x), bot = __fmaf_rn(a, dx1, t.y);
                const float diff = __fsub_rn(ref, __fmaf_rn(b, __fsub_rn(bot, top), top));
                const float c = diff > 0.0f ? -bj : diff < 0.0f ? bj : 0.0f * bj;   // sign 0: a NaN or infinite adjoint stays
                if (c == 0.0f) continue;
                const float a1 = 1.0f - a, b1 = 1.0f - b;
                // taps; the image's last column has no right ones and its last row no lower ones (a or b is 0 there,
                // but their product with an infinite or NaN adjoint is not)
                const bool right = uj < fW1, lower = vj < fH1;
                const float ct = c * b1, cb = lower ? c * b : 0.0f;
                float tl = ct * a1, tr = right ? ct * a : 0.0f;
                Pending& q = pend[j];
                if (q.idx == idx) {
                    tl += q.l;
                    tr += q.r;
                } else {
                    flush(q);
                }
                red_add(gi, idx, 0, npix, tl);
                red_add(gi, idx, 1, npix, tr);
                q.idx = idx + (unsigned)W;
                q.l = cb * a1;
                q.r = right ? cb * a : 0.0f;
                // pose: P = w (U, V, 1); dP = omega x P + rho upsilon; g = dL/dP * w
                const float dIdu = __fmaf_rn(b, dx1, b1 * dx0);
                const float dIdv = __fmaf_rn(a, t.w - t.z, a1 * (t.y - t.x));
                const float U = (uj - A.cx) * rfx, V = (vj - A.cy) * rfy;
                const float gx = c * dIdu * A.fx, gy = c * dIdv * A.fy;
                const float gz = -__fmaf_rn(gx, U, gy * V);
                const float k = (j ? rho.y : rho.x) * rj;
                gp[0] += __fmaf_rn(V, gz, -gy);
                gp[1] += __fmaf_rn(-U, gz, gx);
                gp[2] += __fmaf_rn(U, gy, -V * gx);
                gp[3] = __fmaf_rn(k, gx, gp[3]);
                gp[4] = __fmaf_rn(k, gy, gp[4]);
                gp[5] = __fmaf_rn(k, gz, gp[5]);
            }
        }
        flush(pend[0]);
        flush(pend[1]);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const float t = warp_sum(gp[i]);
            if (lane == 0) ps[warp][6 * s + i] = t;
        }
    }
    __syncthreads();
    if (tid < 6 * A.S) {
        double t = 0.0;
        for (int w = 0; w < BWARPS; ++w) t += (double)ps[w][tid];
        if (t != 0.0) atomicAdd(A.gP + tid, t);
    }
}

// 16 rows per tile halve the share of the two-row rings against 8; images whose grid of 16-row tiles does not
// give every SM several CTAs take 8 rows.  A row of tiles takes all its planes before the next row, so that the rows
// of the quads that it samples and scatters into stay in the caches: 847 -> 788 us at 640x480x128 with 3 sources against
// the planes outermost.
cudaError_t launch_cost_bwd(const CostBwdArgs& A, cudaStream_t s) {
    const int gx = (A.W + 2 + BQX - 1) / BQX, gz = A.D / BPL;
    const long tall = (long)gx * ((A.H + 2 + 15) / 16) * gz;
    if (tall >= sm_count() * 6) cost_bwd_kernel<16><<<dim3(gx, gz, (A.H + 2 + 15) / 16), 32 * BWARPS, 0, s>>>(A);
    else cost_bwd_kernel<8><<<dim3(gx, gz, (A.H + 2 + 7) / 8), 32 * BWARPS, 0, s>>>(A);
    return cudaGetLastError();
}

template <int PPL> cudaError_t launch_fwd_t(const SgmLaunch& a, const RouteOut& ro, unsigned mask, cudaStream_t s) {
    const PairSet ps = make_pair_set(mask, a.W, a.H, kPairWarps);
    const size_t smem = (size_t)kPairWarps * PF * Ring<PPL, false>::STAGE_B;
    diff_fwd_kernel<PPL><<<ps.start[ps.n], 32 * kPairWarps, smem, s>>>(a, ro, ps);
    return cudaGetLastError();
}
template <int PPL> cudaError_t launch_adj_t(const AdjArgs& a, unsigned mask, cudaStream_t s) {
    const PairSet ps = make_pair_set(mask, a.W, a.H, kPairWarps);
    const size_t smem = (size_t)kPairWarps * PF * 2 * (128 * PPL + 4 * Route<PPL>::WORDS);
    diff_adj_kernel<PPL><<<ps.start[ps.n], 32 * kPairWarps, smem, s>>>(a, ps);
    return cudaGetLastError();
}
template <int PPL> cudaError_t launch_soft_t(const SoftArgs& a, int nv, cudaStream_t s) {
    const int blocks = std::min((a.N + 7) / 8, sm_count() * 16);
    if (nv == 7) soft_kernel<PPL, 7><<<blocks, 256, 0, s>>>(a);
    else soft_kernel<PPL, 3><<<blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}
#define PM_DIFF_BY_PLANES(D, CALL)                       \
    switch ((D) / 32) {                                  \
        case 1: { constexpr int P = 1; return CALL; }    \
        case 2: { constexpr int P = 2; return CALL; }    \
        case 4: { constexpr int P = 4; return CALL; }    \
        case 8: { constexpr int P = 8; return CALL; }    \
        default: return cudaErrorInvalidValue;           \
    }
cudaError_t launch_fwd(const SgmLaunch& a, const RouteOut& ro, unsigned mask, cudaStream_t s) {
    PM_DIFF_BY_PLANES(a.D, (launch_fwd_t<P>(a, ro, mask, s)))
}
cudaError_t launch_adj(const AdjArgs& a, unsigned mask, cudaStream_t s) {
    PM_DIFF_BY_PLANES(a.D, (launch_adj_t<P>(a, mask, s)))
}
cudaError_t launch_soft(const SoftArgs& a, int nv, cudaStream_t s) {
    PM_DIFF_BY_PLANES(a.D, (launch_soft_t<P>(a, nv, s)))
}

}  // namespace
}  // namespace pm

using namespace pm;

struct pm_diff {
    pm_diff_config cfg{};
    size_t N = 0, V = 0;
    float4* quads = nullptr;
    float* C = nullptr;       // costs; from the soft-argmin on, the adjoint of the SGM sum
    uint8_t* invalid = nullptr;
    bool wide = false;        // a volume for each term of the paths' sum (7) instead of 3
    float* vol = nullptr;     // forward: the paths' values; backward: the pairs' adjoints
    uint32_t* codes = nullptr;   // 8 paths' records, N each
    double* sums = nullptr;   // [loss sum, valid count, finished blocks]
    double* gP = nullptr;     // S x 6
    // inputs of the last forward
    const float* ref = nullptr;
    float hom[kMaxSources][12]{};
    float cam[4]{};
    bool have_forward = false;
    cudaEvent_t done = nullptr;   // the last call's work: the next one waits for it, on whichever stream
    size_t bytes = 0;
    std::string err;
};

namespace pm {
namespace {

pm_status dfail(pm_diff* d, pm_status s, const char* msg, cudaError_t e = cudaSuccess) {
    if (d) d->err = std::string(msg) + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : "");
    return s;
}

#define PD_CK(d, call)                                                      \
    do {                                                                    \
        cudaError_t e_ = (call);                                            \
        if (e_ != cudaSuccess) return dfail((d), PM_ERR_CUDA, #call, e_);   \
    } while (0)

struct DGuard {
    int prev = -1;
    explicit DGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

// Orders a call's launches after those of the calls before it, which share the workspaces but not necessarily the
// stream; under capture as nodes of the graph, so that the order holds where it is replayed.
class InOrder {
    pm_diff* d;
    cudaStream_t st;
    bool capturing = false, ended = false;

public:
    InOrder(pm_diff* d_, cudaStream_t st_) : d(d_), st(st_) {}
    cudaError_t begin() {
        cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
        const cudaError_t e = cudaStreamIsCapturing(st, &c);
        if (e != cudaSuccess) return e;
        capturing = c == cudaStreamCaptureStatusActive;
        return cudaStreamWaitEvent(st, d->done, capturing ? cudaEventWaitExternal : cudaEventWaitDefault);
    }
    cudaError_t end() {
        ended = true;
        return cudaEventRecordWithFlags(d->done, st, capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
    }
    ~InOrder() {   // a call that failed on the way
        if (!ended && end() != cudaSuccess) cudaGetLastError();
    }
};

void free_diff(pm_diff* d) {
    if (d->done) cudaEventDestroy(d->done);
    cudaFree(d->quads);
    cudaFree(d->C);
    cudaFree(d->invalid);
    cudaFree(d->vol);
    cudaFree(d->codes);
    cudaFree(d->sums);
    cudaFree(d->gP);
}

}  // namespace
}  // namespace pm

extern "C" {

void pm_diff_config_default(pm_diff_config* c, int width, int height, int num_planes, int num_sources) {
    if (!c) return;
    std::memset(c, 0, sizeof *c);
    c->width = width;
    c->height = height;
    c->num_planes = num_planes;
    c->num_sources = num_sources;
    c->rho0 = 0.1f;
    c->rho_step = num_planes > 1 ? 1.9f / (float)(num_planes - 1) : 1.0f;
    c->temperature = 0.05f;
    c->p1 = 0.003f;
    c->p2 = 0.01f;
    c->tau_so = 3.5f / 255.0f;
    c->q1 = 2.0f;
    c->q2 = 3.0f;
    c->store_paths = 0;
    c->device = 0;
}

pm_status pm_diff_create(const pm_diff_config* c, pm_diff** out) {
    if (!c || !out) return PM_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (c->width < 3 || c->height < 3 || c->num_planes < 32 || c->num_planes > kMaxPlanes ||
        (c->num_planes != 32 && c->num_planes != 64 && c->num_planes != 128 && c->num_planes != 256) ||
        c->num_sources < 1 || c->num_sources > kMaxDiffSources || !(c->temperature > 0.0f) || !(c->rho_step > 0.0f))
        return PM_ERR_INVALID_ARGUMENT;
    pm_diff* d = new pm_diff();
    d->cfg = *c;
    d->N = (size_t)c->width * c->height;
    d->V = d->N * c->num_planes;
    DGuard g(c->device);
    bool ok = true;
    auto alloc = [&](void** p, size_t b) {
        if (!ok) return;
        ok = cudaMalloc(p, b) == cudaSuccess;
        d->bytes += b;
    };
    alloc((void**)&d->quads, 16 * quad_stride(d->N) * c->num_sources);
    alloc((void**)&d->C, 4 * d->V);
    alloc((void**)&d->invalid, d->N);
    // 7 volumes and all paths at once, or 3 and the pairs in three launches: a choice of memory.  The 7 are faster at
    // every size (forward and backward, replayed as graphs: 0.2 M voxels 146 -> 97 us, 1.04 M 239 -> 158, 4.9 M 581 ->
    // 405, 39 M 3042 -> 2550, 59 M 3965 -> 3517), so volumes of up to 4 MB, where they add at most 17 MB, always take
    // them, and larger ones (4.9 M voxels: 179 MB against 101) where store_paths asks for it.
    d->wide = c->store_paths || d->V <= ((size_t)1 << 20);
    alloc((void**)&d->vol, 4 * d->V * (d->wide ? 7 : 3));
    const int ppl = c->num_planes / 32;
    const size_t words = ppl == 1 ? Route<1>::WORDS : ppl == 2 ? Route<2>::WORDS : ppl == 4 ? Route<4>::WORDS : Route<8>::WORDS;
    alloc((void**)&d->codes, 8 * d->N * 4 * words);
    alloc((void**)&d->sums, 3 * sizeof(double));
    alloc((void**)&d->gP, 6 * sizeof(double) * c->num_sources);
    ok = ok && cudaEventCreateWithFlags(&d->done, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        free_diff(d);
        delete d;
        return PM_ERR_OUT_OF_MEMORY;
    }
    *out = d;
    return PM_OK;
}

void pm_diff_destroy(pm_diff* d) {
    if (!d) return;
    DGuard g(d->cfg.device);
    cudaDeviceSynchronize();
    free_diff(d);
    delete d;
}

pm_status pm_diff_memory(const pm_diff* d, size_t* bytes) {
    if (!d || !bytes) return PM_ERR_INVALID_ARGUMENT;
    *bytes = d->bytes;
    return PM_OK;
}

// The forward's launches; loss: device memory (optional).
static pm_status run_forward(pm_diff* d, const float* ref, const float* srcs, const double K[9], const double* R,
                      const double* t, const float* rho_gt, float* rho_hat, double* loss, cudaStream_t st) {
    if (!d || !ref || !srcs || !K || !R || !t || !rho_gt) return PM_ERR_INVALID_ARGUMENT;
    if (!finite_n(K, 9) || K[1] != 0.0 || K[3] != 0.0 || K[6] != 0.0 || K[7] != 0.0 || K[8] != 1.0 || K[0] == 0.0 ||
        K[4] == 0.0)
        return dfail(d, PM_ERR_INVALID_ARGUMENT, "K must be [[fx, 0, cx], [0, fy, cy], [0, 0, 1]]");
    const pm_diff_config& c = d->cfg;
    const int S = c.num_sources, W = c.width, H = c.height, D = c.num_planes;
    if (!finite_n(R, 9 * S) || !finite_n(t, 3 * S)) return dfail(d, PM_ERR_INVALID_ARGUMENT, "poses must be finite");
    InOrder order(d, st);
    PD_CK(d, order.begin());
    d->ref = ref;
    // H1 = K R K^-1, H2 = K t for each source-from-reference pose
    const double Ki[9] = {1.0 / K[0], 0.0, -K[2] / K[0], 0.0, 1.0 / K[4], -K[5] / K[4], 0.0, 0.0, 1.0};
    for (int s = 0; s < S; ++s) {
        double A[9], B[9];
        matmul3(K, R + 9 * s, A);
        matmul3(A, Ki, B);
        double kt[3];
        matvec3(K, t + 3 * s, kt);
        for (int i = 0; i < 9; ++i) d->hom[s][i] = (float)B[i];
        for (int i = 0; i < 3; ++i) d->hom[s][9 + i] = (float)kt[i];
    }
    d->cam[0] = (float)K[0];
    d->cam[1] = (float)K[4];
    d->cam[2] = (float)K[2];
    d->cam[3] = (float)K[5];
    PD_CK(d, launch_to_quad_f(W, H, S, srcs, d->quads, st));
    CostLaunch a;
    std::memset(&a, 0, sizeof a);
    a.ref = ref;
    a.srcq = d->quads;
    a.W = W;
    a.H = H;
    a.D = D;
    a.nsrc = S;
    a.rho0 = c.rho0;
    a.drho = c.rho_step;
    a.mode = PM_COST_CORRECTED;
    set_floor_bias(a);
    for (int s = 0; s < S; ++s)
        for (int i = 0; i < 12; ++i) a.hom[s][i] = d->hom[s][i];
    a.cost = d->C;
    PD_CK(d, launch_cost(a, st));

    SgmLaunch g0;
    std::memset(&g0, 0, sizeof g0);
    g0.cost = d->C;
    g0.ref = ref;
    g0.W = W;
    g0.H = H;
    g0.D = D;
    g0.num_paths = 8;
    g0.p1 = c.p1; g0.p2 = c.p2; g0.tau = c.tau_so; g0.q1 = c.q1; g0.q2 = c.q2;
    RouteOut ro;
    ro.codes = d->codes;
    ro.invalid = d->invalid;
    ro.vol = d->vol;
    // S = ((((((L0 + L1) + L2) + L3) + L4) + L5) + L6) + L7: L0 and L1 meet in volume 0, the others have their own
    if (d->wide) {
        ro.slots = 0x65432100u;
        PD_CK(d, launch_fwd(g0, ro, 0xfu, st));
    } else {
        ro.slots = 0x21212100u;
        const unsigned pairs[3] = {0x3u, 0x4u, 0x8u};
        for (int i = 0; i < 3; ++i) {
            if (i) {
                float4* const v = reinterpret_cast<float4*>(d->vol);
                fold_kernel<<<sm_count() * 8, 256, 0, st>>>(v, v + d->V / 4, v + d->V / 2, d->V / 4);
                PD_CK(d, cudaGetLastError());
            }
            PD_CK(d, launch_fwd(g0, ro, pairs[i], st));
        }
    }
    SoftArgs sa;
    std::memset(&sa, 0, sizeof sa);
    sa.vol = d->vol;
    PD_CK(d, cudaMemsetAsync(d->sums, 0, 3 * sizeof(double), st));
    sa.rho_gt = rho_gt;
    sa.invalid = d->invalid;
    sa.rho_hat = rho_hat;
    sa.gS = d->C;
    sa.sums = d->sums;
    sa.loss = loss;
    sa.N = (int)d->N;
    sa.D = D;
    sa.rho0 = c.rho0;
    sa.drho = c.rho_step;
    sa.T = c.temperature;
    PD_CK(d, launch_soft(sa, d->wide ? 7 : 3, st));
    PD_CK(d, order.end());
    d->have_forward = true;
    return PM_OK;
}

// The backward's launches; grad_pose: device memory, 6 doubles per source.
static pm_status run_backward(pm_diff* d, float* grad_srcs, double* grad_pose, cudaStream_t st) {
    if (!d || !grad_srcs || !grad_pose) return PM_ERR_INVALID_ARGUMENT;
    if (!d->have_forward) return dfail(d, PM_ERR_BAD_STATE, "backward before forward");
    InOrder order(d, st);
    PD_CK(d, order.begin());
    const pm_diff_config& c = d->cfg;
    const int S = c.num_sources, D = c.num_planes;
    AdjArgs aa;
    std::memset(&aa, 0, sizeof aa);
    aa.gS = d->C;
    aa.codes = d->codes;
    aa.W = c.width;
    aa.H = c.height;
    aa.D = D;
    const int nv = d->wide ? 4 : 3;
    aa.vol = d->vol;
    aa.slots = d->wide ? 0u | 1u << 2 | 2u << 4 | 3u << 6 : 0u | 0u << 2 | 1u << 4 | 2u << 6;
    if (d->wide) {
        PD_CK(d, launch_adj(aa, 0xfu, st));
    } else {
        PD_CK(d, launch_adj(aa, 0xdu, st));
        aa.acc = 0x2u;
        PD_CK(d, launch_adj(aa, 0x2u, st));
    }
    PD_CK(d, cudaMemsetAsync(grad_srcs, 0, 4 * d->N * S, st));
    PD_CK(d, cudaMemsetAsync(grad_pose, 0, 6 * sizeof(double) * S, st));
    CostBwdArgs A;
    std::memset(&A, 0, sizeof A);
    A.ref = d->ref;
    A.quads = d->quads;
    for (int v = 0; v < nv; ++v) A.gC[v] = d->vol + (size_t)v * d->V;
    A.nv = nv;
    A.count = d->sums + 1;
    A.invalid = d->invalid;
    for (int s = 0; s < S; ++s)
        for (int i = 0; i < 12; ++i) A.hom[s][i] = d->hom[s][i];
    A.fx = d->cam[0];
    A.fy = d->cam[1];
    A.cx = d->cam[2];
    A.cy = d->cam[3];
    A.W = c.width;
    A.H = c.height;
    A.D = D;
    A.S = S;
    A.rho0 = c.rho0;
    A.drho = c.rho_step;
    A.gI = grad_srcs;
    A.gP = grad_pose;
    PD_CK(d, launch_cost_bwd(A, st));
    PD_CK(d, order.end());
    return PM_OK;
}

pm_status pm_diff_forward(pm_diff* d, const float* ref, const float* srcs, const double K[9], const double* R,
                          const double* t, const float* rho_gt, float* rho_hat, double* loss, void* stream) {
    if (!d || !loss) return PM_ERR_INVALID_ARGUMENT;
    DGuard g(d->cfg.device);
    cudaStream_t st = (cudaStream_t)stream;
    const pm_status r = run_forward(d, ref, srcs, K, R, t, rho_gt, rho_hat, nullptr, st);
    if (r != PM_OK) return r;
    double h[2];
    PD_CK(d, cudaMemcpyAsync(h, d->sums, sizeof h, cudaMemcpyDeviceToHost, st));
    PD_CK(d, cudaStreamSynchronize(st));
    *loss = h[1] > 0 ? h[0] / h[1] : 0.0;
    return PM_OK;
}

pm_status pm_diff_forward_async(pm_diff* d, const float* ref, const float* srcs, const double K[9], const double* R,
                                const double* t, const float* rho_gt, float* rho_hat, double* loss, void* stream) {
    if (!d || !loss) return PM_ERR_INVALID_ARGUMENT;
    DGuard g(d->cfg.device);
    return run_forward(d, ref, srcs, K, R, t, rho_gt, rho_hat, loss, (cudaStream_t)stream);
}

pm_status pm_diff_backward(pm_diff* d, float* grad_srcs, double* grad_pose, void* stream) {
    if (!d || !grad_pose) return PM_ERR_INVALID_ARGUMENT;
    DGuard g(d->cfg.device);
    cudaStream_t st = (cudaStream_t)stream;
    const pm_status r = run_backward(d, grad_srcs, d->gP, st);
    if (r != PM_OK) return r;
    PD_CK(d, cudaMemcpyAsync(grad_pose, d->gP, 6 * sizeof(double) * d->cfg.num_sources, cudaMemcpyDeviceToHost, st));
    PD_CK(d, cudaStreamSynchronize(st));
    return PM_OK;
}

pm_status pm_diff_backward_async(pm_diff* d, float* grad_srcs, double* grad_pose, void* stream) {
    if (!d) return PM_ERR_INVALID_ARGUMENT;
    DGuard g(d->cfg.device);
    return run_backward(d, grad_srcs, grad_pose, (cudaStream_t)stream);
}

const char* pm_diff_last_error(const pm_diff* d) { return d ? d->err.c_str() : "null handle"; }

}  // extern "C"
