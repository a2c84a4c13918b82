// yk_gofr.cuh -- the pair-distance histogram of the two-particle correlation
// function g(r) (subroutine g, g.f:55-66; the reference has the routine but
// its calls are commented out, md.F:64, 154, 184).
//
// For every unique pair: rr = pdist(i, j) (gen_utils.f:115-128: per axis
// min(|d|, xl - |d|), the root of the sum of squares, plus the REAL*4 literal
// 1.e-15), and bin ii = min(nbin, int(fac2 rr + 1)), fac2 = 2.*float(nbin) /
// sqrt(3.) / xlmin.  Every operation is the reference's, correctly rounded and
// unfused, so each pair lands in the same bin as in the reference's loop; the
// counts are integers, exact in any order.
//
// Work: units (target tile R, source tile C >= R) of 128 x 128 slot pairs,
// spread over a fixed grid; each CTA keeps one histogram in shared memory over
// all its units (32-bit counters; a CTA takes at most GOFR_CTA_UNITS units, so
// that even all its pairs in one bin stay below 2^32) and adds it to the 64-bit
// global histogram once at the end.
//
// The exact arithmetic is about 30 FP64 instructions and a square root per
// pair, but it only matters for a pair whose distance is next to a bin edge.
// So every pair is placed in FP32 first (two sources per packed instruction),
// with a bound on the error of the place: fac2 r from FP32 copies of the
// coordinates is within GofrArgs::eps of the reference's fac2 rr, so a place
// that far or farther from both edges of its bin is the reference's.  The rest
// (1 in 1,000 on 500 bins) take the exact arithmetic.  27,000 ions, 500 bins:
// 1,037 -> 489 us a call, bound by instruction issue.  (min(|d|, L - |d|) is
// continuous in d, and |d - L rint(d / L)| is the same value, so no pair's
// image matters to the bound.)  The bound grows with the bins and with the
// box's longest edge over its shortest, and a warp takes the exact arithmetic
// as soon as one of its pairs needs it: past GOFR_PLACE_EPS every pair takes it
// in a kernel of its own (k_gofr_exact).
#pragma once

#include <algorithm>
#include <cmath>

#include "yk_force.cuh"

namespace yk {

constexpr int GOFR_BLOCK = 128;
constexpr int GOFR_MAX_BINS = 8192;          // 32 KB of shared counters
constexpr long long GOFR_CTA_UNITS = (1LL << 32) / (GOFR_BLOCK * GOFR_BLOCK) - 1;

struct GofrArgs {
    double xl[3];
    double fac2;                             // (double)(REAL*4 2*nbin/sqrt(3)) / xlmin
    double tiny;                             // (double)1.e-15f
    int nbin, n, M;                          // bins, particles, 128-slot tiles
    // FP32 place: box, 1 / box, fac2, and half a bin less eps
    float xlf[3], ixlf[3], fac2f, in_bin;
};

// Widest bound of the FP32 place, and that of small boxes, whose few units wait
// for each other's exact pairs.  FP32 place / every pair exact: 27,000 ions 4,000
// bins (eps 0.005) 731 / 1,045 us, 2,000 bins at an edge ratio of 4 (0.0089) 890
// / 1,041, 8,192 bins (0.0098) 1,037 / 1,069, 4,000 bins at 4 (0.018) 1,140 /
// 1,045; 8,000 ions 6,000 bins (0.0072) 138 / 157, 8,192 bins 169 / 157; 4,000
// ions 4,000 bins 82 / 85, 6,000 bins 92 / 90; 2,000 ions 4,000 bins 74 / 75,
// 2,000 bins at 4 78 / 70.
constexpr double GOFR_PLACE_EPS = 0.009, GOFR_PLACE_EPS_SMALL = 0.005;
constexpr int GOFR_SMALL_N = 4096;

// eps: the largest difference of the FP32 place from the reference's, in bins,
// for coordinates from -L/8 to 9L/8 on each axis (then |d| <= 5L/4, where the
// nearest image gives the reference's min(|d|, L - |d|) up to its sign).  With
// u = 2^-24, per axis: two casts 2.25 L u, the difference 1.25 L u, the FP32
// box in the image shift L u, the shift's rounding L u / 2: 5 L u, 8.7 L u for
// r (L the largest edge); r <= 0.87 L carries three relative roundings of r^2
// (1.5 u) and 2^-23 of the hardware square root, 3.1 L u: 11.8 L u in all, 14
// with a margin.  fac2 as FP32, its product with r and the subtraction of one
// half add three roundings of at most fac2 r + 1 (4 with the reference's own,
// far smaller, ones and its 1.e-15).
//
// Fills in the place's values; returns whether it is to be used.
inline bool gofr_place(GofrArgs& g)
{
    const double u = 1.0 / 16777216.0;
    const double lmax = std::max(g.xl[0], std::max(g.xl[1], g.xl[2]));
    const double wmax = g.fac2 * 0.5 * std::sqrt(g.xl[0] * g.xl[0] + g.xl[1] * g.xl[1] + g.xl[2] * g.xl[2]) + 1.0;
    const double eps = g.fac2 * (14.0 * u * lmax + 1e-15) + 4.0 * u * wmax;
    for (int k = 0; k < 3; ++k) {
        g.xlf[k] = (float)g.xl[k];
        g.ixlf[k] = (float)(1.0 / g.xl[k]);
    }
    g.fac2f = (float)g.fac2;
    g.in_bin = (float)(0.5 - eps) - 1e-6f;
    // none for boxes whose squares leave its range or with bins below it
    return eps <= (g.n <= GOFR_SMALL_N ? GOFR_PLACE_EPS_SMALL : GOFR_PLACE_EPS) && wmax < 1e6 && lmax < 1e18 && lmax > 1e-15;
}

// The reference's bin (0-based) of the pair.
__device__ __forceinline__ int gofr_bin(const GofrArgs& g, const double4& pi, const double4& pj)
{
    const double ci[3] = {pi.x, pi.y, pi.z}, cj[3] = {pj.x, pj.y, pj.z};
    double rr = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        double yy = fabs(__dsub_rn(ci[k], cj[k]));
        yy = fmin(yy, __dsub_rn(g.xl[k], yy));
        rr = __dadd_rn(rr, __dmul_rn(yy, yy));
    }
    rr = __dadd_rn(__dsqrt_rn(rr), g.tiny);
    return min(g.nbin, __double2int_rz(__dadd_rn(__dmul_rn(g.fac2, rr), 1.0))) - 1;
}

// Unit u = C (C + 1) / 2 + R with 0 <= R <= C.
__device__ __forceinline__ void gofr_tiles(long long u, int& R, int& C)
{
    C = (int)((sqrt(8.0 * (double)u + 1.0) - 1.0) * 0.5);
    while ((long long)(C + 1) * (C + 2) / 2 <= u) ++C;
    while ((long long)C * (C + 1) / 2 > u) --C;
    R = (int)(u - (long long)C * (C + 1) / 2);
}

// Every pair by the exact arithmetic.
static __global__ void __launch_bounds__(GOFR_BLOCK)
k_gofr_exact(const double4* __restrict__ pos, GofrArgs g, unsigned long long* __restrict__ hist)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    double4* tile = reinterpret_cast<double4*>(gsm);
    unsigned* h = reinterpret_cast<unsigned*>(gsm + GOFR_BLOCK * sizeof(double4));
    const int tid = threadIdx.x;
    for (int b = tid; b < g.nbin; b += GOFR_BLOCK) h[b] = 0u;
    const long long units = (long long)g.M * (g.M + 1) / 2;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        int R, C;
        gofr_tiles(u, R, C);
        const int j0 = C * GOFR_BLOCK, i = R * GOFR_BLOCK + tid;
        const int cnt = min(GOFR_BLOCK, g.n - j0);
        __syncthreads();                     // the previous unit's tile is no longer read
        if (tid < cnt) tile[tid] = pos[j0 + tid];
        __syncthreads();
        if (i >= g.n) continue;
        const double4 pi = pos[i];
        for (int jj = C == R ? tid + 1 : 0; jj < cnt; ++jj) atomicAdd(&h[gofr_bin(g, pi, tile[jj])], 1u);
    }
    __syncthreads();
    for (int b = tid; b < g.nbin; b += GOFR_BLOCK)
        if (h[b]) atomicAdd(&hist[b], (unsigned long long)h[b]);
}

// The unit loop's constants, held in registers: opaque moves, because the
// compiler otherwise loads each one from the constant bank in every pass.
struct GofrRegs {
    float il[3], nl[3], f2;
};

__device__ __forceinline__ float gofr_keep(float v)
{
    float r;
    asm volatile("mov.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

__device__ __forceinline__ float2 gofr_dup(float v) { return make_float2(v, v); }

// One target against the tile's sources jstart <= jj < cnt (EDGE: not all of
// them count; those that do not go to the counter past the last bin).  The
// lanes of a warp start at different sources, so that their counters differ.
template <bool EDGE>
__device__ __forceinline__ void gofr_unit(const GofrArgs& g, const GofrRegs& k, const float2* __restrict__ tx,
                                          unsigned hs, const double4& pi, const float (&xi)[3],
                                          const double4* __restrict__ src, int jstart, int cnt)
{
#pragma unroll 2
    for (int q = 0; q < GOFR_BLOCK / 2; ++q) {
        const int p = (q + threadIdx.x) & (GOFR_BLOCK / 2 - 1);
        float2 r2 = gofr_dup(0.f);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 d = __fadd2_rn(tx[c * (GOFR_BLOCK / 2) + p], gofr_dup(-xi[c]));
            const float2 m = __fadd2_rn(__ffma2_rn(d, gofr_dup(k.il[c]), gofr_dup(12582912.0f)),
                                        gofr_dup(-12582912.0f));
            const float2 y = __ffma2_rn(gofr_dup(k.nl[c]), m, d);
            r2 = __ffma2_rn(y, y, r2);
        }
        float2 r;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(r2.x));
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(r2.y));
        // w: the place from the middle of bin 0; b: its bin, as the low bits of
        // the magic sum; f: the place from the middle of that bin
        const float2 w = __ffma2_rn(gofr_dup(k.f2), r, gofr_dup(-0.5f));
        const float2 b = __fadd2_rn(w, gofr_dup(12582912.0f));
        const float2 f = sub2(w, __fadd2_rn(b, gofr_dup(-12582912.0f)));
        int b0 = min(__float_as_int(b.x) - 0x4B400000, g.nbin - 1);
        int b1 = min(__float_as_int(b.y) - 0x4B400000, g.nbin - 1);
        if (fmaxf(fabsf(f.x), fabsf(f.y)) > g.in_bin) {
            if (fabsf(f.x) > g.in_bin && (!EDGE || 2 * p < cnt)) b0 = gofr_bin(g, pi, src[2 * p]);
            if (fabsf(f.y) > g.in_bin && (!EDGE || 2 * p + 1 < cnt)) b1 = gofr_bin(g, pi, src[2 * p + 1]);
        }
        if constexpr (EDGE) {
            if (2 * p < jstart || 2 * p >= cnt) b0 = g.nbin;
            if (2 * p + 1 < jstart || 2 * p + 1 >= cnt) b1 = g.nbin;
        }
        asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(hs + 4u * (unsigned)b0) : "memory");
        asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(hs + 4u * (unsigned)b1) : "memory");
    }
}

static __global__ void __launch_bounds__(GOFR_BLOCK)
k_gofr(const double4* __restrict__ pos, GofrArgs g, unsigned long long* __restrict__ hist)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    float2* tx = reinterpret_cast<float2*>(gsm);               // x, y, z of the source pairs
    unsigned* h = reinterpret_cast<unsigned*>(gsm + 3 * GOFR_BLOCK * sizeof(float));
    const int tid = threadIdx.x;
    for (int b = tid; b < g.nbin; b += GOFR_BLOCK) h[b] = 0u;
    const unsigned hs = smem_u32(h);
    GofrRegs k;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        k.il[c] = gofr_keep(g.ixlf[c]);
        k.nl[c] = gofr_keep(-g.xlf[c]);
    }
    k.f2 = gofr_keep(g.fac2f);
    const long long units = (long long)g.M * (g.M + 1) / 2;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        int R, C;
        gofr_tiles(u, R, C);
        const int j0 = C * GOFR_BLOCK;
        const int cnt = min(GOFR_BLOCK, g.n - j0);
        const int i = R * GOFR_BLOCK + tid;
        const bool on = i < g.n;
        const double4 pi = pos[on ? i : g.n - 1];
        const float xi[3] = {__double2float_rn(pi.x), __double2float_rn(pi.y), __double2float_rn(pi.z)};
        const double4 pj = pos[min(j0 + tid, g.n - 1)];
        const float xj[3] = {__double2float_rn(pj.x), __double2float_rn(pj.y), __double2float_rn(pj.z)};
        bool in = true;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float mid = 0.5f * g.xlf[c], reach = 0.624f * g.xlf[c];
            in = in && fabsf(xi[c] - mid) <= reach && fabsf(xj[c] - mid) <= reach;
        }
        __syncthreads();                     // the previous unit's tile is no longer read
#pragma unroll
        for (int c = 0; c < 3; ++c) reinterpret_cast<float*>(tx)[c * GOFR_BLOCK + tid] = xj[c];
        const bool place = __syncthreads_and(in);
        const int jstart = on ? ((C == R) ? tid + 1 : 0) : cnt;
        if (!place) {
            for (int jj = jstart; jj < cnt; ++jj) atomicAdd(&h[gofr_bin(g, pi, pos[j0 + jj])], 1u);
            continue;
        }
        if (C != R && cnt == GOFR_BLOCK && (R + 1) * GOFR_BLOCK <= g.n)
            gofr_unit<false>(g, k, tx, hs, pi, xi, pos + j0, 0, GOFR_BLOCK);
        else
            gofr_unit<true>(g, k, tx, hs, pi, xi, pos + j0, jstart, cnt);
    }
    __syncthreads();
    for (int b = tid; b < g.nbin; b += GOFR_BLOCK)
        if (h[b]) atomicAdd(&hist[b], (unsigned long long)h[b]);
}

}  // namespace yk
