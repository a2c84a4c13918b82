// yk_octets.cuh -- the force kernels on octets of targets: half pairs
// (k_force_octets, ions) and every pair from both sides (k_force_octets_all, small
// boxes of ions or nucleons), their job table and combines, and the FP64 form of
// the pairs (Form64; the mixed form is in yk_octets32.cuh).
//
// Units, scratch rows and the tile layout in slots are those of yk_pairs.cuh
// (target block R of 128 slots against source tiles C).  What differs is how a
// warp works through a tile: by octets, 8 consecutive slots of the Hilbert order
// each, and a lane is (a, b) = (lane & 7, lane >> 3): target a of the octet at
// hand and every fourth source of the octet's own source list.
//
//   list    per octet, the tile's sources within the screening radius of the
//           octet's bounding box (FP32, widened as near_groups), one byte each
//   batch   16 list entries, four per lane: 4 pairs per lane, 128 pairs per
//           warp, evaluated without branches so that the four dependent
//           chains interleave; then the 8 lanes of a source add their
//           reactions (4 shuffled doubles per component for 4 sources)
//   row     the sums are added to the warp's own row of the tile
//
// An octet's box is 1.6 times smaller per axis than the box of 32 targets, and
// the list drops single sources instead of groups of 4, so fewer lanes work on
// pairs outside r_c: on the 55,296-ion mixture 74 % of the listed (target,
// source) pairs are inside r_c (67 % with the last batch of a tile padded)
// against 58 % of the pairs of the 4-source groups that 32 targets reach; on
// 51,200 nucleons 38 % against 19 % for the nuclear range.  The reactions of
// a source are added over 8 lanes instead of 32 (6 shuffles per pair instead
// of 9), and no per-pair FP32 screen is needed.
#pragma once

#include <type_traits>

#include <algorithm>

#include "yk_pairs.cuh"
#include "yk_verlet.cuh"

namespace yk {

constexpr int OCTETS = PB / 8;            // octets of a target block
constexpr int OCT_UNITS = 2 * PB;         // 16-byte units of a tile in global memory
constexpr int OCT_PAD = PB;               // list index of the pad source
constexpr int OCT_GAP = 4;                // 16-byte units between a tile's sections in shared memory (the pad's)
constexpr int OCT_ZW = PB + OCT_GAP;      // FP64 form: offset of a source's (z, w) from its (x, y) in shared memory
constexpr int OCT_WIN = 8;                // sources of a window, the unit that jobs are cut in
constexpr int OCT_WPT = PB / OCT_WIN;     // windows per tile
constexpr double OCT_FAR = 1e160;         // its coordinates: r^2 overflows, no cutoff reaches it

// ---- FP64 exp(-t) with the table in the warp's registers ---------------------
// Tang's method as exp_neg_f64, with 32 table entries: -t = (32 m + j) ln2/32 +
// r, |r| <= ln2/64; e^r - 1 from its Taylor polynomial to r^6 (truncation
// 3.5e-18 relative).  Lane l holds 2^{l/32} and the lookup is a warp shuffle
// (which takes the index mod 32), so every lane of the warp must call this
// together.  The high word of the lane's entry is stored less l << 15: adding
// (32 m + j) << 15 to it then puts m into the exponent in one integer
// operation.  At most 1.01 ulp off (0.333 on average, t = 0 .. 690), exp_neg_f64
// 1.31 (0.343).  Two FP64 FMAs more than the 256-entry table, but the lookup
// takes 2 shuffle cycles of an SM instead of a divergent load from a 2 KB
// table (about 4 cycles and a global-load latency).
__device__ __forceinline__ double exp2_32_lane()
{
    const int l = threadIdx.x & 31;
    const double v = g_exp2_256[8 * l];
    return __hiloint2double(__double2hiint(v) - (l << 15), __double2loint(v));
}

// e^{-t} for NQ values per lane into v (sc is scratch).
template <bool RANGE, int NQ>
__device__ __forceinline__ void exp_neg_f64_warp(const double (&t)[NQ], double tab, double (&sc)[NQ], double (&v)[NQ])
{
    const double MAG = 6755399441055744.0;                // 1.5 * 2^52
    const double INV = 46.16624130844683;                 // 32 / ln 2
    const double L1 = 0.02166084939249829;                // ln2/32, rounded
    const double L2 = 7.247021293269686e-19;              // ln2/32 - L1
    double r[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(-t[q], INV, MAG);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int ni = __double2loint(v[q]);
        const double tj = __shfl_sync(0xffffffffu, tab, ni);
        sc[q] = __hiloint2double(__double2hiint(tj) + (ni << 15), __double2loint(tj));
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __dsub_rn(v[q], MAG);
#pragma unroll
    for (int q = 0; q < NQ; ++q) r[q] = __fma_rn(-v[q], L1, -t[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) r[q] = __fma_rn(-v[q], L2, r[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(1.0 / 720.0, r[q], 1.0 / 120.0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(v[q], r[q], 1.0 / 24.0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(v[q], r[q], 1.0 / 6.0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(v[q], r[q], 0.5);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __fma_rn(v[q], r[q], 1.0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = __dmul_rn(v[q], r[q]);           // e^r - 1
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        v[q] = __fma_rn(sc[q], v[q], sc[q]);
        if constexpr (RANGE) v[q] = t[q] > 700.0 ? 0.0 : v[q];
    }
}

// y = 1/sqrt(x) from the hardware's FP64 estimate (rsqrt.approx.ftz.f64), one
// second-order correction as rsqrt_nr64.  The estimate's relative error is
// below 2^-20 (2^-20.05 measured over 2^-1000 .. 2^1000), so e is below 2^-19 and
// the dropped third-order term 5 e^3 / 16 below 2^-58.6, 0.02 ulp: measured over
// r^2 from 1e-6 to 1e12, 0.990 ulp at most and 0.278 on average against 0.986 and
// 0.278 of rsqrt_nr64.  It is one instruction in place of two conversions and
// an FP32 estimate (2.0 against 6.3 cycles of an SM per warp).
template <int NQ>
__device__ __forceinline__ void rsqrt_h64_step(const double (&x)[NQ], double (&y)[NQ])
{
    double e[NQ], ye[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) e[q] = __dmul_rn(x[q], y[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) e[q] = __fma_rn(-e[q], y[q], 1.0);
#pragma unroll
    for (int q = 0; q < NQ; ++q) ye[q] = __dmul_rn(y[q], e[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) e[q] = __fma_rn(e[q], 0.375, 0.5);
#pragma unroll
    for (int q = 0; q < NQ; ++q) y[q] = __fma_rn(ye[q], e[q], y[q]);
}

// The reference's conditional minimum image (int_ion_pure.f:149-150): d - L if
// d > L/2, d + L if d < -L/2.
__device__ __forceinline__ double min_image_abs(double d, double L)
{
    const bool far = fabs(d) > 0.5 * L;
    const int hi = (__double2hiint(L) ^ (__double2hiint(d) & 0x80000000)) ^ 0x80000000;   // -copysign(L, d)
    return __dadd_rn(d, far ? __hiloint2double(hi, __double2loint(L)) : 0.0);
}

// The image numbers of an octet's sources, rint(d / L) per axis, packed 10 bits
// each (from the low bits of the magic sum d / L + 1.5 2^23).
__device__ __forceinline__ unsigned octet_image(float magic_sum, int c)
{
    return (__float_as_uint(magic_sum) & 0x3ffu) << (10 * c);
}

__device__ __forceinline__ int octet_image_of(int code, int c) { return (int)((unsigned)code << (22 - 10 * c)) >> 22; }

// Whether a fold by the packed images is the reference's image of a pair within
// L/2: it takes one edge at most (particles 3/2 L or more apart, outside the
// box, keep the rest).
__device__ __forceinline__ bool octet_image_single(int code)
{
    bool one = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) one = one && abs(octet_image_of(code, c)) <= 1;
    return one;
}

// Sums of one lane over the batches of an octet on a tile.
template <bool MEAS>
struct OctetSum {
    double f[3];
    double s[MEAS ? NSCAL : 1];
    __device__ __forceinline__ void zero()
    {
        f[0] = f[1] = f[2] = 0.0;
#pragma unroll
        for (int k = 0; k < (MEAS ? NSCAL : 1); ++k) s[k] = 0.0;
    }
};

// One batch: the lane's NQ list entries (bytes of w, in the lane's swizzled
// order q ^ sw) against its target pt.  A list pad is index OCT_PAD, a
// source so far away that it is outside every cutoff.  TIMG: the tile's image
// is folded into pt and every listed source counts; otherwise each pair takes
// its own minimum image and counts iff its source index is above lim (the
// diagonal rule) or, without REACT, is not lim (the target itself).  REACT: the
// sums of the 8 lanes of a source go to row[].
template <int SIM, bool MEAS, bool RANGE, bool TIMG, bool REACT, int NQ>
__device__ __forceinline__ void octet_batch(const ForceArgs& fa, const double4& pt, unsigned w, int sw, int lim,
                                            int dup, const double2* __restrict__ tl, double tab, OctetSum<MEAS>& sum,
                                            double* __restrict__ row)
{
    // stage by stage over the lane's NQ pairs, so that their dependent chains
    // interleave
    double d[NQ][3], r2[NQ], y[NQ], sc[NQ], p[NQ], wj[NQ], r[NQ][3];
    bool hit[NQ];
    int j0 = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int jl = (int)__byte_perm(w, 0, 0x4440u | (unsigned)(q ^ sw));
        if (q == 0) j0 = jl;
        const double2 xy = tl[jl], zw = tl[jl + OCT_ZW];
        d[q][0] = __dsub_rn(pt.x, xy.x);
        d[q][1] = __dsub_rn(pt.y, xy.y);
        d[q][2] = __dsub_rn(pt.z, zw.x);
        wj[q] = zw.y;
        hit[q] = TIMG || (REACT ? jl > lim : jl != lim);
    }
    if constexpr (!TIMG) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < NQ; ++q) d[q][c] = min_image_abs(d[q][c], fa.xl[c]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) r2[q] = __dmul_rn(d[q][2], d[q][2]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) r2[q] = __fma_rn(d[q][1], d[q][1], r2[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) r2[q] = __fma_rn(d[q][0], d[q][0], r2[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        hit[q] = r2[q] <= fa.rc2 && hit[q];
        // a masked pair takes an r^2 between 1 and 2 (one select: only the
        // high word is replaced) and a zero factor
        r2[q] = __hiloint2double(hit[q] ? __double2hiint(r2[q]) : 0x3ff00000, __double2loint(r2[q]));
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[q]) : "d"(r2[q]));
    }
    rsqrt_h64_step<NQ>(r2, y);                                            // 1/r
    double mr[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) mr[q] = __dmul_rn(r2[q], y[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) mr[q] = __dmul_rn(mr[q], fa.xmuc);       // mu r
    exp_neg_f64_warp<RANGE, NQ>(mr, tab, sc, p);
#pragma unroll
    for (int q = 0; q < NQ; ++q) p[q] = __dmul_rn(p[q], y[q]);            // e^{-mu r}/r
#pragma unroll
    for (int q = 0; q < NQ; ++q) y[q] = __dmul_rn(y[q], y[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) y[q] = __dmul_rn(p[q], y[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        y[q] = __fma_rn(mr[q], y[q], y[q]);                               // (1 + mu r) e^{-mu r}/r^3
        if (!hit[q]) y[q] = 0.0;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double g = SIM == SIM_MIX ? __dmul_rn(y[q], wj[q]) : y[q];
        if constexpr (MEAS) {
            const double fx = g * d[q][0], fy = g * d[q][1], fz = g * d[q][2];
            sum.f[0] += fx;
            sum.f[1] += fy;
            sum.f[2] += fz;
            const double u = hit[q] ? p[q] - fa.evcut : 0.0;
            sum.s[0] += SIM == SIM_MIX ? u * wj[q] : u;
            sum.s[1] += g * r2[q];
            sum.s[2] += d[q][0] * fx;
            sum.s[3] += d[q][0] * fy;
            sum.s[4] += d[q][0] * fz;
            sum.s[5] += d[q][1] * fy;
            sum.s[6] += d[q][1] * fz;
            sum.s[7] += d[q][2] * fz;
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) sum.f[c] = __fma_rn(g, d[q][c], sum.f[c]);
        }
        if constexpr (REACT) {
            const double h = SIM == SIM_MIX ? __dmul_rn(y[q], pt.w) : y[q];   // reaction: Z_i fs d
#pragma unroll
            for (int c = 0; c < 3; ++c) r[q][c] = __dmul_rn(h, d[q][c]);
        }
    }
    if constexpr (REACT) {
        double t[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if constexpr (NQ == 4) {
                const double a0 = r[0][c] + __shfl_xor_sync(0xffffffffu, r[2][c], 4);
                const double a1 = r[1][c] + __shfl_xor_sync(0xffffffffu, r[3][c], 4);
                t[c] = a0 + __shfl_xor_sync(0xffffffffu, a1, 2);
            } else {
                const double a0 = r[0][c] + __shfl_xor_sync(0xffffffffu, r[1][c], 4);
                t[c] = a0 + __shfl_xor_sync(0xffffffffu, a0, 2);
            }
            t[c] += __shfl_xor_sync(0xffffffffu, t[c], 1);
        }
        // the lane's first entry is the source whose sum it holds; of the 8 / NQ
        // lanes with the same sum one adds it to the row, the others (dup bit of
        // NQ) to the pad's entry, which nothing reads
        double* e = row + 3 * ((dup & NQ) ? OCT_PAD : j0);
        e[0] -= t[0];
        e[1] -= t[1];
        e[2] -= t[2];
    }
}

// octet_batch for nucleons (int_nn.f:208-229): the HPP terms inside rncut, taken
// only if a lane of the warp has such a pair, and, with COUL (the octet and the
// tile hold protons), the p-p Coulomb terms of proton pairs inside rccut.
// Every pair from both sides: no reactions.
template <bool MEAS, bool COUL, bool TIMG, int NQ>
__device__ __forceinline__ void octet_batch_nn(const ForceArgs& fa, const double4& pt, unsigned w, int sw, int lim,
                                               const double2* __restrict__ tl, double tab, OctetSum<MEAS>& sum)
{
    double d[NQ][3], r2[NQ], fs[NQ], u[NQ], wj[NQ];
    bool ok[NQ], hn[NQ], any = false;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int jl = (int)__byte_perm(w, 0, 0x4440u | (unsigned)(q ^ sw));
        const double2 xy = tl[jl], zw = tl[jl + OCT_ZW];
        d[q][0] = __dsub_rn(pt.x, xy.x);
        d[q][1] = __dsub_rn(pt.y, xy.y);
        d[q][2] = __dsub_rn(pt.z, zw.x);
        wj[q] = zw.y;
        ok[q] = TIMG || jl != lim;
    }
    if constexpr (!TIMG) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int q = 0; q < NQ; ++q) d[q][c] = min_image_abs(d[q][c], fa.xl[c]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) r2[q] = __dmul_rn(d[q][2], d[q][2]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) r2[q] = __fma_rn(d[q][1], d[q][1], r2[q]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        r2[q] = __fma_rn(d[q][0], d[q][0], r2[q]);
        hn[q] = fa.nuclear_on && r2[q] <= fa.rn2 && ok[q];
        any = any || hn[q];
        fs[q] = 0.0;
        u[q] = 0.0;
    }
    any = __any_sync(0xffffffffu, any);
    if (!COUL && !any) return;
    double sc[NQ], v[NQ];
    if constexpr (COUL) {
        double x[NQ], y[NQ], mr[NQ];
        bool hc[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            hc[q] = r2[q] <= fa.rc2 && ok[q] && pt.w == 1.0 && wj[q] == 1.0;
            x[q] = __hiloint2double(hc[q] ? __double2hiint(r2[q]) : 0x3ff00000, __double2loint(r2[q]));
            asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[q]) : "d"(x[q]));
        }
        rsqrt_h64_step<NQ>(x, y);
#pragma unroll
        for (int q = 0; q < NQ; ++q) mr[q] = __dmul_rn(x[q], y[q]);
#pragma unroll
        for (int q = 0; q < NQ; ++q) mr[q] = __dmul_rn(mr[q], fa.xmuc);
        exp_neg_f64_warp<true, NQ>(mr, tab, sc, v);
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = __dmul_rn(__dmul_rn(v[q], fa.vc), y[q]);   // vc e^{-mu r}/r
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if constexpr (MEAS) u[q] = hc[q] ? v[q] - fa.evcut : 0.0;
            const double g = __dmul_rn(v[q], __dmul_rn(y[q], y[q]));
            fs[q] = hc[q] ? __fma_rn(mr[q], g, g) : 0.0;
        }
    }
    if (any) {
        double t[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) t[q] = hn[q] ? __dmul_rn(r2[q], fa.xp2i) : 0.0;
        exp_neg_f64_warp<true, NQ>(t, tab, sc, v);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double B = pt.w == wj[q] ? fa.bpc : fa.bmc;
            const double fn = __dmul_rn(__dmul_rn(fa.xpi, __fma_rn(fa.aa2, v[q], B)), v[q]);
            if (hn[q]) {
                fs[q] = __dadd_rn(fs[q], fn);
                if constexpr (MEAS) u[q] += (fa.aa * v[q] + B) * v[q];
            }
        }
    }
    // fs = 0 unless the pair interacts; d and r^2 of a pad or an empty target
    // are as large as OCT_FAR, and only fs d and (MEAS) fs r^2 would see it
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double f[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            f[c] = __dmul_rn(fs[q], d[q][c]);
            sum.f[c] = __dadd_rn(sum.f[c], f[c]);
        }
        if constexpr (MEAS) {
            sum.s[0] += u[q];
            sum.s[1] += fs[q] * (fs[q] != 0.0 ? r2[q] : 0.0);
            sum.s[2] += d[q][0] * f[0];
            sum.s[3] += d[q][0] * f[1];
            sum.s[4] += d[q][0] * f[2];
            sum.s[5] += d[q][1] * f[1];
            sum.s[6] += d[q][1] * f[2];
            sum.s[7] += d[q][2] * f[2];
        }
    }
}

// The octet's source list on a tile: lane l tests sources l, l + 32, ... against
// the octet's box (centre oc, half-width oh).  UNI: oc already carries the one
// image of the whole tile; otherwise each source takes its own minimum image,
// and kcode receives the common image code of the listed sources, or -1.  (A
// bounding sphere in place of the box saves 6 of the 13 instructions of a
// test but lists about 5 % more sources: 55,296 ions FP64 1,314 -> 1,361 us,
// mixed 720 -> 742 us.)
// limp, lim: squared radius for a proton and for any other source (ions: the
// same).
template <bool UNI, bool NUC>
__device__ __forceinline__ int octet_list(const ForceArgs& fa, const float (&oc)[3], const float (&oh)[3], float limp,
                                          float lim, const double2* __restrict__ tl,
                                          const float (*__restrict__ xs)[PB], int jlim, int jmin,
                                          unsigned char* __restrict__ list, int& kcode)
{
    const float MAGIC = 12582912.0f;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned c_and = 0x3fffffffu, c_or = 0u;
    reinterpret_cast<unsigned*>(list)[lane] = OCT_PAD * 0x01010101u;
    __syncwarp();
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < PB / 32; ++q) {
        if (32 * q + 32 <= jmin || 32 * q >= jlim) continue;
        const int j = 32 * q + lane;
        float dist2 = 0.f;
        unsigned code = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float v = xs[c][j] - oc[c];
            if constexpr (!UNI) {
                const float kb = fmaf(v, fa.invLf[c], MAGIC);
                v = fmaf(-fa.Lf[c], kb - MAGIC, v);
                code |= octet_image(kb, c);
            }
            const float m = fmaxf(fabsf(v) - oh[c], 0.f);
            dist2 = fmaf(m, m, dist2);
        }
        bool near = dist2 <= lim;
        if constexpr (NUC) near = near || (dist2 <= limp && tl[j + OCT_ZW].y == 1.0);
        near = near && (unsigned)(j - jmin) < (unsigned)(jlim - jmin);
        if constexpr (!UNI) {
            if (near) {
                c_and &= code;
                c_or |= code;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, near);
        if (near) list[cnt + __popc(m & below)] = (unsigned char)j;
        cnt += __popc(m);
    }
    if constexpr (!UNI) {
        c_and = __reduce_and_sync(0xffffffffu, c_and);
        c_or = __reduce_or_sync(0xffffffffu, c_or);
        kcode = (cnt != 0 && c_and == c_or) ? (int)c_or : -1;
    }
    __syncwarp();
    return cnt;
}

// One octet (target pt, diagonal rule lim) on its list of cnt sources.
template <int SIM, bool MEAS, bool RANGE, bool TIMG, bool REACT, bool COUL>
__device__ __forceinline__ void octet_eval(const ForceArgs& fa, double4 pt, int lim, int kcode, int cnt,
                                           const double2* __restrict__ tl, const unsigned char* __restrict__ list,
                                           double tab, OctetSum<MEAS>& sum, double* __restrict__ row)
{
    const int lane = threadIdx.x & 31, a = lane & 7, b = lane >> 3;
    const int sw4 = 2 * ((a >> 2) & 1) + ((a >> 1) & 1), sw2 = (a >> 2) & 1;
    const int dup = ((a & 1) ? 4 : 0) | ((a & 3) ? 2 : 0);
    if constexpr (TIMG) {
        pt.x = __fma_rn((double)octet_image_of(kcode, 0), fa.xl[0], pt.x);
        pt.y = __fma_rn((double)octet_image_of(kcode, 1), fa.xl[1], pt.y);
        pt.z = __fma_rn((double)octet_image_of(kcode, 2), fa.xl[2], pt.z);
    }
    int k = 0;
#pragma unroll 1
    for (; cnt - k > 8; k += 16) {
        const unsigned w = *reinterpret_cast<const unsigned*>(&list[k + 4 * b]);
        if constexpr (SIM == SIM_NUCLEON)
            octet_batch_nn<MEAS, COUL, TIMG, 4>(fa, pt, w, sw4, lim, tl, tab, sum);
        else
            octet_batch<SIM, MEAS, RANGE, TIMG, REACT, 4>(fa, pt, w, sw4, lim, dup, tl, tab, sum, row);
    }
    if (k < cnt) {
        const unsigned w = *reinterpret_cast<const unsigned short*>(&list[k + 2 * b]);
        if constexpr (SIM == SIM_NUCLEON)
            octet_batch_nn<MEAS, COUL, TIMG, 2>(fa, pt, w, sw2, lim, tl, tab, sum);
        else
            octet_batch<SIM, MEAS, RANGE, TIMG, REACT, 2>(fa, pt, w, sw2, lim, dup, tl, tab, sum, row);
    }
}

// What the octet kernels read of a box: slot-ordered positions by tile, 128
// (x, y) then 128 (z, w), so that the 16 sources of a batch are read from
// shared memory without bank conflicts (interleaved as double4 they took 8
// cycles of the shared-memory pipe per pair instead of 4), and the bounding
// boxes of the octets and tiles (centre, half-width with the rounding margin;
// the centre's w says whether the box holds a proton).  Written by
// k_octet_pack.
struct OctetBox {
    const double4* pos;                   // slot-ordered FP64 positions (mixed nucleon pairs next to |d| = L/2)
    const float4* posq;                   // tiles of OCT_UNITS 16-byte units
    const float4* obox;
    const float4* tbox;
    double* Si;                           // per job: target sums of its block, [PB][3]
    void* Sj;                             // per unit tri(C, R): reactions on tile C, [PB][3]
    unsigned char* Sjf;                   // per unit: 1 if its Sj row was written, 0 if it is zero
    double* Sm;                           // per job: NSCAL measuring sums
    const int4* jobs;                     // (R, s0, s1, -), row by row
    const int* row_start;                 // [M + 1]: first job of every row; [M]: the job count
    int n, M;
};

// One CTA of PB threads per tile.  A particle without a finite position counts as
// none: beyond every cutoff and, should there be others, beyond them too (the
// reference's r <= r_c is false for it; a zero factor times its distance would
// be NaN in every sum that it shares).  GATHER: after a drift, the slots' positions
// (pos) are gathered from the caller's order here (k_pack_slots' part; the FP32
// shadow is not written, no octet kernel reads it).
template <class F, bool GATHER>
static __global__ void __launch_bounds__(PB)
k_octet_pack(double4* __restrict__ pos, int n, ForceArgs fa, float4* __restrict__ posq,
             float4* __restrict__ obox, float4* __restrict__ tbox, const int* __restrict__ perm,
             const double* __restrict__ x, const double* __restrict__ zii)
{
    __shared__ float red[PWARPS][6];
    const int C = blockIdx.x, j = threadIdx.x, lane = j & 31, warp = j >> 5;
    const int i = C * PB + j;
    bool on = i < n;
    double4 p = make_double4(OCT_FAR, OCT_FAR, OCT_FAR, 0.0);
    if (on) {
        if constexpr (GATHER) {
            const int o = perm[i];
            p = make_double4(x[3 * o], x[3 * o + 1], x[3 * o + 2], zii ? zii[o] : 0.0);
            pos[i] = p;
        } else {
            p = pos[i];
        }
        on = isfinite(p.x) && isfinite(p.y) && isfinite(p.z);
        if (!on) {
            const double far = OCT_FAR * (2.0 + i);
            p = make_double4(far, far, far, 0.0);
        }
    }
    F::pack(posq + (size_t)C * OCT_UNITS, j, p, on);
    const float inf = __int_as_float(0x7f800000);
    const float v[3] = {__double2float_rn(p.x), __double2float_rn(p.y), __double2float_rn(p.z)};
    float lo[3], hi[3], cc[3], hh[3], mu[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = on ? v[c] : inf;
        hi[c] = on ? v[c] : -inf;
        // margin: 2^-18 L for the FP32 arithmetic on the boxes and the
        // sources' minimum image (a few roundings of values below L) plus
        // 2^-8 fm; a box without particles reaches nothing
        mu[c] = fmaf(3.814697265625e-6f, fa.Lf[c], (float)(2.0 * SHADOW_Q));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            if (o == 4) {
                cc[c] = lo[c] <= hi[c] ? 0.5f * (lo[c] + hi[c]) : 0.f;
                hh[c] = lo[c] <= hi[c] ? fmaf(0.5f, hi[c] - lo[c], mu[c]) : -1e18f;
            }
        }
    }
    const unsigned pm = __ballot_sync(0xffffffffu, on && p.w == 1.0);
    const int protons = __syncthreads_or(pm != 0);
    if ((j & 7) == 0) {
        float4* o = obox + 2 * ((size_t)C * OCTETS + (j >> 3));
        o[0] = make_float4(cc[0], cc[1], cc[2], (pm >> lane & 0xffu) ? 1.f : 0.f);
        o[1] = make_float4(hh[0], hh[1], hh[2], 0.f);
    }
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            red[warp][c] = lo[c];
            red[warp][3 + c] = hi[c];
        }
    __syncthreads();
    if (j == 0) {
        float a[3], b[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a[c] = fminf(fminf(red[0][c], red[1][c]), fminf(red[2][c], red[3][c]));
            b[c] = fmaxf(fmaxf(red[0][3 + c], red[1][3 + c]), fmaxf(red[2][3 + c], red[3][3 + c]));
        }
        tbox[2 * C] = make_float4(0.5f * (a[0] + b[0]), 0.5f * (a[1] + b[1]), 0.5f * (a[2] + b[2]),
                                  protons ? 1.f : 0.f);
        tbox[2 * C + 1] = make_float4(fmaf(0.5f, b[0] - a[0], mu[0]), fmaf(0.5f, b[1] - a[1], mu[1]),
                                      fmaf(0.5f, b[2] - a[2], mu[2]), 0.f);
    }
}

// Distance^2 of box (c1, h1) from box (c2, h2) in the minimum image, a lower
// bound for every pair of points in them (tile_reaches).
__device__ __forceinline__ float box_dist2(const ForceArgs& fa, const float4& c1, const float4& h1, const float4& c2,
                                           const float4& h2)
{
    const float MAGIC = 12582912.0f;
    const float d[3] = {c1.x - c2.x, c1.y - c2.y, c1.z - c2.z};
    const float h[3] = {h1.x + h2.x, h1.y + h2.y, h1.z + h2.z};
    float dist2 = 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float dm = fmaf(-fa.Lf[c], fmaf(d[c], fa.invLf[c], MAGIC) - MAGIC, d[c]);
        const float m = fmaxf(fabsf(dm) - h[c], 0.f);
        dist2 = fmaf(m, m, dist2);
    }
    return dist2;
}

// Squared radius that counts between two boxes (their centres' words): ions the
// cutoff, nucleons the nuclear range, or the Coulomb cutoff if both hold a
// proton and it is larger.
template <int SIM>
__device__ __forceinline__ float octet_lim(const ForceArgs& fa, float p1, float p2)
{
    if constexpr (SIM != SIM_NUCLEON) return fa.scr_c2;
    return (fa.coulomb_on && p1 != 0.f && p2 != 0.f) ? fmaxf(fa.scr_c2, fa.scr_n2) : fa.scr_n2;
}

// Whether an octet (box oc, oh) reaches a tile (box tc, th).  uni: seen from the
// octet's centre every source of the tile has the image kc (octet_image), and
// that is the reference's image of every pair that counts: it takes one edge at
// most (octet_image_single), and either no pair is as far as L/2 on any axis, or
// none within the cutoff is (warp_box_of's argument).
template <int SIM>
__device__ __forceinline__ bool octet_reach(const ForceArgs& fa, const float4& oc, const float4& oh, const float4& tc,
                                            const float4& th, bool& uni, int& kc)
{
    const float lim = octet_lim<SIM>(fa, oc.w, tc.w);
    const float MAGIC = 12582912.0f;
    const float td[3] = {tc.x - oc.x, tc.y - oc.y, tc.z - oc.z};
    const float thv[3] = {th.x, th.y, th.z}, ohv[3] = {oh.x, oh.y, oh.z};
    float dist2 = 0.f;
    bool one = true, cut = true;
    kc = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float kb = fmaf(td[c], fa.invLf[c], MAGIC);
        const float dm = fabsf(fmaf(-fa.Lf[c], kb - MAGIC, td[c]));
        kc |= (int)octet_image(kb, c);
        const float m = fmaxf(dm - ohv[c] - thv[c], 0.f);
        dist2 = fmaf(m, m, dist2);
        const float half = 0.5f * fa.Lf[c] - 1.0f;
        one = one && dm + thv[c] < half;
        const float s = half - ohv[c];
        cut = cut && (dm + thv[c] + ohv[c] < half || (s > 0.f && s * s > lim));
    }
    uni = one && cut && octet_image_single(kc);
    return dist2 <= lim;
}

// FP32 copies of the tile's coordinates (its unfilled slots are never listed).
__device__ __forceinline__ void octet_tile_f32(const double2* __restrict__ tl, float (*__restrict__ xs)[PB], int jmin,
                                               int jlim)
{
#pragma unroll
    for (int q = 0; q < PB / 32; ++q) {
        if (32 * q + 32 <= jmin || 32 * q >= jlim) continue;
        const int k = 32 * q + (threadIdx.x & 31);
        const double2 xy = tl[k];
        xs[0][k] = __double2float_rn(xy.x);
        xs[1][k] = __double2float_rn(xy.y);
        xs[2][k] = __double2float_rn(tl[k + OCT_ZW].x);
    }
    __syncwarp();
}

// The FP64 form: what the job loops below need of it.  The tile is two sections
// of 128 units, (x, y) and (z, w).
struct Form64 {
    static constexpr int PREC = PREC_FP64, SECTIONS = 2, SEC = PB, ROW = (PB + 1) * 3 + 1;
    struct Extra {
        float xs[3][PB];                  // the tile's coordinates in FP32, for the lists
    };
    using Target = double4;

    static __device__ __forceinline__ void pack(float4* __restrict__ tile, int j, const double4& p, bool)
    {
        double2* t = reinterpret_cast<double2*>(tile);
        t[j] = make_double2(p.x, p.y);
        t[PB + j] = make_double2(p.z, p.w);
    }

    static __device__ __forceinline__ void pad(float4* __restrict__ tile)
    {
        double2* t = reinterpret_cast<double2*>(tile);
        t[OCT_PAD] = make_double2(OCT_FAR, OCT_FAR);
        t[OCT_ZW + OCT_PAD] = make_double2(OCT_FAR, 0.0);
    }

    static __device__ __forceinline__ void tile_ready(const float4* __restrict__ tile, Extra& x, int jmin, int jlim)
    {
        octet_tile_f32(reinterpret_cast<const double2*>(tile), x.xs, jmin, jlim);
    }

    static __device__ __forceinline__ Target target(const float4* __restrict__ posq, int R, int s, bool on)
    {
        const double2* t = reinterpret_cast<const double2*>(posq) + 2 * (size_t)R * PB + s;
        const double2 xy = t[0], zw = t[PB];
        return make_double4(on ? xy.x : -OCT_FAR, xy.y, zw.x, zw.y);      // no target: no pair
    }

    static __device__ __forceinline__ double weight(const Target& t) { return t.w; }

    template <bool UNI, bool NUC>
    static __device__ __forceinline__ int list(const ForceArgs& fa, const float (&oc)[3], const float (&oh)[3],
                                               float limp, float lim, const float4* __restrict__ tile, const Extra& x,
                                               int jlim, int jmin, unsigned char* __restrict__ l, int& kcode)
    {
        return octet_list<UNI, NUC>(fa, oc, oh, limp, lim, reinterpret_cast<const double2*>(tile), x.xs, jlim, jmin, l,
                               kcode);
    }

    template <int SIM, bool MEAS, bool RANGE, bool TIMG, bool REACT, bool COUL>
    static __device__ __forceinline__ void eval(const ForceArgs& fa, const Target& t, int lim, int kcode, int cnt,
                                                const float4* __restrict__ tile, const unsigned char* __restrict__ l,
                                                double tab, OctetSum<MEAS>& sum, double* __restrict__ row,
                                                const double4* __restrict__, const double4* __restrict__)
    {
        octet_eval<SIM, MEAS, RANGE, TIMG, REACT, COUL>(fa, t, lim, kcode, cnt, reinterpret_cast<const double2*>(tile),
                                                        l, tab, sum, row);
    }
};

// Shared memory of one warp (F: Form64 or Form32).  One tile stage: the warps of
// an SM hide each other's copies (a reached tile is tens of batches), and the
// room of a second stage lets a fourth warp live on each SM sub-partition.
template <class F>
struct OctetSmem {
    float4 tile[F::SECTIONS * (F::SEC + OCT_GAP)];   // source tile (TMA) and the pad source, by section
    double row[F::ROW];                   // reactions on the tile's sources (and the pad's)
    double acc[PB * 3];                   // target sums of the job
    typename F::Extra x;
    float4 box[OCTETS][2];                // the block's octet boxes
    alignas(16) unsigned char list[PB];   // the octet's source list
    uint64_t bar;
};

// The octet's list on a tile in the image that octet_reach found, if it did;
// timg: every listed source has image kcode in every pair that counts.
template <class F, bool NUC>
__device__ __forceinline__ int octet_list_any(const ForceArgs& fa, bool uni, const float4 (&box)[2], float limp,
                                              float lim, const float4* __restrict__ tile,
                                              const typename F::Extra& x, int jlim, int jmin,
                                              unsigned char* __restrict__ list, int& kcode, bool& timg)
{
    if (jlim <= jmin) return 0;
    float oc[3] = {box[0].x, box[0].y, box[0].z};
    const float oh[3] = {box[1].x, box[1].y, box[1].z};
    timg = uni;
    if (uni) {
#pragma unroll
        for (int c = 0; c < 3; ++c) oc[c] = fmaf((float)octet_image_of(kcode, c), fa.Lf[c], oc[c]);
        return F::template list<true, NUC>(fa, oc, oh, limp, lim, tile, x, jlim, jmin, list, kcode);
    }
    const int cnt = F::template list<false, NUC>(fa, oc, oh, limp, lim, tile, x, jlim, jmin, list, kcode);
    // the listed sources' one image, where no pair inside r_c has another
    timg = kcode >= 0 && octet_image_single(kcode);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float e = 0.5f * fa.Lf[c] - oh[c] - 1.0f;
        timg = timg && e > 0.f && e * e > limp;
    }
    return cnt;
}

// Asks for units [w0, w1) (slots) of the tile at src.
template <class F>
__device__ __forceinline__ void octet_issue(float4* __restrict__ tile, const float4* __restrict__ src, int w0, int w1,
                                            uint64_t* bar)
{
    constexpr int SLOTS = PB / F::SEC;                 // slots per unit
    const unsigned bytes = (unsigned)((w1 - w0) / SLOTS) * (unsigned)sizeof(float4);
    mbar_arrive_expect_tx(bar, F::SECTIONS * bytes);
#pragma unroll
    for (int k = 0; k < F::SECTIONS; ++k)
        bulk_g2s(tile + k * (F::SEC + OCT_GAP) + w0 / SLOTS, src + k * F::SEC + w0 / SLOTS, bytes, bar);
}

// One octet on the tile at hand (sources jmin <= j < jlim, image as octet_reach
// says): its list, the pairs, the target sums into acc (this lane's target) and
// S, with REACT the reactions into row (zeroed when the first octet of the
// tile has pairs: used).
template <class F, int SIM, bool MEAS, bool RANGE, bool REACT>
__device__ __forceinline__ void octet_visit(const ForceArgs& fa, const float4* __restrict__ posq, int n, int R, int s,
                                            const float4 (&box)[2], const float4* __restrict__ tile,
                                            const typename F::Extra& x, unsigned char* __restrict__ list, bool diag,
                                            int jmin, int jlim, bool uni, int kcode, double tab,
                                            double* __restrict__ acc, double (&S)[MEAS ? NSCAL : 1],
                                            double* __restrict__ row, bool& used, float tile_p,
                                            const double4* __restrict__ pos, int C)
{
    const int lane = threadIdx.x & 31;
    const typename F::Target t = F::target(posq, R, s, R * PB + s < n);
    bool timg;
    const float limp = octet_lim<SIM>(fa, box[0].w, tile_p);
    const float lim1 = SIM == SIM_NUCLEON ? fa.scr_n2 : limp;
    const int cnt = octet_list_any<F, SIM == SIM_NUCLEON>(fa, uni, box, limp, lim1, tile, x, jlim, jmin, list, kcode, timg);
    if (cnt == 0) return;
    if (REACT && !used) {
        used = true;
#pragma unroll
        for (int k = lane; k < PB * 3; k += 32) row[k] = 0.0;
        __syncwarp();
    }
    OctetSum<MEAS> sum;
    sum.zero();
    const double4* pos_t = pos + (size_t)R * PB + s;
    const double4* pos_s = pos + (size_t)C * PB;
    const int lim = diag ? s : -1;
    auto eval = [&](auto timg_c, auto coul_c) {
        F::template eval<SIM, MEAS, RANGE, decltype(timg_c)::value, REACT, decltype(coul_c)::value>(
            fa, t, lim, kcode, cnt, tile, list, tab, sum, row, pos_t, pos_s);
    };
    const bool ti = timg && !diag;
    bool plain = true;
    if constexpr (SIM == SIM_NUCLEON) {
        if (fa.coulomb_on && box[0].w != 0.f && tile_p != 0.f) {
            plain = false;
            if (ti) eval(std::true_type{}, std::true_type{});
            else eval(std::false_type{}, std::true_type{});
        }
    }
    if (plain) {
        if (ti) eval(std::true_type{}, std::false_type{});
        else eval(std::false_type{}, std::false_type{});
    }
    // the target sums over the four source lanes
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        sum.f[c] += __shfl_xor_sync(0xffffffffu, sum.f[c], 8);
        sum.f[c] += __shfl_xor_sync(0xffffffffu, sum.f[c], 16);
    }
    if (lane < 8) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] += sum.f[c];
    }
    if constexpr (MEAS) {
#pragma unroll
        for (int k = 0; k < NSCAL; ++k) S[k] += SIM == SIM_MIX ? sum.s[k] * F::weight(t) : sum.s[k];
    }
    __syncwarp();                        // the list is free; the next octet adds to the same row
}

// Job (R, s0, s1) of box bx, one warp: target block R against the sources of
// windows s0 <= s < s1 (OCT_WIN slots each), writing the target sums to si.
// Tiles whose box is out of reach of the block's are neither loaded nor looked
// at.  A tile shared by two jobs has its row written in parts, by both.  q
// counts the tiles this warp has loaded (stage and mbarrier parity).  Returns
// false if a copy timed out.
template <class F, int SIM, bool MEAS, bool RANGE>
__device__ __forceinline__ bool octets_job(OctetSmem<F>& sm, const ForceArgs& fa, const OctetBox& bx, int R, int s0,
                                           int s1, double* __restrict__ si, double* __restrict__ sm_row,
                                           unsigned* __restrict__ err, unsigned& q, double tab)
{
    const int lane = threadIdx.x & 31, a = lane & 7;
    const int n = bx.n;
    const int C0 = s0 / OCT_WPT, C1 = (s1 + OCT_WPT - 1) / OCT_WPT;

#pragma unroll
    for (int k = lane; k < PB * 3; k += 32) sm.acc[k] = 0.0;
    sm.box[lane >> 1][lane & 1] = bx.obox[2 * R * OCTETS + lane];
    __syncwarp();

    double S[MEAS ? NSCAL : 1] = {};
    for (int Cb = C0; Cb < C1; Cb += 32) {
        // lane l: does tile Cb + l reach the block?  (tile_reaches)
        unsigned tiles;
        {
            const int C = Cb + lane;
            bool on = C < C1;
            if (on && C * OCT_WPT >= s0 && (C + 1) * OCT_WPT <= s1 &&
                box_dist2(fa, bx.tbox[2 * C], bx.tbox[2 * C + 1], bx.tbox[2 * R], bx.tbox[2 * R + 1]) > fa.scr_c2) {
                bx.Sjf[tri_index(C, R)] = 0;
                on = false;
            }
            tiles = __ballot_sync(0xffffffffu, on);
        }
#pragma unroll 1
        for (; tiles; tiles &= tiles - 1, ++q) {
            const int C = Cb + __ffs(tiles) - 1;
            if (lane == 0) octet_issue<F>(sm.tile, bx.posq + (size_t)C * OCT_UNITS, 0, PB, &sm.bar);
            // lane o < 16: octet o against the tile's box
            bool uni;
            int kc;
            const bool reach = octet_reach<SIM>(fa, sm.box[lane & 15][0], sm.box[lane & 15][1], bx.tbox[2 * C],
                                           bx.tbox[2 * C + 1], uni, kc) && lane < OCTETS;
            unsigned om = __ballot_sync(0xffffffffu, reach);
            const unsigned um = __ballot_sync(0xffffffffu, uni);
            if (!mbar_wait_warp(&sm.bar, q & 1u, err)) return false;
            const bool diag = C == R;
            const int w0 = max(0, (s0 - C * OCT_WPT) * OCT_WIN), w1 = min(PB, (s1 - C * OCT_WPT) * OCT_WIN);
            const int jlim = min(n - C * PB, w1);
            F::tile_ready(sm.tile, sm.x, w0, jlim);
            bool used = false;
#pragma unroll 1
            for (; om; om &= om - 1) {
                const int o = __ffs(om) - 1;
                const int s = 8 * o + a;                              // target slot in the block
                octet_visit<F, SIM, MEAS, RANGE, true>(fa, bx.posq, n, R, s, sm.box[o], sm.tile, sm.x, sm.list, diag,
                                                       max(diag ? 8 * o + 1 : 0, w0), jlim, ((um >> o) & 1u) != 0,
                                                       __shfl_sync(0xffffffffu, kc, o), tab, sm.acc + 3 * s, S, sm.row,
                                                       used, bx.tbox[2 * C].w, bx.pos, C);
            }
            const long long u = tri_index(C, R);
            if (!used && w0 == 0 && w1 == PB) {
                if (lane == 0) bx.Sjf[u] = 0;
            } else {
                row_t<F::PREC>* dj = static_cast<row_t<F::PREC>*>(bx.Sj) + (size_t)u * PB * 3;
#pragma unroll 4
                for (int k = 3 * w0 + lane; k < 3 * w1; k += 32) dj[k] = (row_t<F::PREC>)(used ? sm.row[k] : 0.0);
                if (lane == 0) bx.Sjf[u] = 1;
            }
            __syncwarp();                            // the tile is free
        }
    }
#pragma unroll
    for (int k = lane; k < PB * 3; k += 32) si[k] = sm.acc[k];
    if constexpr (MEAS) {
#pragma unroll
        for (int k = 0; k < NSCAL; ++k) {
            const double v = warp_sum(S[k]);
            if (lane == 0) sm_row[k] = v;
        }
    }
    __syncwarp();
    return true;
}

// One warp per CTA.  RANGE: exponents of e^{-mu r} may pass 700 (the host's
// fa.exp_ok is 0).
constexpr int OCT_WARPS = 16;                 // resident warps per SM

template <class F, int SIM, bool MEAS, bool RANGE>
__global__ void __launch_bounds__(32, OCT_WARPS)
k_force_octets(OctetBox bx, int* __restrict__ job_counter, ForceArgs fa, unsigned* __restrict__ err)
{
    __shared__ __align__(128) OctetSmem<F> sm;
    const int lane = threadIdx.x;
    if (lane == 0) {
        F::pad(sm.tile);
        mbar_init(&sm.bar, 1);
        fence_mbar_init();
    }
    __syncwarp();
    const double tab = exp2_32_lane();
    const int njobs = bx.row_start[bx.M];
    unsigned q = 0;
    int next = lane == 0 ? atomicAdd(job_counter, 1) : 0;
    for (;;) {
        const int job = __shfl_sync(0xffffffffu, next, 0);
        if (job >= njobs) break;
        const int4 js = bx.jobs[job];
        if (lane == 0) next = atomicAdd(job_counter, 1);
        if (!octets_job<F, SIM, MEAS, RANGE>(sm, fa, bx, js.x, js.y, js.z, bx.Si + (size_t)job * PB * 3,
                                          bx.Sm + (size_t)job * NSCAL, err, q, tab))
            return;
    }
}

// ---- the job table ---------------------------------------------------------
// How much work a unit holds depends on how many of its octets are within
// reach, from nothing to 16 full lists, so jobs are cut on the device by
// estimated cost, each time the slots are re-ordered: a job is a run of
// windows of one row, and the runs of a row have about equal cost.  Rows are
// dispatched in order, with long jobs first (few target sums to write and add
// up) and short ones at the end, so that the warps finish together: the rows
// up to 3/4 of the work get total / OCT_JOBS per job, the next a quarter of
// that, the last 8 % a twelfth.  (Scheduling the listed costs of 55,296 ions
// over 1,776 warps: 3 % above the mean against 6 to 37 % for row lengths that
// ignore the cost; 131,072 ions with r_c = 149 fm 4 % against 37 to 65 %.)
// No job is cut below OCT_MIN_COST, a quarter of a full unit: shorter ones cost
// more in their own overhead and sums than they balance (FP64 force kernel and
// combine, 20,000 ions with r_c = 149 fm: 174 us without the limit, 147 with it,
// 149 at twice and 212 at four times it).
// The slots of the scratch rows follow from the table, so which warp runs a
// job does not matter to the result.
constexpr int OCT_MIN_COST = 128;
constexpr int OCT_COST_CTAS = 8;
constexpr int OCT_JOBS = 3;                   // jobs per resident warp before the cuts get shorter

// Cost of every window of row R (OCT_COST_CTAS CTAs, each summing its share of
// the row): 0 in a tile out of the block's reach, else 1 and twice the number of
// the block's octets within reach of the window's sources (so 16 a tile and twice
// its (octet, source octet) pairs).
static __global__ void __launch_bounds__(256)
k_octet_cost(const float4* __restrict__ obox, const float4* __restrict__ tbox, int M, ForceArgs fa,
             unsigned char* __restrict__ cost, int* __restrict__ row_cost)
{
    constexpr int step = 8 * OCT_COST_CTAS;
    __shared__ int tot[8];
    const int R = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float4 bc = tbox[2 * R], bh = tbox[2 * R + 1];
    const float4 oc = obox[2 * (R * OCTETS + (lane & 15))], oh = obox[2 * (R * OCTETS + (lane & 15)) + 1];
    int sum = 0;
    for (int C = R + warp + 8 * (int)blockIdx.y; C < M; C += step) {
        unsigned char* out = cost + OCT_WPT * tri_index(C, R);
        int w = 0;
        if (box_dist2(fa, tbox[2 * C], tbox[2 * C + 1], bc, bh) <= fa.scr_c2) {
            // lanes 0-15: source octets 0-7; 16-31: 8-15
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int s = C * OCTETS + 8 * (lane >> 4) + k;
                const unsigned m = __ballot_sync(0xffffffffu, box_dist2(fa, obox[2 * s], obox[2 * s + 1], oc, oh) <=
                                                                  fa.scr_c2);
                if (lane == k) w = 1 + 2 * __popc(m & 0xffffu);
                if (lane == 8 + k) w = 1 + 2 * __popc(m >> 16);
            }
        }
        if (lane < OCT_WPT) out[lane] = (unsigned char)w;
        sum += w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) tot[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < 8; ++w) t += tot[w];
        row_cost[R * OCT_COST_CTAS + blockIdx.y] = t;
    }
}

// Inclusive sum of v over the block's threads (1024); tot receives the total.
__device__ __forceinline__ long long block_scan(long long v, long long* red, long long& tot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    __syncthreads();                              // red is free
    if (lane == 31) red[warp] = v;
    __syncthreads();
    long long before = 0;
    tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        if (w < warp) before += red[w];
        tot += red[w];
    }
    return v + before;
}

__device__ __forceinline__ int octet_row_cost(const int* __restrict__ row_cost, int R)
{
    int t = 0;
#pragma unroll
    for (int y = 0; y < OCT_COST_CTAS; ++y) t += row_cost[R * OCT_COST_CTAS + y];
    return max(t, 1);
}

// Jobs of every row from the row costs (one CTA): row_start[0 .. M].
static __global__ void __launch_bounds__(1024)
k_octet_rows(const int* __restrict__ row_cost, int M, int target, int* __restrict__ row_start)
{
    __shared__ long long red[32];
    long long total = 0, tot;
    for (int b = 0; b < M; b += 1024) {
        const int R = b + threadIdx.x;
        block_scan(R < M ? octet_row_cost(row_cost, R) : 0, red, tot);
        total += tot;
    }
    long long done = 0, jobs = 0;
    for (int b = 0; b < M; b += 1024) {
        const int R = b + threadIdx.x;
        const long long c = R < M ? octet_row_cost(row_cost, R) : 0;
        const long long before = done + block_scan(c, red, tot) - c;
        done += tot;
        const double u = (double)before / (double)total;
        const int f = u < 0.75 ? 1 : (u < 0.92 ? 4 : 12);
        const long long nj =
            R < M ? min(1 + (long long)((double)c * (double)f * (double)target / (double)total),
                        min(1 + c / OCT_MIN_COST, (long long)OCT_WPT * (M - R))) : 0;
        const long long end = jobs + block_scan(nj, red, tot);
        jobs += tot;
        if (R < M) row_start[R + 1] = (int)end;
    }
    if (threadIdx.x == 0) row_start[0] = 0;
}

// At most this many jobs for M rows and `target` (the shares of the work that
// the factors 1, 4 and 12 of k_octet_rows apply to are at most 1, 0.25, 0.08).
inline long long octet_jobs_cap(int M, int target) { return M + 3LL * target; }

// The jobs of row R (one CTA): window i belongs to job floor(before(i) nj /
// cost), before(i) being the cost of the windows ahead of it.  Jobs that hold
// the work of a few tiles or more are cut at tile boundaries (before(i) of the
// tile's first window), so that no tile is worked in two parts.
constexpr int OCT_SNAP_COST = 2 * OCT_WPT * (1 + 2 * OCTETS);
static __global__ void __launch_bounds__(1024)
k_octet_jobs(const unsigned char* __restrict__ cost, const int* __restrict__ row_cost, int M,
             const int* __restrict__ row_start, int4* __restrict__ jobs)
{
    __shared__ int wsum[32], ksh[1024], bsh[1024];
    const int R = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j0 = row_start[R], nj = row_start[R + 1] - j0;
    const int nw = OCT_WPT * (M - R), rc = octet_row_cost(row_cost, R);
    const double scale = (double)nj / (double)rc;
    const bool snap = (long long)rc >= (long long)nj * OCT_SNAP_COST;
    int carry = 0, last = -1;                     // cost and job index before this stretch
    for (int b = 0; b < nw; b += 1024) {
        const int i = b + tid;
        const int c = i < nw ? cost[OCT_WPT * tri_index(R + i / OCT_WPT, R) + i % OCT_WPT] : 0;
        int v = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        __syncthreads();
        if (lane == 31) wsum[warp] = v;
        __syncthreads();
        int w = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += u;
        }
        const int ahead = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
        bsh[tid] = carry + v - c + (warp > 0 ? ahead : 0);
        carry += __shfl_sync(0xffffffffu, w, 31);
        __syncthreads();
        const int k = min(nj - 1, (int)((double)bsh[snap ? tid & ~(OCT_WPT - 1) : tid] * scale));
        ksh[tid] = k;
        __syncthreads();
        const int prev = tid > 0 ? ksh[tid - 1] : last;
        if (i < nw)
            for (int u = prev + 1; u <= k; ++u) {
                jobs[j0 + u].x = R;
                jobs[j0 + u].y = OCT_WPT * R + i;
                if (u > 0) jobs[j0 + u - 1].z = OCT_WPT * R + i;
            }
        last = ksh[min(1023, nw - 1 - b)];
    }
    if (tid == 0) {
        // jobs that no window starts (the row's last ones) are empty
        for (int u = last + 1; u < nj; ++u) {
            jobs[j0 + u].x = R;
            jobs[j0 + u].y = OCT_WPT * M;
            jobs[j0 + u - 1].z = OCT_WPT * M;
        }
        jobs[j0 + nj - 1].z = OCT_WPT * M;
    }
}

// Per slot: its target sums (Si of the row's jobs) and reactions (the written
// Sj rows) in a fixed order, the reference's scaling and the store to the
// caller's order, as k_combine; measuring, also the row's sums of Sm into
// rsum[R][NSCAL].
template <int SIM, int PREC, bool MEAS>
__global__ void __launch_bounds__(COMB_THREADS)
k_octet_combine(OctetBox bx, const int* __restrict__ perm, const double* __restrict__ zii,
                const double* __restrict__ aii, ForceArgs fa, double* __restrict__ a_out, double* __restrict__ rsum)
{
    __shared__ double part[COMB_GROUPS][PB * 3];
    __shared__ int nz_count;
    extern __shared__ int comb_dyn[];             // comb_smem_bytes(M)
    const int R = bx.M - 1 - (int)blockIdx.x;
    const int g = threadIdx.x / (PB * 3), t = threadIdx.x % (PB * 3);
    constexpr size_t ROW = (size_t)PB * 3;
    const int j0 = bx.row_start[R], j1 = bx.row_start[R + 1];
    double F = 0.0;
    {
        const double* si = bx.Si + (size_t)j0 * ROW + t;
        const int nj = j1 - j0;
#pragma unroll 4
        for (int s = g; s < nj; s += COMB_GROUPS) F += si[(size_t)s * ROW];
    }
    {
        // as k_combine: one warp lists the written rows in ascending order
        unsigned char* sfl = reinterpret_cast<unsigned char*>(comb_dyn);
        int* nzl = comb_dyn + (R + 4) / 4;
        const unsigned char* fl = bx.Sjf + tri_index(R, 0);
        for (int r = threadIdx.x; r <= R; r += blockDim.x) sfl[r] = fl[r];
        __syncthreads();
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int cnt = 0;
            for (int b = 0; b <= R; b += 32) {
                const bool on = b + lane <= R && sfl[b + lane] != 0;
                const unsigned m = __ballot_sync(0xffffffffu, on);
                if (on) nzl[cnt + __popc(m & ((1u << lane) - 1u))] = b + lane;
                cnt += __popc(m);
            }
            if (lane == 0) nz_count = cnt;
        }
        __syncthreads();
        const int cnt = nz_count;
        const row_t<PREC>* sj = static_cast<const row_t<PREC>*>(bx.Sj) + (size_t)tri_index(R, 0) * ROW + t;
#pragma unroll 8
        for (int q = g; q < cnt; q += COMB_GROUPS) F += (double)sj[(size_t)nzl[q] * ROW];
    }
    part[g][t] = F;
    __syncthreads();
    const int l = threadIdx.x;
    const int p = R * PB + l;
    if (l < PB && p < fa.n) {
        double Fv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = part[0][3 * l + c];
#pragma unroll
            for (int q = 1; q < COMB_GROUPS; ++q) v += part[q][3 * l + c];
            Fv[c] = v;
        }
        const int orig = perm[p];
        store_accel<SIM>(fa, orig, SIM == SIM_MIX ? zii[orig] : 0.0, aii, Fv, a_out);
    }
    if constexpr (MEAS) {
        // warp k of the last eight sums component k over the row's jobs
        const int k = (threadIdx.x >> 5) - (COMB_THREADS / 32 - NSCAL), lane = threadIdx.x & 31;
        if (k >= 0) {
            double v = 0.0;
            for (int j = j0 + lane; j < j1; j += 32) v += bx.Sm[(size_t)j * NSCAL + k];
            v = warp_sum(v);
            if (lane == 0) rsum[(size_t)R * NSCAL + k] = v;
        }
    }
}

// ---- small boxes: every pair from both sides -----------------------------------
// A box of a few thousand particles has too few units to fill the GPU: at
// N = 4,096 the 528 half-pair units are one or two warps per SM sub-partition,
// and a single unit (16 octets, up to 128 batches in a row) takes as long as the
// whole call should.  Here each warp takes a group of four octets against a
// chunk of the sources and sums its targets' forces only: twice the pairs, but
// no reactions to add up (31 FP64 instructions per pair instead of 41, 2
// shuffles instead of 9), no source-side rows, and chunks as short as the box
// needs.  One warp per CTA and one CTA per job: the hardware hands them out.
template <class F>
struct OctetAllSmem {
    float4 tile[2][F::SECTIONS * (F::SEC + OCT_GAP)];
    double acc[32 * 3];
    typename F::Extra x;
    float4 box[4][2];
    alignas(16) unsigned char list[PB];
    uint64_t bar[2];
};

constexpr int OCT_ALL_WARPS = 16;             // resident warps per SM

// Source chunk length of k_force_octets_all for n particles: about 48 chunks, a
// power of two from 16 up to a tile and then whole tiles (no tile in two
// pieces).  Shorter chunks cost more in job overhead than they balance
// (N = 2,000: 64 sources 34.6 us per force call, 32 38, 16 44), longer ones
// leave the last jobs running alone (seen at N = 12,345, beyond the sizes that
// the kernel is given: 256 sources 115 us, 512 136).
inline int octet_all_len(int n)
{
    int len = 16;
    while (len < PB && 48 * len < n) len *= 2;
    if (len >= PB) len = std::max(len, (n / 48 + PB / 2) / PB * PB);
    return len;
}

// Largest box that takes k_force_octets_all, by form and for FP64 by cutoff (see
// the engine's octets_all).
constexpr int OCT_ALL_MAX_N64 = 9216, OCT_ALL_MAX_N64_WIDE = 8704, OCT_ALL_MAX_N64_UNCUT = 7168;
constexpr int OCT_ALL_MAX_N32 = 6144;

// posq etc. as OctetBox; part: target sums [chunk][slot][3], np slots; Sm: per job.
template <class F, int SIM, bool MEAS, bool RANGE>
__global__ void __launch_bounds__(32, OCT_ALL_WARPS)
k_force_octets_all(OctetBox bx, int chunks, int len, double* __restrict__ part, ForceArgs fa,
                   unsigned* __restrict__ err)
{
    __shared__ __align__(128) OctetAllSmem<F> sm;
    const int lane = threadIdx.x, a = lane & 7;
    const int n = bx.n;
    const int g = blockIdx.x / chunks, ch = blockIdx.x % chunks;   // target group, source chunk
    const int j0 = ch * len, j1 = min(n, j0 + len);                // sources
    const int C0 = j0 / PB, C1 = (j1 + PB - 1) / PB;
    const int R = g / (PB / 32);
    if (lane == 0) {
        mbar_init(&sm.bar[0], 1);
        mbar_init(&sm.bar[1], 1);
        fence_mbar_init();
    }
    __syncwarp();
    // the slots of tile C that the chunk covers, in pieces of 8
    auto issue = [&](int C, unsigned qq) {
        octet_issue<F>(sm.tile[qq & 1], bx.posq + (size_t)C * OCT_UNITS, max(0, j0 - C * PB),
                       min(PB, ((j1 - C * PB) + 7) & ~7), &sm.bar[qq & 1]);
    };
    // a chunk inside one tile asks for it at once
    const bool single = C1 - C0 == 1;
    if (single && lane == 0) issue(C0, 0u);
    if (lane < 8) sm.box[lane >> 1][lane & 1] = bx.obox[8 * g + lane];
    if (lane < 2) F::pad(sm.tile[lane]);
    const double tab = exp2_32_lane();
#pragma unroll
    for (int k = lane; k < 32 * 3; k += 32) sm.acc[k] = 0.0;
    double S[MEAS ? NSCAL : 1] = {};
    unsigned q = 0;
    bool ok = true;
    __syncwarp();
    for (int Cb = C0; ok && Cb < C1; Cb += 32) {
        // lane l: does any octet of the group reach tile Cb + l?
        bool on = false;
        if (!single && Cb + lane < C1) {
            const float4 tc = bx.tbox[2 * (Cb + lane)], th = bx.tbox[2 * (Cb + lane) + 1];
#pragma unroll
            for (int o = 0; o < 4; ++o)
                on = on || box_dist2(fa, tc, th, sm.box[o][0], sm.box[o][1]) <=
                               octet_lim<SIM>(fa, tc.w, sm.box[o][0].w);
        }
        unsigned tiles = single ? 1u : __ballot_sync(0xffffffffu, on), ahead = tiles, asked = q;
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (ahead) {
                if (!single && lane == 0) issue(Cb + __ffs(ahead) - 1, asked);
                ++asked;
                ahead &= ahead - 1;
            }
#pragma unroll 1
        for (; tiles; tiles &= tiles - 1, ++q) {
            const int C = Cb + __ffs(tiles) - 1;
            const int st = q & 1;
            bool uni;
            int kc;
            const bool reach = octet_reach<SIM>(fa, sm.box[lane & 3][0], sm.box[lane & 3][1], bx.tbox[2 * C],
                                           bx.tbox[2 * C + 1], uni, kc) && lane < 4;
            unsigned om = __ballot_sync(0xffffffffu, reach);
            const unsigned um = __ballot_sync(0xffffffffu, uni);
            if (!mbar_wait_warp(&sm.bar[st], (q >> 1) & 1u, err)) {
                ok = false;
                break;
            }
            const bool diag = C == R;
            const int jmin = max(0, j0 - C * PB), jlim = min(PB, j1 - C * PB);
            F::tile_ready(sm.tile[st], sm.x, jmin, jlim);
            bool used = false;
#pragma unroll 1
            for (; om; om &= om - 1) {
                const int o = __ffs(om) - 1;
                octet_visit<F, SIM, MEAS, RANGE, false>(fa, bx.posq, n, R, 32 * (g % (PB / 32)) + 8 * o + a, sm.box[o],
                                                        sm.tile[st], sm.x, sm.list, diag, jmin, jlim,
                                                        ((um >> o) & 1u) != 0, __shfl_sync(0xffffffffu, kc, o), tab,
                                                        sm.acc + 3 * (8 * o + a), S, nullptr, used, bx.tbox[2 * C].w,
                                                        bx.pos, C);
            }
            if (ahead) {
                if (lane == 0) issue(Cb + __ffs(ahead) - 1, asked);
                ++asked;
                ahead &= ahead - 1;
            }
        }
        // a copy never completed: wait (bounded) for the other one in flight
        if (!ok && asked - q > 1) mbar_wait_bounded(&sm.bar[(q + 1) & 1], ((q + 1) >> 1) & 1u, err);
    }
    if (!ok) return;
    __syncwarp();
    double* out = part + ((size_t)ch * bx.M * PB + 32 * g) * 3;
#pragma unroll
    for (int k = lane; k < 32 * 3; k += 32) out[k] = sm.acc[k];
    if constexpr (MEAS) {
#pragma unroll
        for (int k = 0; k < NSCAL; ++k) {
            const double v = warp_sum(S[k]);
            if (lane == 0) bx.Sm[(size_t)blockIdx.x * NSCAL + k] = v;
        }
    }
}

// Per slot: the sum of its chunks in order (two halves), the reference's scaling and the store;
// measuring, also the block's sums of Sm (rows of its four groups) into rsum.
// TAIL: the rest of the step too (step_tail_particle, step_tail_finish).  A
// small box's step is mostly kernels of 1.5 to 4 us and the gaps between them:
// with GATHER and TAIL a plain one has four instead of seven (4,096 ions, 100
// steps: FP64 6.26 -> 5.87 ms, mixed 4.54 -> 4.16).
template <int SIM, bool MEAS, bool TAIL>
__global__ void __launch_bounds__(COMB_THREADS)
k_octet_all_combine(const double* __restrict__ part, const double* __restrict__ Sm, int chunks, int M,
                    const int* __restrict__ perm, const double* __restrict__ zii, const double* __restrict__ aii,
                    ForceArgs fa, double* __restrict__ a_out, double* __restrict__ rsum, StepTail tail)
{
    __shared__ double half[COMB_GROUPS][PB * 3];
    const int R = blockIdx.x;
    const int g = threadIdx.x / (PB * 3), t = threadIdx.x % (PB * 3);
    const size_t stride = (size_t)M * PB * 3;
    const double* p = part + (size_t)R * PB * 3 + t;
    double F = 0.0;
#pragma unroll 8
    for (int s = g; s < chunks; s += COMB_GROUPS) F += p[(size_t)s * stride];
    half[g][t] = F;
    __syncthreads();
    const int l = threadIdx.x;
    if (l < PB && R * PB + l < fa.n) {
        double Fv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double v = half[0][3 * l + c];
#pragma unroll
            for (int q = 1; q < COMB_GROUPS; ++q) v += half[q][3 * l + c];
            Fv[c] = v;
        }
        const int orig = perm[R * PB + l];
        store_accel<SIM>(fa, orig, SIM == SIM_MIX ? zii[orig] : 0.0, aii, Fv, a_out);
        if constexpr (TAIL) step_tail_particle(tail, a_out, orig);
    }
    if (TAIL && R == 0 && threadIdx.x >= COMB_THREADS - 32) step_tail_finish(tail, a_out);
    if constexpr (MEAS) {
        const int k = (threadIdx.x >> 5) - (COMB_THREADS / 32 - NSCAL), lane = threadIdx.x & 31;
        if (k >= 0) {
            double v = 0.0;
            const int r0 = R * (PB / 32) * chunks, r1 = r0 + (PB / 32) * chunks;
            for (int j = r0 + lane; j < r1; j += 32) v += Sm[(size_t)j * NSCAL + k];
            v = warp_sum(v);
            if (lane == 0) rsum[(size_t)R * NSCAL + k] = v;
        }
    }
}

}  // namespace yk
