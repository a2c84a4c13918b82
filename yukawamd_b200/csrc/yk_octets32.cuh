// yk_octets32.cuh -- the octet kernels' mixed form (Form32: ions with fa.lo,
// nucleons with fa.hilo).
//
// The arithmetic of a pair is that of disp_tile_x2 / screen_d_x2 and
// ion_terms_x2: exact FP32 differences of grid-rounded coordinates plus a
// correction, the hardware root and base-2 exponential.  A lane works on two
// neighbouring sources at a time, the halves of the packed FP32x2
// instructions, so the tile is stored and listed by source pairs: four
// sections of 64 units, unit p of
//   section 0  hi x0, x1, hi y0, y1     of sources 2p, 2p + 1
//   section 1  hi z0, z1, w0, w1
//   section 2  lo x0, x1, lo y0, y1
//   section 3  lo z0, z1, -, -
// A list entry is a pair of sources of which at least one is within reach; a
// batch is 16 entries, four per lane: 8 pairs per lane, 256 per warp.
//
// Sums: a batch's 8 pairs per target are added in FP32 by fours, as the tiles'
// groups of four were, and then to FP64 sums.  The measuring sums likewise, but
// for half pairs, whose lanes add up an octet's list on the tile (up to 32 pairs)
// before they go on in FP64 (the two-target kernel that had these boxes added a
// whole tile).  The 8 lanes of a source add their reactions in FP32, and those
// sums enter the warp's FP64 row of the tile, stored as FP32 (the one rounding
// that the source-side rows of the mixed form always had).  Sums of all eight in
// FP32, and of the list for all pairs too, took 48.2 and 66.3 us a step (4,096
// ions, force only and measuring) where these take 49.1 and 71.0, force error
// against FP64 2.23e-7 / 2.17e-7.
#pragma once

#include "yk_octets.cuh"

namespace yk {

// Lo part of what is beyond every cutoff: list pads, empty slots, targets that
// are none.  In the hi part it would go through the image shift, which takes
// it to exactly 0 in a box whose edge is a power of two.
constexpr float OCT_FAR32 = 1e18f;

__device__ __forceinline__ float2 oct_dup(float v) { return make_float2(v, v); }

__device__ __forceinline__ float rsqrt_ftz(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct Target32 {
    float h[3], l[3];                     // hi and lo parts, negated
    float w;
};

// One lane's measuring sums: of a batch, four pairs in each half, or (half pairs)
// of an octet on a tile.
template <bool MEAS>
struct Sum32 {
    float2 s[MEAS ? NSCAL : 1];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int k = 0; k < (MEAS ? NSCAL : 1); ++k) s[k] = oct_dup(0.f);
    }
    __device__ __forceinline__ void flush(OctetSum<MEAS>& sum)
    {
#pragma unroll
        for (int k = 0; k < (MEAS ? NSCAL : 1); ++k) sum.s[k] += (double)s[k].x + (double)s[k].y;
        zero();
    }
};

// One batch: the lane's NQ list entries (bytes of w in the lane's order q ^ sw)
// against its target.  As octet_batch: TIMG, lim and REACT mean the same; a
// pad entry is 64.
template <int SIM, bool MEAS, bool TIMG, bool REACT, int NQ>
__device__ __forceinline__ void octet_batch32(const ForceArgs& fa, const Target32& t, unsigned w, int sw, int lim,
                                              const float4* __restrict__ tile, OctetSum<MEAS>& sum, Sum32<MEAS>& ms,
                                              double* __restrict__ row)
{
    constexpr int SEC = PB / 2 + OCT_GAP;
    const int a = threadIdx.x & 7;
    float2 d[NQ][3], fs[NQ], f[3];
    int j0 = 0;
    f[0] = f[1] = f[2] = oct_dup(0.f);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int p = (int)__byte_perm(w, 0, 0x4440u | (unsigned)(q ^ sw));
        if (q == 0) j0 = 2 * p;
        const float4 A = tile[p], B = tile[p + SEC], Cc = tile[p + 2 * SEC];
        const float2 Dz = *reinterpret_cast<const float2*>(&tile[p + 3 * SEC]);
        const float2 xh[3] = {make_float2(A.x, A.y), make_float2(A.z, A.w), make_float2(B.x, B.y)};
        const float2 xl[3] = {make_float2(Cc.x, Cc.y), make_float2(Cc.z, Cc.w), Dz};
        const float2 wj = make_float2(B.z, B.w);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 dh = __fadd2_rn(xh[c], oct_dup(t.h[c]));             // exact
            float2 dl = __fadd2_rn(xl[c], oct_dup(t.l[c]));
            if constexpr (TIMG) {
                d[q][c] = __fadd2_rn(dh, dl);
            } else {
                const float2 MAG = oct_dup(12582912.0f), NMAG = oct_dup(-12582912.0f);
                const float2 k = __fadd2_rn(__ffma2_rn(dh, oct_dup(fa.invLf[c]), MAG), NMAG);
                dl = __ffma2_rn(oct_dup(-fa.Ll[c]), k, dl);
                d[q][c] = __fadd2_rn(__ffma2_rn(oct_dup(-fa.Lh[c]), k, dh), dl);
            }
        }
        float2 r2 = __fmul2_rn(d[q][2], d[q][2]);
        r2 = __ffma2_rn(d[q][1], d[q][1], r2);
        r2 = __ffma2_rn(d[q][0], d[q][0], r2);
        bool hx = r2.x <= fa.rc2f, hy = r2.y <= fa.rc2f;
        if constexpr (!TIMG) {
            hx = hx && (REACT ? 2 * p > lim : 2 * p != lim);
            hy = hy && (REACT ? 2 * p + 1 > lim : 2 * p + 1 != lim);
        }
        // ion_terms_x2: a masked pair takes r^2 = 1e36, its factor rounds to 0
        const float2 r2s = make_float2(hx ? r2.x : 1e36f, hy ? r2.y : 1e36f);
        const float2 ri = make_float2(rsqrt_ftz(r2s.x), rsqrt_ftz(r2s.y));
        const float2 mr = __fmul2_rn(oct_dup(fa.xmucf), __fmul2_rn(r2s, ri));
        const float2 y = __fmul2_rn(mr, oct_dup(-1.44269502162933349609375f));
        const float2 er = __fmul2_rn(make_float2(ex2_approx(y.x), ex2_approx(y.y)), ri);
        const float2 qq = __fmul2_rn(er, __fmul2_rn(ri, ri));
        fs[q] = __ffma2_rn(mr, qq, qq);
        const float2 g = SIM == SIM_MIX ? __fmul2_rn(fs[q], wj) : fs[q];
        if constexpr (MEAS) {
            float2 gd[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gd[c] = __fmul2_rn(g, d[q][c]);
                f[c] = __fadd2_rn(f[c], gd[c]);
            }
            const float2 u = make_float2(hx ? er.x - fa.evcutf : 0.f, hy ? er.y - fa.evcutf : 0.f);
            ms.s[0] = SIM == SIM_MIX ? __ffma2_rn(u, wj, ms.s[0]) : __fadd2_rn(ms.s[0], u);
            ms.s[1] = __ffma2_rn(g, make_float2(hx ? r2.x : 0.f, hy ? r2.y : 0.f), ms.s[1]);
            const int P[6] = {0, 0, 0, 1, 1, 2}, Q[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
            for (int k = 0; k < 6; ++k) ms.s[2 + k] = __ffma2_rn(d[q][P[k]], gd[Q[k]], ms.s[2 + k]);
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] = __ffma2_rn(g, d[q][c], f[c]);
        }
    }
    // d = x_j - x_i: the target's terms carry a minus sign (int_ion_mix.f:179)
#pragma unroll
    for (int c = 0; c < 3; ++c) sum.f[c] -= (double)f[c].x + (double)f[c].y;
    if constexpr (MEAS && !REACT) ms.flush(sum);
    if constexpr (REACT) {
        float v[3];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float2 h = SIM == SIM_MIX ? __fmul2_rn(fs[q], oct_dup(t.w)) : fs[q];
#pragma unroll
            for (int c = 0; c < 3; ++c) d[q][c] = __fmul2_rn(h, d[q][c]);
        }
        // the 8 lanes of a source: entries over xor 4 (and xor 2), then the
        // halves of the pair, then (NQ = 2) a last sum
        const bool odd = NQ == 4 ? (a & 1) : ((a >> 1) & 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float2 r;
            if constexpr (NQ == 4) {
                const float2 r0 = __fadd2_rn(d[0][c], make_float2(__shfl_xor_sync(0xffffffffu, d[2][c].x, 4),
                                                                  __shfl_xor_sync(0xffffffffu, d[2][c].y, 4)));
                const float2 r1 = __fadd2_rn(d[1][c], make_float2(__shfl_xor_sync(0xffffffffu, d[3][c].x, 4),
                                                                  __shfl_xor_sync(0xffffffffu, d[3][c].y, 4)));
                r = __fadd2_rn(r0, make_float2(__shfl_xor_sync(0xffffffffu, r1.x, 2),
                                               __shfl_xor_sync(0xffffffffu, r1.y, 2)));
                v[c] = (odd ? r.y : r.x) + __shfl_xor_sync(0xffffffffu, odd ? r.x : r.y, 1);
            } else {
                r = __fadd2_rn(d[0][c], make_float2(__shfl_xor_sync(0xffffffffu, d[1][c].x, 4),
                                                    __shfl_xor_sync(0xffffffffu, d[1][c].y, 4)));
                v[c] = (odd ? r.y : r.x) + __shfl_xor_sync(0xffffffffu, odd ? r.x : r.y, 2);
                v[c] += __shfl_xor_sync(0xffffffffu, v[c], 1);
            }
        }
        // NQ = 2: the two lanes with the same sum add it once (the other to
        // the pad's entry)
        double* e = row + 3 * ((NQ == 2 && (a & 1)) ? PB : j0 + (odd ? 1 : 0));
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c] += (double)v[c];
    }
}

// octet_batch32 for nucleons (fa.hilo; pair_group_nn_lo's arithmetic).  With
// per-pair images a pair whose hi-part displacement is hLmin or more on an
// axis takes the reference's conditional image of the FP64 positions (pt the
// target's, ps the tile's), unless no term reaches that far (no Coulomb term
// and fa.nn_short).  The terms inside rncut are taken only where a lane of
// the warp has such a pair, and, with COUL, the p-p Coulomb terms of proton
// pairs inside rccut.  Every pair from both sides: no reactions.
template <bool MEAS, bool COUL, bool TIMG, int NQ>
__device__ __forceinline__ void octet_batch32_nn(const ForceArgs& fa, const Target32& t, unsigned w, int sw, int lim,
                                                 const float4* __restrict__ tile, OctetSum<MEAS>& sum,
                                                 Sum32<MEAS>& ms,
                                                 const double4* __restrict__ pt, const double4* __restrict__ ps)
{
    constexpr int SEC = PB / 2 + OCT_GAP;
    const float rn2 = fminf(fa.rn2f, 1e35f);              // (pads and empty slots are at 1e36 or more)
    float2 d[NQ][3], r2[NQ], wj[NQ], f[3];
    unsigned ok = ~0u, fl = 0;                            // bits 2q, 2q + 1: the two pairs of entry q
    f[0] = f[1] = f[2] = oct_dup(0.f);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int p = (int)__byte_perm(w, 0, 0x4440u | (unsigned)(q ^ sw));
        const float4 A = tile[p], B = tile[p + SEC], Cc = tile[p + 2 * SEC];
        const float2 Dz = *reinterpret_cast<const float2*>(&tile[p + 3 * SEC]);
        const float2 xh[3] = {make_float2(A.x, A.y), make_float2(A.z, A.w), make_float2(B.x, B.y)};
        const float2 xl[3] = {make_float2(Cc.x, Cc.y), make_float2(Cc.z, Cc.w), Dz};
        wj[q] = make_float2(B.z, B.w);
        if constexpr (!TIMG) {
            if (2 * p == lim) ok &= ~(1u << (2 * q));
            if (2 * p + 1 == lim) ok &= ~(2u << (2 * q));
        }
        float2 mx = oct_dup(0.f);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float2 dh = __fadd2_rn(xh[c], oct_dup(t.h[c]));             // exact
            float2 dl = __fadd2_rn(xl[c], oct_dup(t.l[c]));
            if constexpr (TIMG) {
                d[q][c] = __fadd2_rn(dh, dl);
            } else {
                const float2 MAG = oct_dup(12582912.0f), NMAG = oct_dup(-12582912.0f);
                const float2 k = __fadd2_rn(__ffma2_rn(dh, oct_dup(fa.invLf[c]), MAG), NMAG);
                const float2 d1 = __ffma2_rn(oct_dup(-fa.Lh[c]), k, dh);      // exact
                mx = make_float2(fmaxf(mx.x, fabsf(d1.x)), fmaxf(mx.y, fabsf(d1.y)));
                dl = __ffma2_rn(oct_dup(-fa.Ll[c]), k, dl);
                d[q][c] = __fadd2_rn(d1, dl);
            }
        }
        if constexpr (!TIMG) {
            if (mx.x >= fa.hLmin) fl |= 1u << (2 * q);
            if (mx.y >= fa.hLmin) fl |= 2u << (2 * q);
        }
    }
    if constexpr (!TIMG) {
        if ((COUL || !fa.nn_short) && __any_sync(0xffffffffu, (fl & ok) != 0)) {
            // d = x_j - x_i from the reference's d = x_i - x_j and its image; a
            // pad, an empty slot or an empty target (|d| far on x) has no FP64
            // position
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int p = (int)__byte_perm(w, 0, 0x4440u | (unsigned)(q ^ sw));
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (((fl & ok) >> (2 * q + h) & 1u) && fabsf(h ? d[q][0].y : d[q][0].x) < 1e17f) {
                        const double4 pi = *pt, pj = ps[2 * p + h];
                        const float ex = -__double2float_rn(min_image(__dsub_rn(pi.x, pj.x), fa.xl[0], fa.hlb[0]));
                        const float ey = -__double2float_rn(min_image(__dsub_rn(pi.y, pj.y), fa.xl[1], fa.hlb[1]));
                        const float ez = -__double2float_rn(min_image(__dsub_rn(pi.z, pj.z), fa.xl[2], fa.hlb[2]));
                        if (h) d[q][0].y = ex, d[q][1].y = ey, d[q][2].y = ez;
                        else d[q][0].x = ex, d[q][1].x = ey, d[q][2].x = ez;
                    }
                }
            }
        }
    }
    unsigned mn = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        r2[q] = __fmul2_rn(d[q][2], d[q][2]);
        r2[q] = __ffma2_rn(d[q][1], d[q][1], r2[q]);
        r2[q] = __ffma2_rn(d[q][0], d[q][0], r2[q]);
        if (r2[q].x <= rn2) mn |= 1u << (2 * q);
        if (r2[q].y <= rn2) mn |= 2u << (2 * q);
    }
    mn = fa.nuclear_on ? mn & ok : 0u;
    const bool any = __any_sync(0xffffffffu, mn != 0);
    if (!COUL && !any) return;
    float2 fs[NQ], u[NQ], wv[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) fs[q] = u[q] = wv[q] = oct_dup(0.f);
    if constexpr (COUL) {
        const bool ip = t.w == 1.f;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const bool cx = ip && wj[q].x == 1.f && r2[q].x <= fa.rc2f && (TIMG || (ok >> (2 * q) & 1u));
            const bool cy = ip && wj[q].y == 1.f && r2[q].y <= fa.rc2f && (TIMG || (ok >> (2 * q + 1) & 1u));
            coulomb_terms_x2<MEAS>(fa, r2[q], make_float2(cx ? 1.f : 0.f, cy ? 1.f : 0.f), fs[q], u[q], wv[q]);
        }
    }
    if (any) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float2 Bc = make_float2(wj[q].x == t.w ? fa.bpcf : fa.bmcf, wj[q].y == t.w ? fa.bpcf : fa.bmcf);
            nuclear_terms_x2<MEAS>(fa, r2[q], make_float2(mn >> (2 * q) & 1u ? 1.f : 0.f,
                                                          mn >> (2 * q + 1) & 1u ? 1.f : 0.f), Bc, fs[q], u[q], wv[q]);
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        if constexpr (MEAS) {
            ms.s[0] = __fadd2_rn(ms.s[0], u[q]);
            ms.s[1] = __fadd2_rn(ms.s[1], wv[q]);
            const int P[6] = {0, 0, 0, 1, 1, 2}, Q[6] = {0, 1, 2, 1, 2, 2};
            float2 gd[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) gd[c] = __fmul2_rn(fs[q], d[q][c]);
#pragma unroll
            for (int k = 0; k < 6; ++k) ms.s[2 + k] = __ffma2_rn(d[q][P[k]], gd[Q[k]], ms.s[2 + k]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] = __ffma2_rn(fs[q], d[q][c], f[c]);
    }
    // d = x_j - x_i: the target's terms carry a minus sign (int_nn.f:230-240)
#pragma unroll
    for (int c = 0; c < 3; ++c) sum.f[c] -= (double)f[c].x + (double)f[c].y;
    if constexpr (MEAS) ms.flush(sum);
}

struct Form32 {
    static constexpr int PREC = PREC_MIXED, SECTIONS = 4, SEC = PB / 2, ROW = (PB + 2) * 3;
    struct Extra {};
    using Target = Target32;
    static constexpr int SMEM_SEC = SEC + OCT_GAP;

    static __device__ __forceinline__ void pack(float4* __restrict__ tile, int j, const double4& p, bool on)
    {
        float* t = reinterpret_cast<float*>(tile) + 4 * (j >> 1) + (j & 1);
        const double x[3] = {p.x, p.y, p.z};
        float h[3], l[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            // an empty slot is beyond every cutoff (OCT_FAR32, in the lo part)
            const double hd = on ? shadow_hi(x[c]) : 0.0;
            h[c] = __double2float_rn(hd);
            l[c] = on ? __double2float_rn(__dsub_rn(x[c], hd)) : OCT_FAR32;
        }
        t[0] = h[0];
        t[2] = h[1];
        t[4 * SEC] = h[2];
        t[4 * SEC + 2] = on ? (float)p.w : 0.f;
        t[8 * SEC] = l[0];
        t[8 * SEC + 2] = l[1];
        t[12 * SEC] = l[2];
        t[12 * SEC + 2] = 0.f;
    }

    static __device__ __forceinline__ void pad(float4* __restrict__ tile)
    {
        tile[SEC] = make_float4(0.f, 0.f, 0.f, 0.f);
        tile[SEC + SMEM_SEC] = make_float4(0.f, 0.f, 0.f, 0.f);
        tile[SEC + 2 * SMEM_SEC] = make_float4(OCT_FAR32, OCT_FAR32, OCT_FAR32, OCT_FAR32);
        tile[SEC + 3 * SMEM_SEC] = make_float4(OCT_FAR32, OCT_FAR32, 0.f, 0.f);
    }

    static __device__ __forceinline__ void tile_ready(const float4*, Extra&, int, int) {}

    static __device__ __forceinline__ Target target(const float4* __restrict__ posq, int R, int s, bool)
    {
        const float* t = reinterpret_cast<const float*>(posq + (size_t)R * OCT_UNITS) + 4 * (s >> 1) + (s & 1);
        Target r;
        r.h[0] = -t[0];
        r.h[1] = -t[2];
        r.h[2] = -t[4 * SEC];
        r.w = t[4 * SEC + 2];
        // no target: far from every source, the empty slots' too
        r.l[0] = t[8 * SEC] == OCT_FAR32 ? OCT_FAR32 : -t[8 * SEC];
        r.l[1] = -t[8 * SEC + 2];
        r.l[2] = -t[12 * SEC];
        return r;
    }

    static __device__ __forceinline__ double weight(const Target& t) { return (double)t.w; }

    // lane l tests pairs l and l + 32, both sources at once
    template <bool UNI, bool NUC>
    static __device__ __forceinline__ int list(const ForceArgs& fa, const float (&oc)[3], const float (&oh)[3],
                                               float limp, float lim, const float4* __restrict__ tile, const Extra&,
                                               int jlim, int jmin, unsigned char* __restrict__ l, int& kcode)
    {
        const int lane = threadIdx.x & 31;
        const unsigned below = (1u << lane) - 1u;
        unsigned c_and = 0x3fffffffu, c_or = 0u;
        reinterpret_cast<unsigned short*>(l)[lane] = SEC * 0x0101;
        __syncwarp();
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < SEC / 32; ++q) {
            if (64 * q + 64 <= jmin || 64 * q >= jlim) continue;
            const int p = 32 * q + lane;
            const float4 A = tile[p];
            const float2 x[3] = {make_float2(A.x, A.y), make_float2(A.z, A.w),
                                 *reinterpret_cast<const float2*>(&tile[p + SMEM_SEC])};
            float2 d2 = oct_dup(0.f);
            unsigned c0 = 0, c1 = 0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                // distance of the source outside the box on the axis
                float2 m;
                if constexpr (UNI) {
                    const float2 t1 = __fadd2_rn(x[c], oct_dup(-(oc[c] + oh[c])));
                    const float2 t2 = sub2(oct_dup(oc[c] - oh[c]), x[c]);
                    m = make_float2(fmaxf(fmaxf(t1.x, t2.x), 0.f), fmaxf(fmaxf(t1.y, t2.y), 0.f));
                } else {
                    float2 v = __fadd2_rn(x[c], oct_dup(-oc[c]));
                    const float2 kb = __ffma2_rn(v, oct_dup(fa.invLf[c]), oct_dup(12582912.0f));
                    v = __ffma2_rn(oct_dup(-fa.Lf[c]), __fadd2_rn(kb, oct_dup(-12582912.0f)), v);
                    c0 |= octet_image(kb.x, c);
                    c1 |= octet_image(kb.y, c);
                    m = make_float2(fmaxf(fabsf(v.x) - oh[c], 0.f), fmaxf(fabsf(v.y) - oh[c], 0.f));
                }
                d2 = __ffma2_rn(m, m, d2);
            }
            const unsigned span = (unsigned)(jlim - jmin);
            bool n0 = d2.x <= lim, n1 = d2.y <= lim;
            if constexpr (NUC) {
                const float2 wj = reinterpret_cast<const float2*>(&tile[p + SMEM_SEC])[1];
                n0 = n0 || (d2.x <= limp && wj.x == 1.f);
                n1 = n1 || (d2.y <= limp && wj.y == 1.f);
            }
            n0 = n0 && (unsigned)(2 * p - jmin) < span;
            n1 = n1 && (unsigned)(2 * p + 1 - jmin) < span;
            if constexpr (!UNI) {
                if (n0) {
                    c_and &= c0;
                    c_or |= c0;
                }
                if (n1) {
                    c_and &= c1;
                    c_or |= c1;
                }
            }
            const bool near = n0 || n1;
            const unsigned m = __ballot_sync(0xffffffffu, near);
            if (near) l[cnt + __popc(m & below)] = (unsigned char)p;
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

    template <int SIM, bool MEAS, bool RANGE, bool TIMG, bool REACT, bool COUL>
    static __device__ __forceinline__ void eval(const ForceArgs& fa, Target t, int lim, int kcode, int cnt,
                                                const float4* __restrict__ tile, const unsigned char* __restrict__ l,
                                                double, OctetSum<MEAS>& sum, double* __restrict__ row,
                                                const double4* __restrict__ pt, const double4* __restrict__ ps)
    {
        const int lane = threadIdx.x & 31, a = lane & 7, b = lane >> 3;
        const int sw4 = 2 * ((a >> 2) & 1) + ((a >> 1) & 1), sw2 = (a >> 2) & 1;
        if constexpr (TIMG) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float k = (float)octet_image_of(kcode, c);
                t.h[c] = fmaf(-k, fa.Lh[c], t.h[c]);          // exact
                t.l[c] = fmaf(-k, fa.Ll[c], t.l[c]);
            }
        }
        Sum32<MEAS> ms;
        ms.zero();
        int k = 0;
#pragma unroll 1
        for (; cnt - k > 8; k += 16) {
            const unsigned w = *reinterpret_cast<const unsigned*>(&l[k + 4 * b]);
            if constexpr (SIM == SIM_NUCLEON)
                octet_batch32_nn<MEAS, COUL, TIMG, 4>(fa, t, w, sw4, lim, tile, sum, ms, pt, ps);
            else
                octet_batch32<SIM, MEAS, TIMG, REACT, 4>(fa, t, w, sw4, lim, tile, sum, ms, row);
        }
        if (k < cnt) {
            const unsigned w = *reinterpret_cast<const unsigned short*>(&l[k + 2 * b]);
            if constexpr (SIM == SIM_NUCLEON)
                octet_batch32_nn<MEAS, COUL, TIMG, 2>(fa, t, w, sw2, lim, tile, sum, ms, pt, ps);
            else
                octet_batch32<SIM, MEAS, TIMG, REACT, 2>(fa, t, w, sw2, lim, tile, sum, ms, row);
        }
        if constexpr (MEAS && REACT) {
#pragma unroll
            for (int q = 0; q < NSCAL; ++q) sum.s[q] = (double)(ms.s[q].x + ms.s[q].y);
        }
    }
};

}  // namespace yk
