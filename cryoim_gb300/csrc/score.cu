// score.cu — cross-common-line phase-residual scoring and symmetrised insertion.
//
// k_pr_omega is the hot kernel of the global search (cal_crosslin_PR_omega.f90 for
// every asymmetric-unit view of every particle).  One CTA owns one (particle, view):
//   * the particle's band-limited Fourier window (W x W float2) sits in shared memory
//     for the whole CTA, so every bilinear tap is a shared-memory load;
//   * thread (g, k) owns omega index k (and k + half a turn where the grid has it) and
//     accumulates PR1(k), PR2(k) in registers over the valid lines g, g+G, ... of every
//     template (no cross-thread reduction until the end of the view), with per-line FP32
//     partial sums folded into Kahan-compensated running sums;
//   * per template, the 60 x nR template line samples (template x CTF, bilinear) are
//     staged once into shared memory as (amplitude or -1 if below Fcut, phase);
//   * the per-view argmin over omega is folded into a per-particle 64-bit key
//     (PR bits << 32 | column-major index) with atomicMin, which reproduces Fortran
//     minloc's first-occurrence rule.
// The sampling positions x = FR*cos + nx/2 are rounded exactly as the reference
// rounds them (separate multiply and add), so the bilinear taps and weights match it.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "geom.cuh"
#include "reduce.cuh"
#include "kernels.h"
#include "launch.h"

namespace cryoim {
namespace {

__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}
// h + l += x with Knuth's TwoSum: the pair holds the running sum to ~2^-48 relative in
// FP32 arithmetic (GB300's FP64 pipe is far slower than its FP32 pipe)
__device__ __forceinline__ void two_sum_acc(float& h, float& l, float x) {
    const float s2 = h + x, bb = s2 - h;
    l += (h - (s2 - bb)) + (x - bb);
    h = s2;
}

__device__ __forceinline__ float bilerp(float ax, float ay, float v00, float v10, float v01,
                                        float v11) {
    float bx = 1.0f - ax, by = 1.0f - ay;
    return bx * by * v00 + ax * by * v10 + bx * ay * v01 + ax * ay * v11;
}

struct Consts {
    float d2r, r2d, pi, tpi;
    float margin;  // k_pr_omega in pairs: share of a cut within which an amplitude is in doubt
};

// Template line sample (template x CTF, bilinear) at angle alpha2, radius fr.
__device__ __forceinline__ void tmpl_sample_cs(const float2* __restrict__ tb, const float* __restrict__ cb,
                                               int W, int offW, float nxh, float cs, float sn, float fr,
                                               float* re, float* im) {
    float x = __fadd_rn(__fmul_rn(fr, cs), nxh), y = __fadd_rn(__fmul_rn(fr, sn), nxh);
    int lx = (int)x, ly = (int)y;
    float ax = __fsub_rn(x, (float)lx), ay = __fsub_rn(y, (float)ly);
    int b0 = ly * W + lx - offW;
    float2 t00 = tb[b0], t10 = tb[b0 + 1], t01 = tb[b0 + W], t11 = tb[b0 + W + 1];
    if (cb) {
        float c00 = cb[b0], c10 = cb[b0 + 1], c01 = cb[b0 + W], c11 = cb[b0 + W + 1];
        t00.x = __fmul_rn(t00.x, c00); t00.y = __fmul_rn(t00.y, c00);
        t10.x = __fmul_rn(t10.x, c10); t10.y = __fmul_rn(t10.y, c10);
        t01.x = __fmul_rn(t01.x, c01); t01.y = __fmul_rn(t01.y, c01);
        t11.x = __fmul_rn(t11.x, c11); t11.y = __fmul_rn(t11.y, c11);
    }
    *re = bilerp(ax, ay, t00.x, t10.x, t01.x, t11.x);
    *im = bilerp(ax, ay, t00.y, t10.y, t01.y, t11.y);
}

// The same sample from a band stored as (pixel, right neighbour) pairs: two 16-byte loads
// carry the four taps, the values and the arithmetic are tmpl_sample_cs's.
__device__ __forceinline__ void tmpl_sample_pairs(const float4* __restrict__ tb, int W, int offW, float nxh, float cs,
                                                  float sn, float fr, float* re, float* im) {
    float x = __fadd_rn(__fmul_rn(fr, cs), nxh), y = __fadd_rn(__fmul_rn(fr, sn), nxh);
    int lx = (int)x, ly = (int)y;
    float ax = __fsub_rn(x, (float)lx), ay = __fsub_rn(y, (float)ly);
    int b0 = ly * W + lx - offW;
    const float4 r0 = tb[b0], r1 = tb[b0 + W];
    *re = bilerp(ax, ay, r0.x, r0.z, r1.x, r1.z);
    *im = bilerp(ax, ay, r0.y, r0.w, r1.y, r1.w);
}

__device__ __forceinline__ void tmpl_sample(const float2* __restrict__ tb, const float* __restrict__ cb,
                                            int W, int offW, float nxh, float alpha2, float fr,
                                            float d2r, float* re, float* im) {
    float ang = __fmul_rn(alpha2, d2r);
    tmpl_sample_cs(tb, cb, W, offW, nxh, cosf(ang), sinf(ang), fr, re, im);
}

// Angle between two complex numbers z1, z2 from their cross and dot products, in [0, pi]:
// |arg(z2 conj z1)| = the reference's |phase2 - phase1| folded into [0, pi]
// (cal_crosslin_PR_omega.f90:53-60).  atan on [0, 1] is a 6-term odd polynomial fitted
// to atan(t)/t by reweighted least squares on [0, 1] (max error 1.7e-6 rad in FP32).
__device__ __forceinline__ float angle_between(float cross, float dot, float pi) {
    const float a = fabsf(cross), b = fabsf(dot);
    const float mx = fmaxf(a, b), mn = fminf(a, b);
    const float t = mn * __frcp_rn(mx);
    const float s = t * t;
    float p = fmaf(s, -0.011719364672899246f, 0.05264794081449509f);
    p = fmaf(p, s, -0.11642702668905258f);
    p = fmaf(p, s, 0.19354058802127838f);
    p = fmaf(p, s, -0.33262285590171814f);
    p = fmaf(p, s, 0.9999772310256958f);
    float r = t * p;
    r = (a > b) ? 0.5f * pi - r : r;
    return (dot < 0.0f) ? pi - r : r;
}

// angle_between with the hardware reciprocal estimate (relative error ~2^-23, below the
// polynomial's 1.7e-6 rad) in place of the correctly rounded one.
__device__ __forceinline__ float angle_between_est(float cross, float dot, float pi) {
    const float a = fabsf(cross), b = fabsf(dot);
    const float mx = fmaxf(a, b), mn = fminf(a, b);
    float rc;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(mx));
    const float t = mn * rc;
    const float s = t * t;
    float p = fmaf(s, -0.011719364672899246f, 0.05264794081449509f);
    p = fmaf(p, s, -0.11642702668905258f);
    p = fmaf(p, s, 0.19354058802127838f);
    p = fmaf(p, s, -0.33262285590171814f);
    p = fmaf(p, s, 0.9999772310256958f);
    float r = t * p;
    r = (a > b) ? 0.5f * pi - r : r;
    return (dot < 0.0f) ? pi - r : r;
}

// One PR term of a particle sample z (Re, -Im): the angle to the template sample e (a, b, half
// amplitude) and the weight.
struct OmegaTerm {
    float2 z;
    float amp, w;
};
// The particle's sample at radius fr in direction csn of the band in shared memory.
__device__ __forceinline__ OmegaTerm omega_sample(const float2* sband, int W, int offW, float fr, float2 csn,
                                                  float nxh, float half2) {
    // sample position (x, y) = FR (cos, sin) + nx/2, then its cell
    const float2 xy = __ffma2_rn(make_float2(fr, fr), csn, make_float2(nxh, nxh));
    const int lx = (int)xy.x, ly = (int)xy.y;
    const float2 f = __fadd2_rn(xy, make_float2(-(float)lx, -(float)ly));
    const int b0 = ly * W + lx - offW;
    const float2 t00 = sband[b0], t10 = sband[b0 + 1];
    const float2 t01 = sband[b0 + W], t11 = sband[b0 + W + 1];
    // bilinear on (re, im) pairs: lerp in x on both rows, then in y
    const float2 ax2 = make_float2(f.x, f.x), ay2 = make_float2(f.y, f.y);
    const float2 m1 = make_float2(-1.f, -1.f);
    const float2 v0 = __ffma2_rn(ax2, __ffma2_rn(t00, m1, t10), t00);
    const float2 v1 = __ffma2_rn(ax2, __ffma2_rn(t01, m1, t11), t01);
    OmegaTerm r;
    r.z = __ffma2_rn(ay2, __ffma2_rn(v0, m1, v1), v0);
    const float2 zz = __fmul2_rn(r.z, r.z);
    const float sq = zz.x + zz.y;
    r.amp = sq * rsqrtf(sq);  // NaN for 0: fails the cut
    r.w = fmaf(0.5f, r.amp, half2);
    return r;
}

// HALF: thread (g, k) owns omega k and k + nomega / 2, half a turn apart.  The particle's
// samples along a line and along its reverse are complex conjugates (the image is real), so one
// sample, its amplitude, cut and weight serve both; the cross and dot products differ by the
// sign of one of the two products each.  The two samples' positions round differently (at box 256 and
// maxR 64 by 1e-5 px, 8e-5 at most), so where the amplitude lies within a margin of its cut the second
// omega's sample is taken by itself.  The margin is a rule of thumb: the amplitudes near a cut
// were seen to differ by up to 3e-4 of it for noise and particles at box 256, 6e-4 beside lattice peaks, and
// by as much more in a larger box as its positions round more.  A term in doubt beyond it may count
// at one omega of the pair and not in the search by single omegas, which is then 1 / terms off (2e-5 at
// 60,000 terms), as the other rounding of a position can have it anyway.
// Issue-bound (76 %; by single omegas 80 %, and the L1 data pipe 76 %): a particle of box 256 on
// the 1-degree grid takes 13.1 ms in pairs, 17.8 by single omegas.  The margin's terms are marked
// and taken after each 32 radii: inside the unrolled loop they cost more than the pairs gain (19
// ms).  Cells by the add of 2^23 in place of conversions (which wait for the reciprocals'
// quarter-rate pipe) gained nothing.
constexpr float PAIR_MARGIN = 5.0e-4f;  // of the cut, up to box 256; beyond (LARGE) as the box
// SHARE: blockIdx.z takes its share of the omegas (an instance of its own: the indices cost the other 2 %).
template <bool HALF, bool SHARE, bool LARGE>
__global__ void __launch_bounds__(768, 1) k_pr_omega(PrOmegaArgs a, int nall, int Gall, Consts K) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const Band bd = a.bd;
    const int W = bd.W, nr = bd.nr, minR = bd.min_r;
    float2* sband = reinterpret_cast<float2*>(smraw);
    // per (line, radius): template sample (a2, b2), half amplitude (-1 below its cut),
    // particle cut at that radius
    float4* sline = reinterpret_cast<float4*>(sband + W * W);
    float2* sred = reinterpret_cast<float2*>(sline);  // [1 or 2][threads], once a view's lines are done
    float* sfc0 = reinterpret_cast<float*>(sline + max(60 * nr, (int)blockDim.x / (HALF ? 1 : 2)));
    unsigned long long* skey = reinterpret_cast<unsigned long long*>(sfc0 + ((nr + 3) & ~3));
    float* salpha = reinterpret_cast<float*>(skey + 32);  // particle line angles of the template's valid lines
    int* sjl = reinterpret_cast<int*>(salpha + 64);       // and which lines they are
    int* snv = sjl + 64;

    const int p = blockIdx.y, t = threadIdx.x;
    // this block's omegas: k0 .. k0 + nown - 1 of nall (and, HALF, those half a turn on)
    const int share = SHARE ? (nall + (int)gridDim.z - 1) / (int)gridDim.z : nall;
    const int k0 = SHARE ? (int)blockIdx.z * share : 0;
    const int nown = SHARE ? min(share, nall - k0) : nall;
    if (SHARE && nown < 1) return;  // uniform over the block
    // thread (g, k): group g's lines, omega k0 + k; as many groups as fit the block, and no more than
    // there are lines; no padding between groups (a warp may hold the end of one and the start of the next)
    const int G = SHARE ? min(60, (int)blockDim.x / nown) : Gall;
    const int g = t / nown, k = t - g * nown;
    const bool own = g < G;
    {
        const float4* gb = reinterpret_cast<const float4*>(a.band + (long)p * W * W);
        float4* sb4 = reinterpret_cast<float4*>(sband);
        for (int q = t; q < (W * W) / 2; q += blockDim.x) sb4[q] = gb[q];
        for (int q = t; q < nr; q += blockDim.x) sfc0[q] = a.fcut0[(long)p * nr + q];
    }
    const float nxh = (float)(bd.nx / 2);
    const int offW = bd.off * W + bd.off;
    const float* ctfp = a.ctf ? a.ctf + (long)p * W * W : nullptr;
    const float* tfc = a.tfcut + (long)p * a.tfcut_pstride;
    const float womega = __fmul_rn(a.step, (float)(SHARE ? k0 + k : k));
    const int nwarps = blockDim.x >> 5;

    for (int v = blockIdx.x; v < a.V; v += gridDim.x) {
        float pr1 = 0.f, pr2 = 0.f, c1 = 0.f, c2 = 0.f;
        float qr1 = 0.f, qr2 = 0.f, d1 = 0.f, d2 = 0.f;  // HALF: of omega k + nomega / 2
        for (int i = 0; i < a.T; ++i) {
            __syncthreads();
            const float2* al = a.alpha + ((long)v * a.T + i) * 60;
            if (t < 32) {  // the valid lines, in order
                int n = 0;
                for (int h = 0; h < 2; ++h) {
                    const int j = 32 * h + t;
                    const float2 aa = j < 60 ? al[j] : make_float2(1000.f, 1000.f);
                    const bool ok = aa.x < 999.0f && aa.y < 999.0f;
                    const unsigned m = __ballot_sync(0xffffffffu, ok);
                    if (ok) {
                        const int at = n + __popc(m & ((1u << t) - 1u));
                        salpha[at] = aa.x;
                        sjl[at] = j;
                    }
                    n += __popc(m);
                }
                if (t == 0) *snv = n;
            }
            const float2* tb = a.tband + (long)i * W * W;
            const float* fct = tfc + (long)i * nr;
            for (int q = t; q < 60 * nr; q += blockDim.x) {
                int j = q / nr, iq = q - j * nr;
                float2 aa = al[j];
                float4 e = make_float4(0.f, 0.f, -1.0f, sfc0[iq]);
                if (aa.x < 999.0f && aa.y < 999.0f) {
                    float re, im;
                    tmpl_sample(tb, ctfp, W, offW, nxh, aa.y, (float)(minR + iq), K.d2r, &re, &im);
                    float amp = sqrtf(re * re + im * im);
                    if (amp >= fct[iq]) { e.x = re; e.y = im; e.z = 0.5f * amp; }
                }
                sline[q] = e;
            }
            __syncthreads();
            const int nv = *snv;
            for (int jj = own ? g : nv; jj < nv; jj += G) {
                const float al1 = salpha[jj];
                const float ang = __fmul_rn(__fsub_rn(al1, womega), K.d2r);
                float sn, cs;
                sincosf(ang, &sn, &cs);
                const float2 csn = make_float2(cs, sn);
                const float4* sl = sline + sjl[jj] * nr;
                float2 acc = make_float2(0.f, 0.f), acd = make_float2(0.f, 0.f);  // (sum diff*w, sum w) of this line
                for (int q0 = 0; q0 < nr; q0 += 32) {
                    const int q1 = min(nr, q0 + 32);
                    unsigned near = 0u, bit = 1u;  // HALF: radii whose amplitude is within the margin of its cut
#pragma unroll 8
                    for (int iq = q0; iq < q1; ++iq, bit <<= 1) {
                        const float4 e = sl[iq];
                        if (e.z < 0.0f) continue;
                        const OmegaTerm u = omega_sample(sband, W, offW, (float)(minR + iq), csn, nxh, e.z);
                        // the particle's cut as a select: ~70 % of the lanes pass it, so a
                        // branch would run both sides anyway
                        const float2 pd = __fmul2_rn(u.z, make_float2(e.x, e.y));
                        const float2 pc = __fmul2_rn(u.z, make_float2(e.y, -e.x));
                        const float d = angle_between_est(pc.x + pc.y, pd.x + pd.y, K.pi);
                        const float2 na = __ffma2_rn(make_float2(d, 1.0f), make_float2(u.w, u.w), acc);
                        const bool ok = u.amp >= e.w;
                        acc.x = ok ? na.x : acc.x;
                        acc.y = ok ? na.y : acc.y;
                        if constexpr (HALF) {
                            // conj z: (zx ey + zy ex, zx ex - zy ey)
                            const float dc = angle_between_est(pc.x - pc.y, pd.x - pd.y, K.pi);
                            const bool nr_cut = fabsf(u.amp - e.w) <= (LARGE ? K.margin : PAIR_MARGIN) * e.w;
                            const float2 nc = __ffma2_rn(make_float2(dc, 1.0f), make_float2(u.w, u.w), acd);
                            near |= nr_cut ? bit : 0u;
                            acd.x = ok && !nr_cut ? nc.x : acd.x;
                            acd.y = ok && !nr_cut ? nc.y : acd.y;
                        }
                    }
                    if constexpr (HALF) {
                        if (near) {  // (about one radius of a lane's line in 30)
                            const float w2 = __fmul_rn(a.step, (float)(SHARE ? k0 + k + nall : k + nown));
                            float2 csn2;
                            sincosf(__fmul_rn(__fsub_rn(al1, w2), K.d2r), &csn2.y, &csn2.x);
                            do {
                                const int iq = q0 + __ffs(near) - 1;
                                near &= near - 1u;
                                const float4 e = sl[iq];
                                const OmegaTerm x = omega_sample(sband, W, offW, (float)(minR + iq), csn2, nxh, e.z);
                                const float2 xd = __fmul2_rn(x.z, make_float2(e.x, e.y));
                                const float2 xc = __fmul2_rn(x.z, make_float2(e.y, -e.x));
                                const float dx = angle_between_est(xc.x + xc.y, xd.x + xd.y, K.pi);
                                if (x.amp >= e.w) {
                                    acd.x = fmaf(dx, x.w, acd.x);
                                    acd.y += x.w;
                                }
                            } while (near);
                        }
                    }
                }
                kahan_add(pr1, c1, acc.x);
                kahan_add(pr2, c2, acc.y);
                if constexpr (HALF) {
                    kahan_add(qr1, d1, acd.x);
                    kahan_add(qr2, d2, acd.y);
                }
            }
        }
        __syncthreads();
        sred[t] = make_float2(pr1, pr2);
        if constexpr (HALF) sred[blockDim.x + t] = make_float2(qr1, qr2);
        __syncthreads();
        unsigned long long key = ~0ull;
        // the block's omegas, then those half a turn on
        for (int q = t; q < (SHARE ? (HALF ? 2 : 1) * nown : a.nomega); q += blockDim.x) {
            const int o = SHARE ? (q >= nown ? k0 + q - nown + nall : k0 + q) : q;
            const float2* sr = sred + (q >= nown ? blockDim.x + q - nown : q);
            float s1 = 0.f, s2 = 0.f;
            for (int gg = 0; gg < G; ++gg) {
                s1 += sr[gg * nown].x;
                s2 += sr[gg * nown].y;
            }
            const float pr = (s2 > 1.0e-10f) ? s1 / s2 * K.r2d : 999.0f;
            const int base = __float_as_int(a.views[(long)v * 4 + 2]);
            if (a.pr_array) a.pr_array[(long)p * a.per + base + o] = pr;
            const unsigned long long kk = ((unsigned long long)__float_as_uint(pr) << 32) | (unsigned)(base + o);
            key = kk < key ? kk : key;
        }
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
            key = other < key ? other : key;
        }
        if ((t & 31) == 0) skey[t >> 5] = key;
        __syncthreads();
        if (t < 32) {
            key = (t < nwarps) ? skey[t] : ~0ull;
            for (int o = 16; o > 0; o >>= 1) {
                unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
                key = other < key ? other : key;
            }
            if (t == 0) atomicMin(a.best + p, key);
        }
    }
}

// cal_crosslin_PR.f90:2-71 for the 11 candidates of each particle; the candidate
// origin shift (img2d_FT_centshift.f90) is applied to each bilinear tap, which is the
// same per-pixel arithmetic as shifting the whole transform first.
__global__ void __launch_bounds__(512) k_pr_single(PrSingleArgs a, Consts K) {
    __shared__ double sh[2][32];
    __shared__ float sline[4][60];  // cos, sin of the particle line; cos, sin of the template line
    __shared__ int svalid[60];
    const Band bd = a.bd;
    const int W = bd.W, nr = bd.nr, minR = bd.min_r, nx = bd.nx;
    const int c = blockIdx.x, p = blockIdx.y;
    if (a.ncount && c >= a.ncount[p]) return;  // padding slot (whole block)
    const float* cd = a.cand + ((long)p * a.ncand + c) * 5;
    const float nxh = (float)(nx / 2);
    const float xs = __fadd_rn(cd[3], nxh), ys = __fadd_rn(cd[4], nxh);
    const int offW = bd.off * W + bd.off;
    const float2* pb = a.band + (long)p * W * W;
    const float* ctfp = a.ctf ? a.ctf + (long)p * W * W : nullptr;
    const float* fc0 = a.fcut0 + (long)p * nr;
    const float* tfc = a.tfcut + (long)p * a.tfcut_pstride;
    const float twopi = __fmul_rn(2.0f, K.pi);
    float h1 = 0.f, l1 = 0.f, h2 = 0.f, l2 = 0.f;  // per-thread sums as TwoSum pairs
    for (int i = 0; i < a.T; ++i) {
        const float2* al = a.alpha + (((long)p * a.ncand + c) * a.T + i) * 60;
        const float2* tb = a.tband + (long)i * W * W;
        const float* fct = tfc + (long)i * nr;
        // the two in-plane directions of each common line, once per line
        __syncthreads();
        if (threadIdx.x < 60) {
            const float2 aa = al[threadIdx.x];
            const bool ok = aa.x < 999.0f && aa.y < 999.0f;
            svalid[threadIdx.x] = ok;
            if (ok) {
                const float a1 = __fmul_rn(aa.x, K.d2r), a2 = __fmul_rn(aa.y, K.d2r);
                sline[0][threadIdx.x] = cosf(a1);
                sline[1][threadIdx.x] = sinf(a1);
                sline[2][threadIdx.x] = cosf(a2);
                sline[3][threadIdx.x] = sinf(a2);
            }
        }
        __syncthreads();
        for (int q = threadIdx.x; q < 60 * nr; q += blockDim.x) {
            int j = q / nr, iq = q - j * nr;
            if (!svalid[j]) continue;
            const float fr = (float)(minR + iq);
            // particle sample with the candidate origin shift on each tap
            float cs = sline[0][j], sn = sline[1][j];
            float x = __fadd_rn(__fmul_rn(fr, cs), nxh), y = __fadd_rn(__fmul_rn(fr, sn), nxh);
            int lx = (int)x, ly = (int)y;
            float ax = __fsub_rn(x, (float)lx), ay = __fsub_rn(y, (float)ly);
            float tr[4], ti[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int tx = lx + (u & 1), ty = ly + (u >> 1);
                float2 vv = pb[ty * W + tx - offW];
                int hx = tx - nx / 2, ky = ty - nx / 2;
                float ph = __fdiv_rn(__fmul_rn(twopi, __fadd_rn(__fmul_rn(xs, (float)hx), __fmul_rn(ys, (float)ky))),
                                     (float)nx);
                float s, co;
                sincosf(ph, &s, &co);
                tr[u] = __fadd_rn(__fmul_rn(vv.x, co), __fmul_rn(vv.y, s));
                ti[u] = __fadd_rn(__fmul_rn(-vv.x, s), __fmul_rn(vv.y, co));
            }
            float re1 = bilerp(ax, ay, tr[0], tr[1], tr[2], tr[3]);
            float im1 = bilerp(ax, ay, ti[0], ti[1], ti[2], ti[3]);
            float re2, im2;
            tmpl_sample_cs(tb, ctfp, W, offW, nxh, sline[2][j], sline[3][j], fr, &re2, &im2);
            float amp1 = sqrtf(re1 * re1 + im1 * im1);
            float amp2 = sqrtf(re2 * re2 + im2 * im2);
            if (amp1 >= fc0[iq] && amp2 >= fct[iq]) {
                float ph1 = atan2f(im1, re1), ph2 = atan2f(im2, re2);
                float d = fabsf(ph2 - ph1);
                d = fminf(d, K.tpi - d);
                float w = 0.5f * (amp1 + amp2);
                two_sum_acc(h1, l1, d * w);
                two_sum_acc(h2, l2, w);
            }
        }
    }
    double p1 = (double)h1 + (double)l1, p2 = (double)h2 + (double)l2;
    for (int o = 16; o > 0; o >>= 1) {
        p1 += __shfl_xor_sync(0xffffffffu, p1, o);
        p2 += __shfl_xor_sync(0xffffffffu, p2, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) { sh[0][w] = p1; sh[1][w] = p2; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s1 = 0, s2 = 0;
        for (int q = 0; q < nw; ++q) { s1 += sh[0][q]; s2 += sh[1][q]; }
        if (a.part) {
            a.part[(long)p * a.ncand + c] = make_double2(s1, s2);
            return;
        }
        float f1 = (float)s1, f2 = (float)s2;
        a.pr[(long)p * a.ncand + c] = (f2 > 1.0e-10f) ? f1 / f2 * 180.0f / K.pi : 1000.0f;
    }
}

// Grouped rescoring: up to RG candidates of one particle that share a view (theta,
// phi) and differ in omega.  The template side of a term (line direction, taps, cut)
// does not depend on omega, so each (template, line, radius) sample of the templates
// is taken once and compared with the RG particle samples.  groups[g] = (particle,
// first candidate slot, count).  Every candidate sits at the particle's origin (band
// pre-shifted, templates pre-multiplied by the particle's CTF), and the per-term
// arithmetic is the exhaustive scorer's (angle_between, Kahan sums per thread), so its
// values match k_pr_omega's.
constexpr int RG = 4;
__global__ void __launch_bounds__(512) k_pr_rescore_g(PrSingleArgs a, const int4* __restrict__ groups, Consts K) {
    extern __shared__ float rsm[];
    __shared__ double sh[2 * RG][32];
    const Band bd = a.bd;
    const int W = bd.W, nr = bd.nr, minR = bd.min_r, nx = bd.nx, T = a.T;
    const int4 gr = groups[blockIdx.x];
    const int p = gr.x, c0 = gr.y, m = gr.z;
    float* spl = rsm;                          // [RG][T][60][2]: cos, sin of the particle lines
    float* stl = spl + (long)RG * T * 120;     // [T][60][2]: cos, sin of the template lines
    float* sfc = stl + (long)T * 120;          // [T + 1][nr]: template cuts, then the particle's
    int* sval = reinterpret_cast<int*>(sfc + (long)(T + 1) * nr);  // [T][60]
    for (int q = threadIdx.x; q < T * 60; q += blockDim.x) {
        const float2 aa = a.alpha[((long)p * a.ncand + c0) * T * 60 + q];
        const bool ok = aa.x < 999.0f && aa.y < 999.0f;
        sval[q] = ok;
        if (ok) {
            const float a2 = __fmul_rn(aa.y, K.d2r);
            stl[2 * q] = cosf(a2);
            stl[2 * q + 1] = sinf(a2);
        }
    }
    for (int q = threadIdx.x; q < m * T * 60; q += blockDim.x) {
        const int g = q / (T * 60), r = q - g * T * 60;
        const float2 aa = a.alpha[((long)p * a.ncand + c0 + g) * T * 60 + r];
        const float a1 = __fmul_rn(aa.x, K.d2r);
        spl[2 * q] = cosf(a1);
        spl[2 * q + 1] = sinf(a1);
    }
    const float* tfc = a.tfcut + (long)p * a.tfcut_pstride;
    for (int q = threadIdx.x; q < T * nr; q += blockDim.x) sfc[q] = tfc[q];
    for (int q = threadIdx.x; q < nr; q += blockDim.x) sfc[T * nr + q] = a.fcut0[(long)p * nr + q];
    __syncthreads();
    const float nxh = (float)(nx / 2);
    const int offW = bd.off * W + bd.off;
    const float4* sb = a.sband + (long)p * W * W;
    const float4* tbc0 = a.tbandc ? a.tbandc + (long)p * T * W * W : nullptr;
    const float* ctfp = a.ctf ? a.ctf + (long)p * W * W : nullptr;
    const int per_t = 60 * nr;
    float f1[RG], f2[RG], k1[RG], k2[RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) { f1[g] = 0.f; f2[g] = 0.f; k1[g] = 0.f; k2[g] = 0.f; }
    // (template i, line j, radius iq) of the flat index q = (i * 60 + j) * nr + iq, advanced
    // by blockDim.x per iteration without integer divisions
    const int step_j = (int)blockDim.x / nr, step_iq = (int)blockDim.x - step_j * nr;
    int i = (int)threadIdx.x / per_t, j = ((int)threadIdx.x - i * per_t) / nr;
    int iq = (int)threadIdx.x - i * per_t - j * nr;
    auto advance = [&]() {
        iq += step_iq;
        j += step_j;
        if (iq >= nr) { iq -= nr; ++j; }
        while (j >= 60) { j -= 60; ++i; }
    };
    for (int q = threadIdx.x; q < T * per_t; q += blockDim.x, advance()) {
        const int lj = i * 60 + j;
        if (!sval[lj]) continue;
        const float fr = (float)(minR + iq);
        float re2, im2;
        if (tbc0)
            tmpl_sample_pairs(tbc0 + (long)i * W * W, W, offW, nxh, stl[2 * lj], stl[2 * lj + 1], fr, &re2, &im2);
        else
            tmpl_sample_cs(a.tband + (long)i * W * W, ctfp, W, offW, nxh, stl[2 * lj], stl[2 * lj + 1], fr, &re2,
                           &im2);
        const float amp2 = sqrtf(re2 * re2 + im2 * im2);
        if (!(amp2 >= sfc[i * nr + iq])) continue;
        const float cut1 = sfc[T * nr + iq];
#pragma unroll
        for (int g = 0; g < RG; ++g) {
            if (g >= m) break;
            const float cs = spl[2 * ((long)g * T * 60 + lj)], sn = spl[2 * ((long)g * T * 60 + lj) + 1];
            const float x = __fadd_rn(__fmul_rn(fr, cs), nxh), y = __fadd_rn(__fmul_rn(fr, sn), nxh);
            const int lx = (int)x, ly = (int)y;
            const float ax = __fsub_rn(x, (float)lx), ay = __fsub_rn(y, (float)ly);
            const int b0 = ly * W + lx - offW;
            const float4 r0 = sb[b0], r1 = sb[b0 + W];  // (tap, right tap) of rows y, y + 1
            const float2 t00 = make_float2(r0.x, r0.y), t10 = make_float2(r0.z, r0.w);
            const float2 t01 = make_float2(r1.x, r1.y), t11 = make_float2(r1.z, r1.w);
            const float re1 = bilerp(ax, ay, t00.x, t10.x, t01.x, t11.x);
            const float im1 = bilerp(ax, ay, t00.y, t10.y, t01.y, t11.y);
            const float amp1 = sqrtf(re1 * re1 + im1 * im1);
            if (amp1 >= cut1) {
                const float d = angle_between(re1 * im2 - im1 * re2, re1 * re2 + im1 * im2, K.pi);
                const float w = 0.5f * (amp1 + amp2);
                kahan_add(f1[g], k1[g], d * w);
                kahan_add(f2[g], k2[g], w);
            }
        }
    }
    double sums[2 * RG];
#pragma unroll
    for (int g = 0; g < RG; ++g) {
        sums[2 * g] = (double)f1[g];
        sums[2 * g + 1] = (double)f2[g];
    }
    block_sums<2 * RG>(sums, sh);
    if (threadIdx.x < m) {
        const int g = threadIdx.x;
        const float g1 = (float)sh[2 * g][0], g2 = (float)sh[2 * g + 1][0];
        a.pr[(long)p * a.ncand + c0 + g] = (g2 > 1.0e-10f) ? g1 / g2 * 180.0f / K.pi : 1000.0f;
    }
}

// Grouped rescoring with the particle's shifted band in shared memory.  The groups, the
// tables and the template side are k_pr_rescore_g's; the particle side reads its four
// taps from a [W][SP] float2 copy of the band in shared memory (SP = the smallest pitch
// >= W that is 3 mod 16: 8-byte taps of a line of radii fall on distinct bank pairs
// for vertical lines and spread over 4-8 for diagonal ones) instead of 16-byte
// pixel pairs from L1, and its per-term arithmetic is k_pr_omega's in packed FP32x2
// operations, so a term has the value the exhaustive search gives it.  One block of
// RS_THREADS threads per SM (the band is 136 KB at W = 130).
// A two-phase variant (per template: the template samples that pass their cut compacted
// into a shared-memory list by a block-wide scan, then the candidates over the list with
// full warps) was built and measured 1.7x slower (4.72 against 2.79 ms for the four
// launches of the profile case): its four barriers per template leave the template
// samples' L2 latency exposed with one block per SM, where the flat loop overlaps it.
// Measured alternatives of the flat loop on the same 256-particle workload (rescoring
// time, one lane): the candidate loop with a run-time count and branches on the cuts
// 1.12x, a per-warp queue of the samples that pass the template cut (full warps in the
// candidate loop, but a longer shared-memory dependency chain) 1.36x, the template taps
// fetched one iteration ahead 1.12x (no gain: not latency-bound), 768 threads 1.07x, 512
// threads 1.34x, branch-free items or two items per iteration 1.07x.
// The sums at the end: 10 us of a block's 90 as a butterfly and a serial sum per candidate (FP64
// pipe), 4 so (block_sums): 443 -> 418 us a launch of 760 groups.
constexpr int RS_THREADS = 1024;
__host__ __device__ inline int rescore_pitch(int W) { return W + ((3 - W % 16) + 16) % 16; }
__global__ void __launch_bounds__(RS_THREADS, 1) k_pr_rescore_s(PrSingleArgs a, const int4* __restrict__ groups,
                                                                  Consts K) {
    extern __shared__ __align__(16) float rsm[];
    __shared__ double sh[2 * RG][32];
    const Band bd = a.bd;
    const int W = bd.W, nr = bd.nr, minR = bd.min_r, nx = bd.nx, T = a.T;
    const int SP = rescore_pitch(W);
    const int4 gr = groups[blockIdx.x];
    const int p = gr.x, c0 = gr.y, m = gr.z;
    float2* sbd = reinterpret_cast<float2*>(rsm);   // [W][SP] shifted particle band
    float* spl = rsm + 2L * W * SP;                 // [RG][T][60][2]: cos, sin of the particle lines
    float* stl = spl + (long)RG * T * 120;          // [T][60][2]: cos, sin of the template lines
    float* sfc = stl + (long)T * 120;               // [T + 1][nr]: template cuts, then the particle's
    int* sval = reinterpret_cast<int*>(sfc + (long)(T + 1) * nr);  // [T][60]
    const float4* sb = a.sband + (long)p * W * W;
    for (int row = threadIdx.x >> 5; row < W; row += RS_THREADS / 32)
        for (int col = threadIdx.x & 31; col < W; col += 32) {
            const float4 v = sb[(long)row * W + col];
            sbd[row * SP + col] = make_float2(v.x, v.y);
        }
    // line directions from the view table, as k_pr_omega computes them: the template's
    // cos/sin of alpha2, the particle's sincos of (alpha1 - omega) for each candidate
    const int* co = a.corient + (long)p * a.ncand + c0;
    const float2* va = a.valpha + (long)(co[0] / a.nom) * T * 60;
    for (int q = threadIdx.x; q < T * 60; q += RS_THREADS) {
        const float2 aa = va[q];
        const bool ok = aa.x < 999.0f && aa.y < 999.0f;
        sval[q] = ok;
        if (ok) {
            const float a2 = __fmul_rn(aa.y, K.d2r);
            stl[2 * q] = cosf(a2);
            stl[2 * q + 1] = sinf(a2);
        }
    }
    for (int q = threadIdx.x; q < m * T * 60; q += RS_THREADS) {
        const int g = q / (T * 60), r = q - g * T * 60;
        const float2 aa = va[r];
        const float womega = __fmul_rn(a.step, (float)(co[g] % a.nom));
        const float ang = __fmul_rn(__fsub_rn(aa.x, womega), K.d2r);
        float sn, cs;
        sincosf(ang, &sn, &cs);
        spl[2 * q] = cs;
        spl[2 * q + 1] = sn;
    }
    const float* tfc = a.tfcut + (long)p * a.tfcut_pstride;
    for (int q = threadIdx.x; q < T * nr; q += RS_THREADS) sfc[q] = tfc[q];
    for (int q = threadIdx.x; q < nr; q += RS_THREADS) sfc[T * nr + q] = a.fcut0[(long)p * nr + q];
    __syncthreads();
    const float nxh = (float)(nx / 2);
    const int offW = bd.off * W + bd.off, offS = bd.off * SP + bd.off;
    const float4* tbc0 = a.tbandc ? a.tbandc + (long)p * T * W * W : nullptr;
    const float* ctfp = a.ctf ? a.ctf + (long)p * W * W : nullptr;
    const int per_t = 60 * nr;
    const int step_j = RS_THREADS / nr, step_iq = RS_THREADS - step_j * nr;
    int i = (int)threadIdx.x / per_t, j = ((int)threadIdx.x - i * per_t) / nr;
    int iq = (int)threadIdx.x - i * per_t - j * nr;
    auto advance = [&]() {
        iq += step_iq;
        j += step_j;
        if (iq >= nr) { iq -= nr; ++j; }
        while (j >= 60) { j -= 60; ++i; }
    };
    const float2 nxh2 = make_float2(nxh, nxh);
    // The group's candidate count M is a compile-time constant of each instance of the
    // loop, so the M candidates' terms of one template sample are independent chains that
    // the compiler interleaves; the two amplitude cuts are selects, not branches (with
    // ~70 % of the samples passing each cut, a warp runs both sides of such a branch
    // anyway).  A term that fails a cut leaves the sums unchanged.
    auto run = [&](auto mc) {
        constexpr int M = decltype(mc)::value;
        // (PR numerator, weight) sums: per thread a plain FP32 pair over its ~40 terms of a
        // candidate (like k_pr_omega's per-line partials), then FP64 across the block
        float2 fs[M];
#pragma unroll
        for (int g = 0; g < M; ++g) fs[g] = make_float2(0.f, 0.f);
        for (int q = threadIdx.x; q < T * per_t; q += RS_THREADS, advance()) {
            const int lj = i * 60 + j;
            if (!sval[lj]) continue;
            const float fr = (float)(minR + iq);
            float re2, im2;
            if (tbc0)
                tmpl_sample_pairs(tbc0 + (long)i * W * W, W, offW, nxh, stl[2 * lj], stl[2 * lj + 1], fr, &re2,
                                  &im2);
            else
                tmpl_sample_cs(a.tband + (long)i * W * W, ctfp, W, offW, nxh, stl[2 * lj], stl[2 * lj + 1], fr,
                               &re2, &im2);
            const float amp2 = sqrtf(re2 * re2 + im2 * im2);
            const bool ok2 = amp2 >= sfc[i * nr + iq];
            const float cut1 = sfc[T * nr + iq];
            const float2 fr2 = make_float2(fr, fr), e2 = make_float2(re2, im2), e2c = make_float2(im2, -re2);
            const float half2 = 0.5f * amp2;
            const float2 m1 = make_float2(-1.f, -1.f);
#pragma unroll
            for (int g = 0; g < M; ++g) {
                // k_pr_omega's per-term arithmetic: position by FMA, bilinear as lerps on
                // (re, im) pairs, amplitude sq * rsqrt(sq), weight 0.5 amp1 + 0.5 amp2
                const float2 cs = *reinterpret_cast<const float2*>(&spl[2 * ((long)g * T * 60 + lj)]);
                const float2 xy = __ffma2_rn(fr2, cs, nxh2);
                const int lx = (int)xy.x, ly = (int)xy.y;
                const float2 f = __fadd2_rn(xy, make_float2(-(float)lx, -(float)ly));
                const float2* tp = sbd + (ly * SP + lx - offS);
                const float2 t00 = tp[0], t10 = tp[1], t01 = tp[SP], t11 = tp[SP + 1];
                const float2 ax2 = make_float2(f.x, f.x), ay2 = make_float2(f.y, f.y);
                const float2 v0 = __ffma2_rn(ax2, __ffma2_rn(t00, m1, t10), t00);
                const float2 v1 = __ffma2_rn(ax2, __ffma2_rn(t01, m1, t11), t01);
                const float2 z = __ffma2_rn(ay2, __ffma2_rn(v0, m1, v1), v0);
                const float2 zz = __fmul2_rn(z, z);
                const float sq = zz.x + zz.y;
                const float amp1 = sq * rsqrtf(sq);  // NaN for 0: fails the cut
                const float2 pd = __fmul2_rn(z, e2);
                const float2 pc = __fmul2_rn(z, e2c);
                const float d = angle_between_est(pc.x + pc.y, pd.x + pd.y, K.pi);
                const float w = fmaf(0.5f, amp1, half2);
                const float2 nf = __ffma2_rn(make_float2(d, 1.0f), make_float2(w, w), fs[g]);
                const bool ok = ok2 && amp1 >= cut1;
                fs[g].x = ok ? nf.x : fs[g].x;
                fs[g].y = ok ? nf.y : fs[g].y;
            }
        }
        constexpr int N = M == 1 ? 2 : M == 2 ? 4 : 8;
        double sums[N];
#pragma unroll
        for (int g = 0; g < N / 2; ++g) {
            sums[2 * g] = g < M ? (double)fs[g < M ? g : 0].x : 0.0;
            sums[2 * g + 1] = g < M ? (double)fs[g < M ? g : 0].y : 0.0;
        }
        block_sums<N>(sums, sh);
    };
    switch (m) {
        case 1: run(std::integral_constant<int, 1>()); break;
        case 2: run(std::integral_constant<int, 2>()); break;
        case 3: run(std::integral_constant<int, 3>()); break;
        default: run(std::integral_constant<int, RG>()); break;
    }
    if (threadIdx.x < m) {
        const int g = threadIdx.x;
        const float g1 = (float)sh[2 * g][0], g2 = (float)sh[2 * g + 1][0];
        a.pr[(long)p * a.ncand + c0 + g] = (g2 > 1.0e-10f) ? g1 / g2 * 180.0f / K.pi : 1000.0f;
    }
}

// A refinement step's candidates: block (candidate, particle, split) scores its share of the
// templates.  cal_crosslin_PR.f90's terms as k_pr_single has them, arranged for the work they
// repeat: the band is shifted to the candidate's origin once per pixel into shared memory (four
// sincos a term before), the valid lines of the templates are listed with their directions, the
// templates come multiplied by the CTF, and the phase difference is one arctangent of the cross
// and dot products (two and a fold before; error 1e-7 rad either way).  Sums are TwoSum pairs per
// thread as there, FP64 across the block and the splits.  Issue-bound.  64 particles of box
// 256, 20 templates: 861 us a step by k_pr_single, 468 so.
__device__ __forceinline__ float2 shifted_pixel(const float2* band, int m, int W, int off, int nx, float xs,
                                                float ys, float twopi);
constexpr int RF_THREADS = 1024;
__global__ void __launch_bounds__(RF_THREADS, 1) k_pr_refine(PrSingleArgs a, Consts K, double2* __restrict__ part) {
    extern __shared__ __align__(16) float rsm[];
    __shared__ double sh[2][32];
    __shared__ int snv;
    const Band bd = a.bd;
    const int W = bd.W, nr = bd.nr, minR = bd.min_r, nx = bd.nx;
    const int SP = rescore_pitch(W);
    const int c = blockIdx.x, p = blockIdx.y, S = gridDim.z;
    const int t0 = a.T * (int)blockIdx.z / S, t1 = a.T * ((int)blockIdx.z + 1) / S, nt = t1 - t0;
    float2* sbd = reinterpret_cast<float2*>(rsm);                        // [W][SP] shifted particle band
    float4* sln = reinterpret_cast<float4*>(rsm + ((2L * W * SP + 3) & ~3L));  // listed lines: cos, sin of particle, of template
    int* stm = reinterpret_cast<int*>(sln + nt * 60);                    // and their templates (of this share)
    float* sfc = reinterpret_cast<float*>(stm + nt * 60);                // [nt + 1][nr]: template cuts, the particle's
    const float* cd = a.cand + ((long)p * a.ncand + c) * 5;
    const float nxh = (float)(nx / 2);
    const float xs = __fadd_rn(cd[3], nxh), ys = __fadd_rn(cd[4], nxh);
    const float2* pb = a.band + (long)p * W * W;
    const float twopi = __fmul_rn(2.0f, K.pi);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {  // the valid lines in order
        const float2* al = a.alpha + (((long)p * a.ncand + c) * a.T + t0) * 60;
        int n = 0;
        for (int q0 = 0; q0 < nt * 60; q0 += 32) {
            const int q = q0 + lane;
            const float2 aa = q < nt * 60 ? al[q] : make_float2(1000.f, 1000.f);
            const bool ok = aa.x < 999.0f && aa.y < 999.0f;
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const int at = n + __popc(m & ((1u << lane) - 1u));
                const float a1 = __fmul_rn(aa.x, K.d2r), a2 = __fmul_rn(aa.y, K.d2r);
                sln[at] = make_float4(cosf(a1), sinf(a1), cosf(a2), sinf(a2));
                stm[at] = q / 60;
            }
            n += __popc(m);
        }
        if (lane == 0) snv = n;
    } else {
        for (int row = warp - 1; row < W; row += RF_THREADS / 32 - 1)
            for (int col = lane; col < W; col += 32)
                sbd[row * SP + col] = shifted_pixel(pb, row * W + col, W, bd.off, nx, xs, ys, twopi);
    }
    const float* tfc = a.tfcut + (long)p * a.tfcut_pstride + (long)t0 * nr;
    for (int q = threadIdx.x; q < nt * nr; q += RF_THREADS) sfc[q] = tfc[q];
    for (int q = threadIdx.x; q < nr; q += RF_THREADS) sfc[nt * nr + q] = a.fcut0[(long)p * nr + q];
    __syncthreads();
    const int offW = bd.off * W + bd.off, offS = bd.off * SP + bd.off;
    const float4* tbc = a.tbandc ? a.tbandc + ((long)p * a.T + t0) * W * W : nullptr;
    const int total = snv * nr;
    const int step_l = RF_THREADS / nr, step_iq = RF_THREADS - step_l * nr;
    int l = (int)threadIdx.x / nr, iq = (int)threadIdx.x - l * nr;
    float h1 = 0.f, l1 = 0.f, h2 = 0.f, l2 = 0.f;  // per-thread sums as TwoSum pairs
    for (int q = threadIdx.x; q < total; q += RF_THREADS) {
        const float4 ln = sln[l];
        const int i = stm[l];
        const float fr = (float)(minR + iq);
        float re2, im2;
        if (tbc)
            tmpl_sample_pairs(tbc + (long)i * W * W, W, offW, nxh, ln.z, ln.w, fr, &re2, &im2);
        else
            tmpl_sample_cs(a.tband + (long)(t0 + i) * W * W, nullptr, W, offW, nxh, ln.z, ln.w, fr, &re2, &im2);
        const float x = __fadd_rn(__fmul_rn(fr, ln.x), nxh), y = __fadd_rn(__fmul_rn(fr, ln.y), nxh);
        const int lx = (int)x, ly = (int)y;
        const float ax = __fsub_rn(x, (float)lx), ay = __fsub_rn(y, (float)ly);
        const float2* tp = sbd + (ly * SP + lx - offS);
        const float2 t00 = tp[0], t10 = tp[1], t01 = tp[SP], t11 = tp[SP + 1];
        const float re1 = bilerp(ax, ay, t00.x, t10.x, t01.x, t11.x);
        const float im1 = bilerp(ax, ay, t00.y, t10.y, t01.y, t11.y);
        const float amp1 = sqrtf(re1 * re1 + im1 * im1);
        const float amp2 = sqrtf(re2 * re2 + im2 * im2);
        if (amp1 >= sfc[nt * nr + iq] && amp2 >= sfc[i * nr + iq]) {
            const float d = atan2f(fabsf(re1 * im2 - im1 * re2), re1 * re2 + im1 * im2);
            const float w = 0.5f * (amp1 + amp2);
            two_sum_acc(h1, l1, d * w);
            two_sum_acc(h2, l2, w);
        }
        iq += step_iq;
        l += step_l;
        if (iq >= nr) { iq -= nr; ++l; }
    }
    double sums[2] = {(double)h1 + (double)l1, (double)h2 + (double)l2};
    block_sums<2>(sums, sh);
    if (threadIdx.x == 0) part[((long)p * a.ncand + c) * S + blockIdx.z] = make_double2(sh[0][0], sh[1][0]);
}

// The particle transform shifted to the origin its candidates share (cand[p][0][3..4]):
// per pixel the same phase rotation k_pr_single applies to each bilinear tap
// (img2d_FT_centshift.f90), computed once per pixel instead of once per tap.
// Stored as pairs: out[p][m] = (pixel m, its right neighbour m + 1; zero past the row's
// end), so a bilinear sample reads two aligned 16-byte pairs instead of four taps.
__device__ __forceinline__ float2 shifted_pixel(const float2* band, int m, int W, int off, int nx, float xs,
                                                float ys, float twopi) {
    const int by = m / W, bx = m - by * W;
    const int hx = bx + off - nx / 2, ky = by + off - nx / 2;
    const float2 vv = band[m];
    float ph = __fdiv_rn(__fmul_rn(twopi, __fadd_rn(__fmul_rn(xs, (float)hx), __fmul_rn(ys, (float)ky))),
                         (float)nx);
    float s, co;
    sincosf(ph, &s, &co);
    return make_float2(__fadd_rn(__fmul_rn(vv.x, co), __fmul_rn(vv.y, s)),
                       __fadd_rn(__fmul_rn(-vv.x, s), __fmul_rn(vv.y, co)));
}
__global__ void k_shift_band(const float2* __restrict__ band, const float* __restrict__ cand, int ncand, Band bd,
                             Consts K, float4* __restrict__ out) {
    const int W = bd.W, nx = bd.nx, p = blockIdx.y;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= W * W) return;
    const float* cd = cand + (long)p * ncand * 5;
    const float nxh = (float)(nx / 2);
    const float xs = __fadd_rn(cd[3], nxh), ys = __fadd_rn(cd[4], nxh);
    const float twopi = __fmul_rn(2.0f, K.pi);
    const float2* b = band + (long)p * W * W;
    const float2 v0 = shifted_pixel(b, m, W, bd.off, nx, xs, ys, twopi);
    const float2 v1 = (m % W) + 1 < W ? shifted_pixel(b, m + 1, W, bd.off, nx, xs, ys, twopi) : make_float2(0.f, 0.f);
    out[(long)p * W * W + m] = make_float4(v0.x, v0.y, v1.x, v1.y);
}

// reconstruct.f90:103-145: rotate each half-plane sample, apply the operators,
// fold to z >= 0 and splat (a*ctf, b*ctf*signz, ctf^2) trilinearly.  One thread per
// (operator, sample), consecutive threads on consecutive samples of one operator: the
// samples run along hx, so a warp's splats land on neighbouring voxels and its float4
// vector reductions share L2 sectors (the three sums of a voxel are one reduction).
// Bound by those reductions in L2 (8 a splat).  All 60 operators of a particle cost 12.9 us at
// maxR 64.  Twelve of them (the rotations that permute and negate the axes, the tetrahedral
// group) take the voxel grid to itself, and a trilinear splat commutes with those: so the
// particles of a call are splatted with one operator of each of their five cosets, 1.1 us a
// particle, and the box is summed over the twelve once (k_sym_octant, k_sym_add: 18 us).  The
// plane z = 0 of the half box is apart: which of v and -v a sample lands on there depends on
// the sign of its own z, which the sums over the cyclic permutations no longer hold.  The half
// turns about the axes keep it: after the fold a sample at (x, y, z > 0) is also one at
// (-x, -y, z) and its conjugate at (-x, y, z) and (x, -y, z); one at z = 0 exactly is not folded,
// so at all four it is itself.  So the plane's cells are splatted under one operator of each
// coset of those (fifteen; k_insert_plane0, only the samples within 1 of the plane) and summed
// over the four (k_sym_plane0).
__device__ __forceinline__ void mv3_rn(const float* m, const float* v, float* o) {
    float t0 = __fmul_rn(m[0], v[0]); t0 = __fadd_rn(t0, __fmul_rn(m[1], v[1])); t0 = __fadd_rn(t0, __fmul_rn(m[2], v[2]));
    float t1 = __fmul_rn(m[3], v[0]); t1 = __fadd_rn(t1, __fmul_rn(m[4], v[1])); t1 = __fadd_rn(t1, __fmul_rn(m[5], v[2]));
    float t2 = __fmul_rn(m[6], v[0]); t2 = __fadd_rn(t2, __fmul_rn(m[7], v[1])); t2 = __fadd_rn(t2, __fmul_rn(m[8], v[2]));
    o[0] = t0; o[1] = t1; o[2] = t2;
}

// PLANE0: only the cells of lz = 0, into a.acc as two planes: of samples off the plane z = 0,
// and (a.acc + AW AW) of samples exactly on it
template <bool PLANE0>
__device__ __forceinline__ void splat(const InsertArgs& a, int p, int k, int2 hk) {
    const Band bd = a.bd;
    const int W = bd.W, R = bd.max_r;
    const float* rot = a.rot + p * 9;
    float xv[3] = {(float)hk.x, (float)hk.y, 0.0f}, x00[3], x0[3];
    mv3_rn(rot, xv, x00);
    mv3_rn(a.ops + k * 9, x00, x0);
    float signz = 1.0f;
    if (x0[2] < 0.0f) { x0[0] = -x0[0]; x0[1] = -x0[1]; x0[2] = -x0[2]; signz = -1.0f; }
    const float zfold = x0[2];
    x0[0] = __fadd_rn(x0[0], a.off_xy);
    x0[1] = __fadd_rn(x0[1], a.off_xy);
    x0[2] = __fadd_rn(x0[2], a.off_z);
    const int lx = (int)x0[0], ly = (int)x0[1], lz = (int)x0[2];
    const float ax = x0[0] - (float)lx, ay = x0[1] - (float)ly, az = x0[2] - (float)lz;
    const float bx = 1.0f - ax, by = 1.0f - ay, bz = 1.0f - az;
    float dx[8];
    dx[0] = __fmul_rn(__fmul_rn(bx, by), bz);
    dx[1] = __fmul_rn(__fmul_rn(ax, by), bz);
    dx[2] = __fmul_rn(__fmul_rn(bx, ay), bz);
    dx[3] = __fmul_rn(__fmul_rn(ax, ay), bz);
    dx[4] = __fmul_rn(__fmul_rn(bx, by), az);
    dx[5] = __fmul_rn(__fmul_rn(ax, by), az);
    dx[6] = __fmul_rn(__fmul_rn(bx, ay), az);
    dx[7] = __fmul_rn(__fmul_rn(ax, ay), az);
    const int bidx = (hk.y + R) * W + (hk.x + R);
    const float2 fv = a.band[(long)p * W * W + bidx];
    const float c = a.ctf ? a.ctf[(long)p * W * W + bidx] : 1.0f;
    const float c2 = __fmul_rn(c, c);
    const int AW = bd.AW;
    const int ix = lx - a.base_xy, iy = ly - a.base_xy, iz = lz - a.base_z;
    if (ix < 0 || iy < 0 || iz < 0 || ix > AW - 2 || iy > AW - 2 || iz > R) return;  // never taken
    if (PLANE0 && iz != 0) return;
    float4* acc = a.acc + (PLANE0 && zfold == 0.0f ? (long)AW * AW : 0L);
    const long base = ((long)iz * AW + iy) * AW + ix;
    const long offs[8] = {0, 1, AW, AW + 1, (long)AW * AW, (long)AW * AW + 1, (long)AW * AW + AW,
                          (long)AW * AW + AW + 1};
#pragma unroll
    for (int j = 0; j < (PLANE0 ? 4 : 8); ++j) {
        float va = __fmul_rn(__fmul_rn(fv.x, dx[j]), c);
        float vb = __fmul_rn(__fmul_rn(__fmul_rn(fv.y, dx[j]), c), signz);
        float vw = __fmul_rn(dx[j], c2);
        atomicAdd(acc + base + offs[j], make_float4(va, vb, vw, 0.0f));
    }
}

__global__ void __launch_bounds__(256) k_insert(InsertArgs a) {
    const int p = blockIdx.y;
    if (!a.sel[p]) return;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)a.nsamples * a.nsym) return;
    const int k = (int)(q / a.nsamples), s = (int)(q - (long)k * a.nsamples);
    splat<false>(a, p, k, a.samples[s]);
}

// One block per (operator, particle), P0_LANES threads per row ky of samples in turn: the stretch of
// hx whose rotated z, by the product of the two rotations, is within 1 (and a margin over the
// rounding the two differ by) is splatted.  Bound by the longest rows, along the plane, and the
// reductions that meet on the cells around the origin: under all 60 operators 81 us a 64-particle
// batch at maxR 64, under one of each of the fifteen cosets of the half turns about the axes 42 us
// by a thread a row, 19 by eight.
constexpr int P0_THREADS = 256, P0_LANES = 8;  // threads of a block, of a row
__global__ void __launch_bounds__(P0_THREADS) k_insert_plane0(InsertArgs a) {
    const int k = blockIdx.x, p = blockIdx.y;
    if (!a.sel[p]) return;
    const float* op = a.ops + k * 9 + 6;
    const float* rot = a.rot + p * 9;
    const float zx = op[0] * rot[0] + op[1] * rot[3] + op[2] * rot[6];
    const float zy = op[0] * rot[1] + op[1] * rot[4] + op[2] * rot[7];
    const int l = threadIdx.x % P0_LANES;
    for (int r = threadIdx.x / P0_LANES; r < 2 * a.lim + 1; r += P0_THREADS / P0_LANES) {
        const int ky = r - a.lim;
        int hmax = (int)sqrtf((float)(a.lim * a.lim - ky * ky));  // samples hx^2 + ky^2 <= lim^2
        while (hmax * hmax + ky * ky > a.lim * a.lim) --hmax;
        while ((hmax + 1) * (hmax + 1) + ky * ky <= a.lim * a.lim) ++hmax;
        const float z0 = zy * (float)ky;
        int h0 = 0, h1 = hmax;
        if (fabsf(zx) * (float)hmax > 1.0e-3f) {  // else z is z0 all along
            const float u = (-1.01f - z0) / zx, v = (1.01f - z0) / zx;
            h0 = max(0, (int)ceilf(fmaxf(fminf(u, v), -1.0e6f)));
            h1 = min(hmax, (int)floorf(fminf(fmaxf(u, v), 1.0e6f)));
        } else if (fabsf(z0) > 1.02f) {
            continue;
        }
        for (int hx = h0 + l; hx <= h1; hx += P0_LANES) splat<true>(a, p, k, make_int2(hx, ky));
    }
}

// Sums over the tetrahedral group.  F(v) of a whole box is the half box acc5 for z > 0, its
// conjugate at -v for z < 0 and acc5(v) + conj acc5(-v) on z = 0.  Over the four rotations by
// half a turn about the axes, B(v) = F(x,y,z) + F(x,-y,-z) + F(-x,y,-z) + F(-x,-y,z) has
// B = conj B under a sign change of any one axis, so the octant x, y, z >= 0 holds it:
// k_sym_octant computes it and leaves acc5 zero (each thread owns the cells it reads).  The
// three cyclic permutations of the axes give the rest: k_sym_add adds B(x,y,z) + B(y,z,x) +
// B(z,x,y), conjugated for an odd number of negative axes, to the cells z >= 1 of acc.
__device__ __forceinline__ long octant(int C, int x, int y, int z) { return ((long)z * C + y) * C + x; }
__global__ void __launch_bounds__(256) k_sym_octant(float4* __restrict__ acc5, Band bd, float4* __restrict__ oct) {
    const int C = bd.max_r + 2;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)C * C * C) return;
    const int x = (int)(q % C), y = (int)((q / C) % C), z = (int)(q / ((long)C * C));
    const long c[4] = {acc_cell(bd, x, y, z), acc_cell(bd, -x, y, z), acc_cell(bd, x, -y, z), acc_cell(bd, -x, -y, z)};
    const float4 v0 = acc5[c[0]], v1 = acc5[c[1]], v2 = acc5[c[2]], v3 = acc5[c[3]];
    float4 s;
    s.x = (v0.x + v3.x) + (v1.x + v2.x);
    s.y = (v0.y + v3.y) - (v1.y + v2.y);
    s.z = (v0.z + v3.z) + (v1.z + v2.z);
    s.w = 0.0f;
    if (z == 0) {  // F(v) + F(-v) is twice the real part
        s.x *= 2.0f;
        s.y = 0.0f;
        s.z *= 2.0f;
    }
    oct[q] = s;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc5[c[i]] = make_float4(0.f, 0.f, 0.f, 0.f);
}
__global__ void __launch_bounds__(256) k_sym_add(const float4* __restrict__ oct, Band bd, float4* __restrict__ acc) {
    const int C = bd.max_r + 2;
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (long)C * C * (C - 1)) return;
    const int x = (int)(q % C), y = (int)((q / C) % C), z = 1 + (int)(q / ((long)C * C));
    const float4 a = oct[octant(C, x, y, z)], b = oct[octant(C, y, z, x)], d = oct[octant(C, z, x, y)];
    const float sx = a.x + b.x + d.x, sy = a.y + b.y + d.y, sz = a.z + b.z + d.z;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if ((i & 1 && x == 0) || (i & 2 && y == 0)) continue;
        float4* o = acc + acc_cell(bd, i & 1 ? -x : x, i & 2 ? -y : y, z);
        float4 v = *o;
        v.x += sx;
        v.y += (i == 1 || i == 2) ? -sy : sy;
        v.z += sz;
        *o = v;
    }
}

// plane0: two planes of AW x AW (samples off and on z = 0), left zero; acc's cells of z = 0 are
// the sums over the four half turns.
__global__ void __launch_bounds__(256) k_sym_plane0(float4* __restrict__ plane0, Band bd, float4* __restrict__ acc) {
    const int C = bd.max_r + 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= C * C) return;
    const int x = q % C, y = q / C;
    const long n = (long)bd.AW * bd.AW;
    const long c[4] = {acc_cell(bd, x, y, 0), acc_cell(bd, -x, y, 0), acc_cell(bd, x, -y, 0), acc_cell(bd, -x, -y, 0)};
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) { a[i] = plane0[c[i]]; b[i] = plane0[n + c[i]]; }
#pragma unroll
    for (int i = 0; i < 4; ++i) { plane0[c[i]] = make_float4(0.f, 0.f, 0.f, 0.f); plane0[n + c[i]] = make_float4(0.f, 0.f, 0.f, 0.f); }
    // the same sums at the four cells, but for the sign of the folded ones' imaginary part
    const float bx = (b[0].x + b[3].x) + (b[1].x + b[2].x), by = (b[0].y + b[3].y) + (b[1].y + b[2].y),
                bz = (b[0].z + b[3].z) + (b[1].z + b[2].z);
    const float ax = (a[0].x + a[3].x) + (a[1].x + a[2].x), ay = (a[0].y + a[3].y) - (a[1].y + a[2].y),
                az = (a[0].z + a[3].z) + (a[1].z + a[2].z);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if ((i & 1 && x == 0) || (i & 2 && y == 0)) continue;
        float4 v = acc[c[i]];
        v.x += ax + bx;
        v.y += (i == 1 || i == 2 ? -ay : ay) + by;
        v.z += az + bz;
        acc[c[i]] = v;
    }
}

__global__ void k_fill4(float4* __restrict__ p, long n, float4 v) {
    const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) p[q] = v;
}

Consts consts() {
    Angles an = host_angles();
    Consts K;
    K.d2r = an.deg2rad;
    K.pi = an.pi;
    K.tpi = an.tpi;
    K.r2d = 180.0f / an.pi;
    K.margin = 0.0f;
    return K;
}

}  // namespace

// omega + nomega / 2 is half a turn on, and its samples are those at omega conjugated
static bool omega_half(const PrOmegaArgs& a) {
    return a.real_image && a.nomega % 2 == 0 && fabsf(a.step * (float)(a.nomega / 2) - 180.0f) < 1e-3f;
}

static int pr_omega_smem_bytes(const Band& bd, int nomega, bool half, int* threads, int* groups) {
    if (nomega < 1 || nomega > 768) return -1;
    const int nown = half ? nomega / 2 : nomega;
    // groups of lines: as many as fit 768 threads, and no more than there are lines
    const int G = std::min(60, 768 / nown), nt = (G * nown + 31) / 32 * 32;
    if (threads) *threads = nt;
    if (groups) *groups = G;
    size_t b = (size_t)bd.W * bd.W * 8 + (size_t)std::max(60 * bd.nr, nt / (half ? 1 : 2)) * 16 +
               (size_t)((bd.nr + 3) & ~3) * 4 + 32 * 8 + 64 * 4 + 64 * 4 + 16;
    return (int)b;
}

cudaError_t launch_pr_omega(const PrOmegaArgs& a, int B, cudaStream_t st) {
    int nt = 0, G = 0;
    const bool half = omega_half(a);
    int sm = pr_omega_smem_bytes(a.bd, a.nomega, half, &nt, &G);
    if (sm < 0) return cudaErrorInvalidValue;
    // A block has an SM to itself: where a block a view and particle leave SMs idle, several share a view's omegas
    // (each repeats the template's samples: 47 views of 90 omegas, one particle, 4 templates, box 64, 78 us by 47
    // blocks, 51 by 94)
    const int nall = half ? a.nomega / 2 : a.nomega;
    auto rounds = [&](int zz) {  // of a template's 60 lines over the block's groups
        const int Gz = std::min(60, nt / ((nall + zz - 1) / zz));
        return (60 + Gz - 1) / Gz;
    };
    int z = 1;
    const int sms = sm_count();
    for (int zz = 2; zz <= 8 && (long)a.V * B * zz <= sms; ++zz)
        if (rounds(zz) < rounds(z)) z = zz;
    const bool large = a.bd.nx > 256;  // (an instance of its own: a margin in a register costs 0.5 %)
    auto kern = z > 1 ? (!half ? k_pr_omega<false, true, false> : large ? k_pr_omega<true, true, true> : k_pr_omega<true, true, false>)
                      : (!half ? k_pr_omega<false, false, false> : large ? k_pr_omega<true, false, true> : k_pr_omega<true, false, false>);
    cudaError_t e = allow_smem(kern, sm);
    if (e != cudaSuccess) return e;
    Consts K = consts();
    K.margin = PAIR_MARGIN * (float)a.bd.nx / 256.0f;
    kern<<<dim3(a.V, B, z), nt, sm, st>>>(a, nall, G, K);
    return cudaGetLastError();
}

cudaError_t launch_shift_band(const float2* band, const float* cand, int ncand, const Band& bd, int B,
                              float4* out, cudaStream_t st) {
    const int n = bd.W * bd.W;
    dim3 grid((n + 255) / 256, B);
    k_shift_band<<<grid, 256, 0, st>>>(band, cand, ncand, bd, consts(), out);
    return cudaGetLastError();
}

// out[p][i] = tband[i] x ctf[p] per band pixel (the products tmpl_sample forms per tap), a pixel's CTF
// and column once for all templates.  Bound: the write of out (346 MB for 64 particles at W = 130
// and 20 templates, 51 us at the measured bandwidth).  With an index split by two 64-bit
// remainders per element 125 us, now 55.
__global__ void __launch_bounds__(256) k_tband_ctf(const float2* __restrict__ tband, int T,
                                                  const float* __restrict__ ctf, int w2, int W,
                                                  float4* __restrict__ out) {
    const int m = blockIdx.x * 256 + threadIdx.x, p = blockIdx.y;
    if (m >= w2) return;
    const float* cp = ctf + (long)p * w2 + m;
    const bool right = m % W + 1 < W;  // a right neighbour in the same row
    const float c = cp[0], c1 = right ? cp[1] : 0.f;
    float4* o = out + (long)p * T * w2 + m;
#pragma unroll 4
    for (int i = 0; i < T; ++i) {
        const float2* tb = tband + (long)i * w2 + m;
        const float2 t = tb[0];
        float2 u = make_float2(0.f, 0.f);
        if (right) {
            const float2 t1 = tb[1];
            u = make_float2(__fmul_rn(t1.x, c1), __fmul_rn(t1.y, c1));
        }
        o[(long)i * w2] = make_float4(__fmul_rn(t.x, c), __fmul_rn(t.y, c), u.x, u.y);
    }
}

cudaError_t launch_tband_ctf(const float2* tband, int T, const float* ctf, const Band& bd, int B, float4* out,
                             cudaStream_t st) {
    const int w2 = bd.W * bd.W;
    k_tband_ctf<<<dim3((w2 + 255) / 256, B), 256, 0, st>>>(tband, T, ctf, w2, bd.W, out);
    return cudaGetLastError();
}

cudaError_t launch_pr_single(const PrSingleArgs& a, int B, cudaStream_t st) {
    dim3 grid(a.ncand, B);
    k_pr_single<<<grid, 512, 0, st>>>(a, consts());
    return cudaGetLastError();
}

static size_t pr_refine_smem(const Band& bd, int nt) {
    return sizeof(float) * ((2 * (size_t)bd.W * rescore_pitch(bd.W) + 3) & ~(size_t)3) +
           (sizeof(float4) + sizeof(int)) * (size_t)nt * 60 + sizeof(float) * (size_t)(nt + 1) * bd.nr;
}
static bool pr_refine_fits(const Band& bd, int nt) { return pr_refine_smem(bd, nt) + 1024 <= 227 * 1024; }

int pr_refine_splits(const Band& bd, int T, int B, int num_sms) {
    // blocks of one SM each: the fewest rounds of them, counting the shift of the band (about a
    // seventh of 20 templates' terms) that every split repeats; 0: not even a split's lines fit
    int best = 0;
    double cost = 1e30;
    for (int S = 1; S <= std::min(T, 16); ++S) {
        if (!pr_refine_fits(bd, (T + S - 1) / S)) continue;
        const double rounds = std::ceil(11.0 * B * S / num_sms) * (1.0 / S + 0.15);
        if (rounds < cost) { cost = rounds; best = S; }
    }
    return best;
}

cudaError_t launch_pr_refine(const PrSingleArgs& a, int B, int S, double2* part, cudaStream_t st) {
    const size_t sm = pr_refine_smem(a.bd, (a.T + S - 1) / S);
    cudaError_t e = allow_smem(k_pr_refine, sm);
    if (e != cudaSuccess) return e;
    k_pr_refine<<<dim3(a.ncand, B, S), RF_THREADS, sm, st>>>(a, consts(), part);
    return cudaGetLastError();
}

cudaError_t launch_pr_rescore_groups(const PrSingleArgs& a, const int4* groups, int ngroups, cudaStream_t st) {
    if (!a.sband || ngroups < 1) return cudaErrorInvalidValue;
    const size_t sm = sizeof(float) * ((size_t)RG * a.T * 120 + (size_t)a.T * 120 + (size_t)(a.T + 1) * a.bd.nr) +
                      sizeof(int) * a.T * 60;
    // the band in shared memory where it fits beside the tables (W <= ~140 at T = 20)
    const size_t sm_s = sm + sizeof(float2) * (size_t)a.bd.W * rescore_pitch(a.bd.W);
    if (pr_rescore_shared_band(a.bd, a.T)) {
        if (!a.valpha || !a.corient || a.nom < 1) return cudaErrorInvalidValue;
        cudaError_t e = allow_smem(k_pr_rescore_s, sm_s);
        if (e != cudaSuccess) return e;
        k_pr_rescore_s<<<ngroups, RS_THREADS, sm_s, st>>>(a, groups, consts());
        return cudaGetLastError();
    }
    if (sm > 200 * 1024) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem(k_pr_rescore_g, sm);
    if (e != cudaSuccess) return e;
    k_pr_rescore_g<<<ngroups, 512, sm, st>>>(a, groups, consts());
    return cudaGetLastError();
}

int pr_rescore_group_size() { return RG; }

bool pr_rescore_shared_band(const Band& bd, int T) {
    const size_t sm = sizeof(float) * ((size_t)RG * T * 120 + (size_t)T * 120 + (size_t)(T + 1) * bd.nr) +
                      sizeof(int) * T * 60;
    const size_t sm_s = sm + sizeof(float2) * (size_t)bd.W * rescore_pitch(bd.W);
    return sm_s + sizeof(double) * 2 * RG * 32 <= 227 * 1024;
}

cudaError_t launch_insert_plane0(const InsertArgs& a, int B, cudaStream_t st) {
    k_insert_plane0<<<dim3(a.nsym, B), P0_THREADS, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sym_add(float4* acc5, float4* plane0, const Band& bd, float4* oct, float4* acc, cudaStream_t st) {
    const long C = bd.max_r + 2, n = C * C * C;
    k_sym_plane0<<<(unsigned)((C * C + 255) / 256), 256, 0, st>>>(plane0, bd, acc);
    k_sym_octant<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(acc5, bd, oct);
    k_sym_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(oct, bd, acc);
    return cudaGetLastError();
}

cudaError_t launch_fill4(float4* p, long n, float4 v, cudaStream_t st) {
    k_fill4<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(p, n, v);
    return cudaGetLastError();
}

cudaError_t launch_insert(const InsertArgs& a, int B, cudaStream_t st) {
    long total = (long)a.nsamples * a.nsym;
    dim3 grid((unsigned)((total + 255) / 256), B);
    k_insert<<<grid, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace cryoim
