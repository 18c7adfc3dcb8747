// sp_node.cuh -- the per-node implicit stream-power update, shared by the
// single-grid sweep (stream_power.cu) and the packed ensemble (ensemble.cu).
#pragma once

#include <cmath>

#include "common.cuh"

namespace lsdtt_gb300
{
namespace
{

struct SpParams
{
    float K, m, n, dt, threshold, slope_clamp, dx, dx_diag;
    int divide_by_dx;
    int n_is_one;
};

// slope^e for the Newton iteration. The stream-power exponents the
// configurations use (n = 1, 1.5, 2, hence e in {0.5, 1, 1.5, 2}) take
// exact identities with one or two correct roundings (x*x, x, sqrt(x),
// x*sqrt(x)), which are at least as accurate as the general double pow
// and avoid its FP64 cost inside the level-ordered sweep; any other
// exponent takes pow.
__device__ __forceinline__ double sp_pow(double x, double e)
{
    if (e == 2.0) return __dmul_rn(x, x);
    if (e == 1.0) return x;
    if (e == 0.5) return __dsqrt_rn(x);
    if (e == 1.5) return __dmul_rn(x, __dsqrt_rn(x));
    return pow(x, e);
}

// K * A^m of one node in the reference's double arithmetic
// (stream_power_cpu.cpp:236-262), or -1 when the node is below the
// incision threshold (not eroded). area_d is the accumulate() total.
__device__ __forceinline__ double sp_kam(const SpParams& P, double area_d, float Ki)
{
    double area = area_d;
    if (P.divide_by_dx) area = __ddiv_rn(area, static_cast<double>(P.dx));
    if (P.threshold > 0.0f && area < static_cast<double>(P.threshold)) return -1.0;
    return __dmul_rn(static_cast<double>(Ki), pow(area, static_cast<double>(P.m)));
}

// ---- the update in two FP32 words -------------------------------------------
// The reference solves a node in FP64 and rounds to float once per step. This
// part's FP64 pipe takes 16 cycles an instruction and warp, and a node is 13
// (n = 1) or several hundred of them (division and square root are sequences),
// so the sweeps were bound by it. The same values are formed here in pairs of
// FP32 words (error-free sums and products), right to about 2^-44 of their
// terms where the FP64 ones are right to 2^-51. Where both ends of that
// interval lead to the same float (and to the same answer of the loop's test),
// it is the float that the FP64 expression gives; where they do not, the FP64
// expression is evaluated. So the bits are the reference's, and FP64 is left
// for about one node in 10^4.

// float((zo + zr spf) / (1 + spf)) = zr + (zo - zr) w for w = 1 / (1 + spf)
// = wh + wl, zr < zo; false where FP64 has to decide.
__device__ __forceinline__ bool sp_linear_pair(float wh, float wl, float zo, float zr, float& zn)
{
    const float d = zo - zr, bb = d - zo, dl = (zo - (d - bb)) - (zr + bb);
    const float ph = d * wh, pl = fmaf(d, wh, -ph) + fmaf(d, wl, dl * wh);
    const float s = zr + ph, t = s - zr, lo = ((zr - (s - t)) + (ph - t)) + pl;
    const float size = fabsf(zr) + fabsf(zo), err = size * 5.6843419e-14f;  // 2^-44
    const float up = s + (lo + err), dn = s + (lo - err);
    zn = up;
    return up == dn && size > 1e-20f && size < 1e30f;
}

// A Newton step of the n = 1.5 or n = 2 update: zn - float(eps) for eps = fz /
// fdz, fz = (zn - zo) + kdt s^n, fdz = 1 + kdt ndx s^(n-1) (kdt = kh + kl, kdt
// ndx = gh + gl), and whether |eps| > tol; false where FP64 has to decide.
__device__ __forceinline__ bool sp_newton_pair(bool square, float s, float kh, float kl, float gh, float gl, float dz,
                                               float tol, float zn, float& z_next, bool& again)
{
    // p = s^n and r = s^(n-1)
    float rh = s, rl = 0.0f;
    if (!square)
    {
        rh = __fsqrt_rn(s);
        rl = 0.5f * fmaf(-rh, rh, s) * __frcp_rn(rh);
    }
    const float ph = s * rh, pl = fmaf(s, rh, -ph) + s * rl;
    const float th = kh * ph, tl = fmaf(kh, ph, -th) + fmaf(kh, pl, kl * ph);
    const float fh = dz + th, a = fh - dz, fl = ((dz - (fh - a)) + (th - a)) + tl;
    const float uh = gh * rh, ul = fmaf(gh, rh, -uh) + fmaf(gh, rl, gl * rh);
    const float qh = 1.0f + uh, b = qh - 1.0f, ql = ((1.0f - (qh - b)) + (uh - b)) + ul;
    const float inv = __frcp_rn(qh), e0 = fh * inv;
    const float e1 = (fmaf(-e0, qh, fh) + fmaf(-e0, ql, fl)) * inv;
    const float err = (fabsf(dz) + th) * inv * 2.2737368e-13f;  // 2^-42
    const float up = e0 + (e1 + err), dn = e0 + (e1 - err);
    z_next = zn - up;
    const float au = fabsf(up), ad = fabsf(dn);
    again = au > tol;
    const bool clear = fminf(au, ad) > tol * 1.000001f || fmaxf(au, ad) < tol * 0.999999f;
    return z_next == zn - dn && clear && th < 1e30f && uh < 1e30f && err > 1e-36f;
}

// The implicit update of one node (stream_power_cpu.cpp:263-318): its new
// elevation from its own old elevation zo, its receiver's final elevation
// zr, kam = sp_kam(...) and the step length to the receiver. Returns zo when
// the node is not eroded.
// tol_dx: the length the elevation tolerance slope_clamp * tol_dx is taken
// over (the step length to the receiver for D8; the cardinal cell size for
// D-infinity, stream_power_cpu.cpp:437).
__device__ __forceinline__ float sp_solve_tol(const SpParams& P, bool diagonal, double kam, float zo, float zr,
                                              float tol_dx)
{
    if (zr >= zo) return zo;
    const float dx_eff = diagonal ? P.dx_diag : P.dx;
    const double tol = __dmul_rn(static_cast<double>(P.slope_clamp), static_cast<double>(tol_dx));
    float zn = zo;
    if (P.n_is_one)
    {
        // w = 1 / (1 + spf) from spf in two words
        const float q = __fdiv_rn(P.dt, dx_eff);
        const float kh = static_cast<float>(kam), kl = static_cast<float>(kam - static_cast<double>(kh));
        const float sh = kh * q, sl = fmaf(kh, q, -sh) + kl * q;
        const float dh = 1.0f + sh, b = dh - 1.0f, dl = ((1.0f - (dh - b)) + (sh - b)) + sl;
        const float wh = __frcp_rn(dh), wl = (fmaf(-wh, dh, 1.0f) - wh * dl) * wh;
        if (sh < 1e15f && sh > 1e-30f && sp_linear_pair(wh, wl, zo, zr, zn))
        {
            if (__fsub_rn(zn, zo) > static_cast<float>(tol) || isnan(zn)) zn = zo;
            return zn;
        }
        const double spf = __dmul_rn(kam, static_cast<double>(__fdiv_rn(P.dt, dx_eff)));
        const double num = __dadd_rn(static_cast<double>(zo), __dmul_rn(static_cast<double>(zr), spf));
        zn = static_cast<float>(__ddiv_rn(num, __dadd_rn(1.0, spf)));
        if (__fsub_rn(zn, zo) > static_cast<float>(tol) || isnan(zn)) zn = zo;
    }
    else
    {
        double eps = 0.0;
        int it = 0;
        const double nd = static_cast<double>(P.n);
        const double kdt = __dmul_rn(kam, static_cast<double>(P.dt));
        const float ndxf = __fdiv_rn(P.n, dx_eff);
        const double ndx = static_cast<double>(ndxf);
        const bool square = P.n == 2.0f;
        const float kh = static_cast<float>(kdt), kl = static_cast<float>(kdt - static_cast<double>(kh));
        const float gh = kh * ndxf, gl = fmaf(kh, ndxf, -gh) + kl * ndxf, tolf = static_cast<float>(tol);
        const bool pair = (square || P.n == 1.5f) && kh > 1e-25f && gh > 1e-25f;
        for (;;)
        {
            const float sf = __fdiv_rn(__fsub_rn(zn, zr), dx_eff);
            if (sf <= 0.0f) eps = 0.0;
            else
            {
                float next;
                bool again;
                if (pair && it < 100 && sf > 1e-10f &&
                    sp_newton_pair(square, sf, kh, kl, gh, gl, __fsub_rn(zn, zo), tolf, zn, next, again))
                {
                    zn = next;
                    ++it;
                    if (again) continue;
                    break;
                }
                const double slope = static_cast<double>(sf);
                const double fz = __dadd_rn(static_cast<double>(__fsub_rn(zn, zo)), __dmul_rn(kdt, sp_pow(slope, nd)));
                const double fdz =
                    __dadd_rn(1.0, __dmul_rn(__dmul_rn(kdt, ndx), sp_pow(slope, __dsub_rn(nd, 1.0))));
                eps = __ddiv_rn(fz, fdz);
            }
            zn = __fsub_rn(zn, static_cast<float>(eps));
            ++it;
            if (it > 100) eps = tol / 2.0;
            if (!(fabs(eps) > tol)) break;
        }
        if (__fsub_rn(zn, zo) > static_cast<float>(tol) || isnan(zn)) zn = zo;
        if (zn < zr) zn = __fadd_rn(zr, __fmul_rn(P.slope_clamp, dx_eff));
    }
    return zn;
}

__device__ __forceinline__ float sp_solve(const SpParams& P, bool diagonal, double kam, float zo, float zr)
{
    return sp_solve_tol(P, diagonal, kam, zo, zr, diagonal ? P.dx_diag : P.dx);
}

// sp_solve for node `flat` with its own loads and store. Any receiver-
// before-donor order gives the reference's bits: a node reads only
// z_old[self] and z[receiver]. Indices are those of the arrays passed
// (n = their length). kCoherent reads the receiver's elevation from L2
// (bypassing L1), for sweeps whose levels are written by other SMs of the
// same launch.
template <bool kCoherent = false>
__device__ __forceinline__ void sp_node_kam(const SpParams& P, std::int64_t n, std::int64_t flat,
                                            const std::int64_t* __restrict__ receiver,
                                            const std::uint8_t* __restrict__ dir, double kam,
                                            const float* __restrict__ z_old, float* __restrict__ z)
{
    const std::int64_t recv = receiver[flat];
    if (recv < 0 || recv >= n || kam < 0.0) return;  // outlets, nodata, below threshold
    const float zo = z_old[flat];
    const float zr = kCoherent ? __ldcg(z + recv) : z[recv];
    const float zn = sp_solve(P, (dir[flat] & 1u) != 0, kam, zo, zr);
    z[flat] = zn;  // zo when not eroded: z[flat] already holds it
}

// Both parts for one node.
__device__ __forceinline__ void sp_node(const SpParams& P, std::int64_t n, std::int64_t flat,
                                        const std::int64_t* __restrict__ receiver, const std::uint8_t* __restrict__ dir,
                                        const double* __restrict__ area_d, const float* __restrict__ z_old,
                                        const float* __restrict__ kfield, float* __restrict__ z)
{
    const std::int64_t recv = receiver[flat];
    if (recv < 0 || recv >= n) return;
    const float Ki = kfield ? kfield[flat] : P.K;
    sp_node_kam(P, n, flat, receiver, dir, sp_kam(P, area_d[flat], Ki), z_old, z);
}

}  // namespace
}  // namespace lsdtt_gb300
