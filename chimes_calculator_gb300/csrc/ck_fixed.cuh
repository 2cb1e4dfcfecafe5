// 64-bit fixed-point arithmetic of the FP64 form's 3-/4-body contraction.
//
// GB300 issues one FP64 warp instruction per 16 cycles and SM and one
// 32 x 32 + 64 bit integer multiply-add (IMAD.WIDE) per half cycle (both
// measured), so a multiply-add of two 56-bit numbers held in two limbs of 28
// bits -- three IMAD.WIDE -- costs 1.5 SM cycles against 16.  Every factor of
// the contraction is bounded: |T_n| <= 1, |n U_{n-1}| <= n^2, and a tuple's
// coefficients are scaled by a power of two so that their absolute sum stays
// below one; so no partial sum leaves the format and every rounding is an
// absolute one of 2^-57 or less of full scale (FP64 rounds each partial sum
// at 2^-53 of its own size).
//
//   Fx    value h 2^28 + l, |l| <= 2^27: T, dT, X and Y at 2^56, record sums
//         at 2^59, coefficients at 2^61
//   FxAcc sum of products: hi += a.h b.h, mid += a.h b.l + a.l b.h (the
//         low x low product, below 2^-62 of full scale, is dropped)
#pragma once
#include <cuda_runtime.h>

#include "ck_common.h"
#include "ck_math.cuh"

namespace ck {
namespace {

struct Fx {
    int h, l;
};

__device__ __forceinline__ Fx fx_split(long long v) {
    const int h = (int)((v + (1LL << (kFxLimb - 1))) >> kFxLimb);
    return Fx{h, (int)(v - ((long long)h << kFxLimb))};
}
__device__ __forceinline__ Fx fx_load(const FxPair& q) { return Fx{q.x, q.y}; }
__device__ __forceinline__ FxPair fx_store(const Fx& v) { return FxPair{v.h, v.l}; }

// product of two values, at the sum of their scales less 2^56
__device__ __forceinline__ Fx fx_mul(const Fx& a, const Fx& b) {
    long long m = (long long)a.h * b.l + (1LL << (kFxLimb - 1));
    m += (long long)a.l * b.h;
    return fx_split((long long)a.h * b.h + (m >> kFxLimb));
}

struct FxAcc {
    long long hi = 0, mid = 0;
    __device__ __forceinline__ void mac(const Fx& a, const Fx& b) {
        hi += (long long)a.h * b.h;
        mid += (long long)a.h * b.l;
        mid += (long long)a.l * b.h;
    }
    // the sum as a value, down = bits dropped from its scale
    template <int DOWN>
    __device__ __forceinline__ Fx value() const {
        if constexpr (DOWN == 0) {
            return fx_split(hi + ((mid + (1LL << (kFxLimb - 1))) >> kFxLimb));
        } else {
            return fx_split((hi + (mid >> kFxLimb) + (1LL << (DOWN - 1))) >> DOWN);
        }
    }
    // the sum in units of full scale, for a sum at 2^scale
    __device__ __forceinline__ double real(double unit) const {
        return ((double)hi + (double)mid * (1.0 / (double)(1LL << kFxLimb))) * unit;
    }
};
constexpr int kFxDown = kFxCoef - kFxSum;   // record sums: 2^61 -> 2^59
constexpr double kFxUnit = 1.0 / (double)(1LL << kFxSum);

// 2 x t for x at 2^62 and t at 2^k: at 2^k
__device__ __forceinline__ long long fx_2x(long long x, long long t) {
    const long long hi = __mul64hi(x, t);
    const unsigned long long lo = (unsigned long long)x * (unsigned long long)t;
    return (hi << 3) | (long long)(lo >> 61);
}

// Chebyshev tables and cutoff of one pair (set_cheby_polys, chimesFF.h:542-628,
// set_polys_out_of_range, chimesFF.cpp:1572-1613, get_fcut, chimesFF.h:347-386):
// T[n] and n U_{n-1}(x) 2^-kd, n < nT, at T[n * stride], D[n * stride]; fc and
// fc'; gs with dT_n/dr = gs D[n].  Below the inner cutoff the extrapolated
// T_n + k dT_n can exceed one: both tables are scaled down by 2^s and fc, fc'
// carry the 2^s (every term of S and of the G's has one factor of each pair).
__device__ __forceinline__ void pair_setup_x(const DevParamSet& P, const PairTab& Q, double r, FxPair* T, FxPair* D,
                                             int stride, int nT, int kd, double& fc, double& fcd, double& gs,
                                             int* flags) {
    const double rin = Q.rin;
    const bool oor = r < rin;
    const double rr = oor ? rin : r;
    const double e = exp(-rr * Q.inv_lam);
    const double xd = (e - Q.xavg) * Q.inv_xdiff;
    const double g = -e * Q.inv_lam * Q.inv_xdiff;
    const double finv = Q.fc_inv;
    if (!P.tersoff) {
        const double f0 = 1.0 - r * finv;
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (-3.0 * finv);
    } else {
        const double th = Q.fc_th;
        if (r < th) { fc = 1.0; fcd = 0.0; }
        else if (r > Q.rout) { fc = 0.0; fcd = 0.0; }
        else {
            const double f0 = (r - th) * finv * kPi + kPi / 2.0;
            double sn, cs;
            sincos(f0, &sn, &cs);
            fc = 0.5 + 0.5 * sn;
            fcd = 0.5 * cs * (kPi * finv);
        }
    }
    gs = g * (double)(1 << kd);
    double k = 0.0, damp = 1.0;
    int s = 0;
    if (oor) {
        if (flags) atomicAdd(&flags[4], 1);
        damp = exp((r - rin) / P.inner_smooth);
        k = P.inner_smooth * (damp - 1.0) * g;
        double bound = 1.0 + fabs(k) * (double)(1 << kd);
        while (bound > 1.0 && s < 40) { bound *= 0.5; s++; }
        const double up = (double)(1LL << s);
        fc *= up;
        fcd *= up;
    }
    const long long x = __double2ll_rn(xd * (double)(1LL << 62));
    // T at 2^60 and U at 2^58 along their recursions: tn, tp = T_n, T_{n+1}; um, un = U_{n-1}, U_n
    long long tn = 1LL << 60, tp = x >> 2, um = 0, un = 1LL << 58;
    for (int n = 0; n < nT; n++) {
        long long t = (tn + 8) >> 4;
        long long d = __mul64hi(um, (long long)n << (62 - kd));
        if (oor) {
            const double dn = 1.0 / (double)(1LL << s);
            t = __double2ll_rn(((double)t + k * (double)(1 << kd) * (double)d) * dn);
            d = __double2ll_rn((double)d * damp * dn);
        }
        T[n * stride] = fx_store(fx_split(t));
        D[n * stride] = fx_store(fx_split(d));
        const long long t2 = fx_2x(x, tp) - tn, u2 = fx_2x(x, un) - um;
        tn = tp;
        tp = t2;
        um = un;
        un = u2;
    }
}

}  // namespace
}  // namespace ck
