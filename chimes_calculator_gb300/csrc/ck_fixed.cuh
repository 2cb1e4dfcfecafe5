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
//   Fx    value h 2^28 + l, |l| <= 2^27: T, X and Y at 2^56, dT at 2^57,
//         coefficients at 2^61
//   FxRec, FxAcc sums of products: hi += a.h b.h, mid += a.h b.l + a.l b.h (the
//         low x low product, below 2^-62 of full scale, is dropped)
//
// A sum that goes into a further product is cut to a value at 2^(59 + z), z as many
// bits as that kind of sum stays below the tuple's full scale (a sum over a row, a
// column or a run of them is small beside the whole tuple's, one with dT for a factor
// all the more): 3-body two, three with dT, which the amplitude grants; 4-body by
// tuple (TupleRec::fx_z).  Errors of one cluster against long double, in the mean over
// random clusters of 255 (3-body, 10 powers) and 281 coefficients (4-body, 4 powers),
// force sums relative to the cluster's largest: 2.7e-16 and 1.7e-16 (FP64: 4.1e-16 and
// 2.7e-16; every sum cut at 2^59 and dT at 2^56: 2.0e-15 and 1.7e-15, which made whole
// evaluations of single triplets 2.61e-15 where the FP64 kernels had 2.16e-15; 2.1e-15 now).
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

// v + 2^(kFxLimb - 1) -> the limbs of v (the rounding constant is added by the
// caller where an accumulator starts, so that it costs nothing)
__device__ __forceinline__ Fx fx_limbs(long long v) {
    return Fx{(int)(v >> kFxLimb), (int)((unsigned)v & ((1u << kFxLimb) - 1u)) - (1 << (kFxLimb - 1))};
}

// acc += a b: one IMAD.WIDE (written out: the compiler otherwise splits some
// of these products from their sums, which took a third more instructions)
__device__ __forceinline__ void imad(long long& acc, int a, int b) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(acc) : "r"(a), "r"(b));
}

// product of two values, at the sum of their scales less 2^56
__device__ __forceinline__ Fx fx_mul(const Fx& a, const Fx& b) {
    // (rounding of the shift, and fx_limbs' constant above it)
    long long m = (1LL << (kFxLimb - 1)) + (1LL << (2 * kFxLimb - 1));
    imad(m, a.h, b.l);
    imad(m, a.l, b.h);
    m >>= kFxLimb;
    imad(m, a.h, b.h);
    return fx_limbs(m);
}

// How 4-body record sums become values: shift from 2^63 and the constants of the
// rounding and of fx_limbs, added where a sum starts.
struct FxCut {
    long long hi, mid;
    int sh;
    __device__ __forceinline__ explicit FxCut(int z)
        : hi(1LL << (kFxLimb + 1 - z)), mid(z < kFxZRec ? 1LL << (kFxLimb + 1 - z) : 0), sh(kFxZRec - z) {}
};

// A record sum, kept at 2^kFxCoef (with the constants of its value already in it).
struct FxRec {
    long long hi = 1LL << (kFxLimb - 1), mid = 1LL << (kFxLimb - 1);
    FxRec() = default;
    __device__ __forceinline__ explicit FxRec(const FxCut& c) : hi(c.hi), mid(c.mid) {}
    __device__ __forceinline__ void mac(const Fx& a, const Fx& b) {
        imad(hi, a.h, b.h);
        imad(mid, a.h, b.l);
        imad(mid, a.l, b.h);
    }
    // the sum as a value at its own scale (two bits finer than 2^kFxSum)
    __device__ __forceinline__ Fx value() const { return fx_limbs(hi + (mid >> kFxLimb)); }
    // and at 2^(kFxSum + z)
    __device__ __forceinline__ Fx value(const FxCut& c) const {
        constexpr int D = kFxSum + kFxZRec - kFxCoef;
        return fx_limbs(((hi << D) + (mid >> (kFxLimb - D))) >> c.sh);
    }
};

// A sum of products with record sums or of tables, at the scale of its terms.
struct FxAcc {
    long long hi = 0, mid = 0;
    __device__ __forceinline__ void mac(const Fx& a, const Fx& b) {
        imad(hi, a.h, b.h);
        imad(mid, a.h, b.l);
        imad(mid, a.l, b.h);
    }
    // the sum as an integer at its scale, and as a value with d bits fewer
    __device__ __forceinline__ long long sum() const { return hi + ((mid + (1LL << (kFxLimb - 1))) >> kFxLimb); }
    __device__ __forceinline__ Fx value(int d = 0) const {
        return fx_limbs((sum() + ((1LL << (kFxLimb - 1 + d)) + (1LL << d >> 1))) >> d);
    }
};
constexpr double kFxUnit = 1.0 / (double)(1LL << kFxSum);

// 2 x t for x at 2^62 and t at 2^k: at 2^k
__device__ __forceinline__ long long fx_2x(long long x, long long t) {
    const long long hi = __mul64hi(x, t);
    const unsigned long long lo = (unsigned long long)x * (unsigned long long)t;
    return (hi << 3) | (long long)(lo >> 61);
}

// The Chebyshev recursions at x (in [-1, 1]): f(n, T_n, n U_{n-1} 2^-kd), n =
// 0..nT-1, T at 2^56 and the other at 2^(56 + DER) (T is kept at 2^60 and U, up to
// 31 where it is used, at 2^(57 + DER) on the way).
template <int DER, typename F>
__device__ __forceinline__ void fx_chebyshev(double xd, int nT, int kd, F&& f) {
    const long long x = to_fixed(xd, 62);
    long long tn = 1LL << 60, tp = x >> 2, um = 0, un = 1LL << (57 + DER);   // T_n, T_{n+1}, U_{n-1}, U_n
    for (int n = 0; n < nT; n++) {
        long long d = __mul64hi(um, (long long)n << (63 - kd));
        if (DER > 0) d += ((unsigned)um * (unsigned)n >> kd) & 1u;   // (rounded; without bits to spare cut)
        f(n, (tn + 8) >> 4, d);
        const long long t2 = fx_2x(x, tp) - tn, u2 = fx_2x(x, un) - um;
        tn = tp;
        tp = t2;
        um = un;
        un = u2;
    }
}

// get_fcut (chimesFF.h:347-386) with the precomputed threshold and reciprocal
__device__ __forceinline__ void fcut_x(const DevParamSet& P, double r, double rout, double th, double finv,
                                       double& fc, double& fcd) {
    if (!P.tersoff) {
        const double f0 = 1.0 - r * finv;
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (-3.0 * finv);
    } else if (less_pos(r, th)) {
        fc = 1.0;
        fcd = 0.0;
    } else if (!less_pos(r, rout) && r > rout) {
        fc = 0.0;
        fcd = 0.0;
    } else {
        // f0 = (r - th) finv kPi + kPi / 2 = pi + psi, with kPi - pi = 2.07e-13
        long long sn, cs;
        sincos_fx(((r - th) * finv - 0.5) * kPi + 2.0682310711021444e-13, sn, cs);
        fc = from_fixed((1LL << 61) - sn, -62);
        fcd = from_fixed(-cs, -62) * (kPi * finv);
    }
}

// T_n and D_n (at 2^(56 + DER)) of a pair from its x and dx/dr 2^kd (see pair_setup_x).
template <int DER, typename F>
__device__ __forceinline__ void pair_tables_x(const DevParamSet& P, double r, double rin, double xd, double& gs, int nT,
                                              int kd, double& fc, double& fcd, F&& put) {
    if (!less_pos(r, rin)) {
        fx_chebyshev<DER>(xd, nT, kd, [&](int n, long long t, long long d) { put(n, fx_split(t), fx_split(d)); });
        return;
    }
    const double damp = exp((r - rin) / P.inner_smooth);
    const double k = P.inner_smooth * (damp - 1.0) * gs;
    const double bound = 1.0 + fabs(k);
    const int s = bound > 1.0 ? min((__double2hiint(bound) >> 20) - 1022, 1000) : 0;   // bound < 2^s
    const double up = __longlong_as_double((1023LL + s) << 52), down = __longlong_as_double((1023LL - s) << 52);
    fc *= up;
    fcd *= up;
    gs *= damp * down;
    fx_chebyshev<DER>(xd, nT, kd, [&](int n, long long t, long long d) {
        put(n, fx_split(__double2ll_rn(((double)t + k * (1.0 / (1 << DER)) * (double)d) * down)), fx_split(d));
    });
}

// Chebyshev tables and cutoff of one pair (set_cheby_polys, chimesFF.h:542-628,
// set_polys_out_of_range, chimesFF.cpp:1572-1613): put(n, T_n, D_n) for n <
// nT with D_n = n U_{n-1}(x) 2^-kd; fc and fc'; gs with dT_n/dr = gs D_n.
// ex = exp(-r / lambda).  Below the inner cutoff the extrapolated T_n + k dT_n
// can exceed one: T is scaled down by 2^s, fc, fc' carry the 2^s and gs the
// exponential and 2^-s (every term of S has a T of each pair, those of a G a D of
// its own).
template <typename F>
__device__ __forceinline__ void pair_setup_x(const DevParamSet& P, const PairTab& Q, double r, double ex, int nT,
                                             int kd, double& fc, double& fcd, double& gs, F&& put) {
    const bool oor = less_pos(r, Q.rin);
    if (oor) ex = exp_neg(Q.rin * Q.inv_lam);
    const double xd = (ex - Q.xavg) * Q.inv_xdiff;
    const double g = -ex * Q.inv_lam * Q.inv_xdiff;
    fcut_x(P, r, Q.rout, Q.fc_th, Q.fc_inv, fc, fcd);
    gs = g * __longlong_as_double((1023LL + kd) << 52);
    pair_tables_x<kFxDer>(P, r, Q.rin, xd, gs, nT, kd, fc, fcd, put);
}

// compute_2B (chimesFF.cpp:1644-1775) of one pair below its outer cutoff, as
// pair_2b: energy and force scalar over r, the Chebyshev sum in fixed point.
// ex = exp(-r / lambda), rinv = 1 / r.
__device__ __forceinline__ void pair_2b_x(const DevParamSet& P, const PairRec& pr, double r, double rinv, double ex,
                                          int* flags, double& E, double& fs) {
    const bool oor = less_pos(r, pr.rin);
    if (oor) ex = exp_neg(pr.rin * pr.inv_lam);
    const double xd = (ex - pr.xavg) * pr.inv_xdiff;
    const int kd = fx_kd(P.o2 + 1);
    const double gs = -ex * pr.inv_lam * pr.inv_xdiff * __longlong_as_double((1023LL + kd) << 52);
    const FxPair* a = P.fx2 + pr.coef_off;
    FxAcc s, g;
    fx_chebyshev<kFxDer>(xd, P.o2 + 1, kd, [&](int n, long long t, long long d) {
        const Fx c = fx_load(a[n]);
        s.mac(c, fx_split(t));
        g.mac(c, fx_split(d));
    });
    double S = from_fixed(s.sum(), -kFxCoef) * pr.fx_amp, G = from_fixed(g.sum(), -kFxCoef - kFxDer) * (pr.fx_amp * gs);
    if (oor) {
        atomicAdd(&flags[4], 1);
        const double damp = exp((r - pr.rin) / P.inner_smooth);
        S += P.inner_smooth * (damp - 1.0) * G;
        G *= damp;
    }
    double fc, fcd;
    fcut_x(P, r, pr.rout, pr.fc_th, pr.fc_inv, fc, fcd);
    E = fc * S;
    fs = (fc * G + fcd * S) * rinv;
    // get_penalty (chimesFF.h:388-419)
    if (r - P.pen_dist < pr.rin) {
        const double rp = pr.rin + P.pen_dist - r;
        atomicMax(&flags[2], r < pr.rin ? 2 : 1);
        if (rp > 0.0) {
            atomicAdd(&flags[3], 1);
            E += rp * rp * rp * P.pen_scale;
            fs += (-3.0 * rp * rp * P.pen_scale) / r;
        }
    }
}

}  // namespace
}  // namespace ck
