// Device math shared by the cluster kernels: Morse coordinate, Chebyshev
// tables, smoothing cutoff, cluster pair topology and the per-precision
// coefficient accessors.  Restated from chimesFF (chimesFF/src/chimesFF.h:347-386
// get_fcut, :542-628 set_cheby_polys; chimesFF/src/chimesFF.cpp:1572-1613
// set_polys_out_of_range).
#pragma once
#include <cuda_runtime.h>

#include "ck_common.h"

namespace ck {
namespace {

constexpr double kPi = 3.14159265359;   // the reference's `pi` macro (chimesFF.h:22)

// double(x) without the FP64 pipe, which takes 16 cycles per SM for a warp's
// conversion: the exponent rebased and the significand shifted (zero, subnormal and
// non-finite values convert).
__device__ __forceinline__ double widen(float x) {
    const unsigned b = __float_as_uint(x);
    if (((b >> 23) & 0xffu) - 1u >= 254u) return b << 1 ? double(x) : __hiloint2double((int)b, 0);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// float(x), rounded to nearest even, the same way (out of the normal floats' range:
// converted).
__device__ __forceinline__ float narrow(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    if ((hi & 0x7fffffffu) - 0x38100000u >= 0x0fe00000u) return float(x);
    const unsigned w = __funnelshift_l(lo, hi, 3);                    // significand's top 23 bits, exponent above
    const unsigned up = ((lo & 0x1fffffffu) + 0x0fffffffu + (w & 1u)) >> 29;
    return __uint_as_float((w - 0xc0000000u + up) | (hi & 0x80000000u));
}
template <typename CT>
__device__ __forceinline__ CT to_ct(double x) {
    if constexpr (sizeof(CT) == 4) return narrow(x);
    else return x;
}

// a < b for a >= 0 (not -0) and numbers: the bits compare like integers.
__device__ __forceinline__ bool less_pos(double a, double b) {
    return __double_as_longlong(a) < __double_as_longlong(b);
}

// v 2^S rounded to an integer, |v| 2^S < 2^63; and v 2^E as a double (in the
// normal range), rounded to nearest.
__device__ __forceinline__ long long to_fixed(double v, int S) {
    const long long b = __double_as_longlong(v);
    const int sh = (int)((unsigned long long)b >> 52 & 0x7ffull) - 1075 + S;
    const unsigned long long m = ((unsigned long long)b & ((1ull << 52) - 1)) | 1ull << 52;
    const int r = min(-sh, 63);
    const long long u = (long long)(sh >= 0 ? m << sh : (m + (1ull << (r - 1))) >> r);
    return b < 0 ? -u : u;
}
__device__ __forceinline__ double from_fixed(long long v, int E) {
    unsigned long long a = (unsigned long long)(v < 0 ? -v : v);
    const int z = __clzll((long long)a);
    a <<= z;
    const long long q = (long long)((a >> 11) + ((a >> 10) & 1ull));   // 2^52 .. 2^53
    const long long bits = ((long long)(1085 - z + E) << 52) + q;
    return __longlong_as_double(v == 0 ? 0ll : bits | (v & (long long)0x8000000000000000ull));
}

// Square root and its reciprocal: one third-order Householder step for 1 / sqrt
// from an FP32 estimate (relative error e^3 5/16 < 2^-60 for e < 2^-20), then
// r = s y with one correction.  10 FP64 instructions, where sqrt and a division
// took 19 (163 + 142 SM cycles a warp).
__device__ __forceinline__ void sqrt_rcp(double s, double& r, double& y) {
    if (!(s > 1e-30 && s < 1e30)) {
        r = sqrt(s);
        y = r > 0.0 ? 1.0 / r : 1e20;
        if (s > 1e-300 && s < 1e300) {
            const double t = s * y;
            y = fma(0.5 * y, fma(-t, y, 1.0) - fma(s, y, -t) * y, y);
        }
        return;
    }
    const double y0 = widen(rsqrtf(narrow(s)));
    const double e = fma(-s, y0 * y0, 1.0);   // (the square of an FP32 number is exact)
    y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    const double t = s * y;
    r = fma(fma(-t, t, s), 0.5 * y, t);
}

// exp(-y) and the sine and cosine of the cutoffs in 64-bit integer arithmetic.
// GB300 issues an FP64 warp instruction per 16 cycles and SM: exp took 304 SM
// cycles a warp and sincos 455 (measured), a 64 x 64 bit product's high half
// about 2.  Taylor series after an exact reduction; every product is truncated
// at 2^-62 or below.
//
// exp(-y): y log2(e) = k + j / 4 + f with f < 1/4, exp(-y) = 2^-k 2^(-j/4)
// exp(-f ln 2), twelve terms (z^13 / 13! < 2^-65 for z < 0.1733).  The result is
// within 2^-56 of exp(-y) relatively for y < 64, before its rounding to a double.
__device__ __forceinline__ double exp_neg(double y) {
    if ((unsigned long long)__double_as_longlong(y) >= 0x4050000000000000ull) return exp(-y);   // not in [0, 64)
    const unsigned long long v = (unsigned long long)to_fixed(y, 57);
    const unsigned long long t = __umul64hi(v, 0xb8aa3b295c17f0bcull);                           // y log2(e) at 2^56
    const int k = (int)(t >> 56), j = (int)(t >> 54) & 3;
    const unsigned long long z = __umul64hi((t & ((1ull << 54) - 1)) << 8, 0xb17217f7d1cf79acull);   // f ln 2 at 2^64
    constexpr unsigned long long c[12] = {0x8000000000000000ull, 0x8000000000000000ull, 0x4000000000000000ull,
                                          0x1555555555555555ull, 0x0555555555555555ull, 0x0111111111111111ull,
                                          0x002d82d82d82d82eull, 0x0006806806806807ull, 0x0000d00d00d00d01ull,
                                          0x0000171de3a556c7ull, 0x0000024fc9f6ef14ull, 0x00000035cc8acfebull};   // 2^63 / n!
    unsigned long long p = 0x47bb63bfeull;
#pragma unroll
    for (int n = 11; n >= 0; n--) p = c[n] - __umul64hi(z, p);
    const unsigned long long q0 = j & 1 ? 0x6ba27e656b4eb57aull : 0x8000000000000000ull;   // 2^63 2^(-j/4)
    const unsigned long long q1 = j & 1 ? 0x4c1bf828c6dc54b8ull : 0x5a827999fcef3242ull;
    const unsigned long long m = __umul64hi(p, j & 2 ? q1 : q0);                            // at 2^62
    const unsigned long long q = (m + 256) >> 9;                                            // 2^52 .. 2^53
    return __longlong_as_double(((long long)(1021 - k) << 52) + (long long)q);
}

// sin and cos of psi, |psi| < 2, at 2^61 (both within 2^-59): series of the half
// angle to x^19 and x^18 (remainders below 2^-63), then the double angle.
__device__ __forceinline__ void sincos_fx(double psi, long long& sn, long long& cs) {
    const unsigned long long x = (unsigned long long)to_fixed(fabs(psi), 62) << 1;   // |psi| / 2 at 2^64
    const unsigned long long w = __umul64hi(x, x);
    constexpr unsigned long long s[9] = {0x8000000000000000ull, 0x1555555555555555ull, 0x0111111111111111ull,
                                         0x0006806806806807ull, 0x0000171de3a556c7ull, 0x00000035cc8acfebull,
                                         0x000000005849184full, 0x00000000006b9fd0ull, 0x000000000000654bull};   // 2^63 / (2n + 1)!
    constexpr unsigned long long c[9] = {0x8000000000000000ull, 0x4000000000000000ull, 0x0555555555555555ull,
                                         0x002d82d82d82d82eull, 0x0000d00d00d00d01ull, 0x0000024fc9f6ef14ull,
                                         0x000000047bb63bfeull, 0x00000000064e5d2aull, 0x000000000006b9fdull};   // 2^63 / (2n)!
    unsigned long long p = 0x4cull, q = 0x5a1ull;
#pragma unroll
    for (int n = 8; n >= 0; n--) {
        p = s[n] - __umul64hi(w, p);
        q = c[n] - __umul64hi(w, q);
    }
    // (+ 1: against the truncations' mean)
    const unsigned long long h = __umul64hi(x, p) + 1;        // sin(|psi| / 2) at 2^63
    const long long sv = (long long)__umul64hi(h, q) + 1;     // sin cos at 2^62: sin(psi) at 2^61
    sn = __double_as_longlong(psi) < 0 ? -sv : sv;
    cs = (1LL << 61) - 1 - (long long)__umul64hi(h, h);
}

template <typename CT> __device__ __forceinline__ void csincos(CT x, CT* s, CT* c);
template <> __device__ __forceinline__ void csincos<double>(double x, double* s, double* c) { sincos(x, s, c); }
template <> __device__ __forceinline__ void csincos<float>(float x, float* s, float* c) { sincosf(x, s, c); }

template <typename CT> __device__ __forceinline__ const CT* coef2(const DevParamSet& P);
template <> __device__ __forceinline__ const double* coef2<double>(const DevParamSet& P) { return P.c2d; }
template <> __device__ __forceinline__ const float* coef2<float>(const DevParamSet& P) { return P.c2f; }
template <typename CT, int NB> __device__ __forceinline__ const CT* coefn(const DevParamSet& P);
template <> __device__ __forceinline__ const double* coefn<double, 3>(const DevParamSet& P) { return P.c3d; }
template <> __device__ __forceinline__ const float* coefn<float, 3>(const DevParamSet& P) { return P.c3f; }
template <> __device__ __forceinline__ const double* coefn<double, 4>(const DevParamSet& P) { return P.c4d; }
template <> __device__ __forceinline__ const float* coefn<float, 4>(const DevParamSet& P) { return P.c4f; }

// get_fcut (chimesFF.h:347-386), evaluated in CT
template <typename CT>
__device__ __forceinline__ void fcut_eval(const DevParamSet& P, double r, double rc, CT& fc, CT& fcd) {
    if (!P.tersoff) {
        CT f0 = CT(1.0) - CT(r) / CT(rc);
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (CT(-3.0) / CT(rc));
    } else {
        const double th = rc - P.fcut_var * rc;
        if (r < th) { fc = CT(1); fcd = CT(0); }
        else if (r > rc) { fc = CT(0); fcd = CT(0); }
        else {
            const CT inv = CT(1.0) / CT(rc - th);
            const CT f0 = CT(r - th) * inv * CT(kPi) + CT(kPi / 2.0);
            CT sn, cs;
            csincos<CT>(f0, &sn, &cs);
            fc = CT(0.5) + CT(0.5) * sn;
            fcd = CT(0.5) * cs * (CT(kPi) * inv);
        }
    }
}

// Morse coordinate: x and dx/dr at r (clamped to rin below the inner cutoff).
// The exponential and the map are taken in FP64 in both precision modes: the
// polynomial recursion magnifies an error in x by up to n^2.
__device__ __forceinline__ void morse_x(double r, double rin, double lam, double xavg, double xdiff,
                                        double& x, double& dxdr, bool& oor) {
    oor = r < rin;
    const double rr = oor ? rin : r;
    const double e = exp(-rr / lam);
    x = (e - xavg) / xdiff;
    dxdr = (-e / lam) / xdiff;
}

// Chebyshev table T[0..o], dT/dr[0..o] (set_cheby_polys and
// set_polys_out_of_range, chimesFF.cpp:1572-1613) into a strided array.
template <typename CT>
__device__ __forceinline__ void cheby_table(CT* T, CT* D, double r, double rin, double lam, double xavg,
                                            double xdiff, int order, double inner_smooth, int* flags) {
    double xd, dxdr;
    bool oor;
    morse_x(r, rin, lam, xavg, xdiff, xd, dxdr, oor);
    const CT x = CT(xd), tx = CT(2) * x, g = CT(dxdr);
    CT t0 = CT(1), t1 = x, u0 = CT(1), u1 = tx;
    T[0] = t0; D[0] = CT(0);
    if (order >= 1) { T[1] = t1; D[1] = g * u0; }
    for (int n = 2; n <= order; n++) {
        const CT t2 = tx * t1 - t0;
        const CT u2 = tx * u1 - u0;
        T[n] = t2;
        D[n] = CT(n) * g * u1;
        t0 = t1; t1 = t2; u0 = u1; u1 = u2;
    }
    if (oor) {
        if (flags) atomicAdd(&flags[4], 1);   // global device flags, or null
        const double damp = exp((r - rin) / inner_smooth);
        const CT k = CT(inner_smooth * (damp - 1.0)), dm = CT(damp);
        for (int n = 0; n <= order; n++) {
            T[n] = T[n] + k * D[n];
            D[n] = D[n] * dm;
        }
    }
}

// The same table from a precomputed Morse coordinate (x, dx/dr, r below the
// inner cutoff), entries n = 0..nT-1 only, at T[n*stride], D[n*stride]
// (interleaved per-cluster tables of the factored contraction).
template <typename CT>
__device__ __forceinline__ void cheby_fill_strided(CT* T, CT* D, int stride, int nT, double xd, double dxdr, bool oor,
                                                   double r, double rin, double inner_smooth, int* flags) {
    const CT x = to_ct<CT>(xd), tx = CT(2) * x, g = to_ct<CT>(dxdr);
    CT k = CT(0), dm = CT(1);
    if (oor) {
        if (flags) atomicAdd(&flags[4], 1);
        const double damp = exp((r - rin) / inner_smooth);
        k = CT(inner_smooth * (damp - 1.0));
        dm = CT(damp);
    }
    // n = 0: T = 1, dT = 0
    T[0] = CT(1);
    D[0] = CT(0);
    CT t0 = CT(1), t1 = x, u0 = CT(1), u1 = tx;
    if (nT > 1) {
        const CT d1 = g * u0;
        T[stride] = oor ? t1 + k * d1 : t1;
        D[stride] = oor ? d1 * dm : d1;
    }
    for (int n = 2; n < nT; n++) {
        const CT t2 = tx * t1 - t0;
        const CT u2 = tx * u1 - u0;
        const CT dn = CT(n) * g * u1;
        T[n * stride] = oor ? t2 + k * dn : t2;
        D[n * stride] = oor ? dn * dm : dn;
        t0 = t1; t1 = t2; u0 = u1; u1 = u2;
    }
}

template <int NB>
struct Topo;
template <>
struct Topo<3> {
    static constexpr int NP = 3;
    __device__ static int a(int p) { return p == 2 ? 1 : 0; }
    __device__ static int b(int p) { return p == 0 ? 1 : 2; }
};
template <>
struct Topo<4> {
    static constexpr int NP = 6;
    __device__ static int a(int p) { return p < 3 ? 0 : (p < 5 ? 1 : 2); }
    __device__ static int b(int p) { return p < 3 ? p + 1 : (p == 3 ? 2 : 3); }
};


}  // namespace
}  // namespace ck
