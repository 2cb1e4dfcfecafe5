// The device arithmetic of ck_math.cuh against the native operations and long
// double: prints one "name worst" line each (test_gpu_math.py holds the limits).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "ck_math.cuh"

using namespace ck;

struct Out {
    double wide, r, y, ex;
    float nar, nar0;
    long long fix, sn, cs;
    double back;
};

__global__ void k_check(const double* x, const float* f, const long long* v, int n, Out* o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Out q;
    q.wide = widen(f[i]);
    q.nar = narrow(x[i]);
    q.nar0 = (float)x[i];
    const double a = fabs(x[i]);
    sqrt_rcp(a, q.r, q.y);
    const double e = fmod(a, 70.0);
    q.ex = exp_neg(e);
    const double psi = fmod(x[i], 2.0);
    q.fix = to_fixed(psi, 62);
    sincos_fx(psi, q.sn, q.cs);
    q.back = from_fixed(v[i], -61);
    o[i] = q;
}

static double ulp(double a, long double b) {
    if (std::isnan(a) || std::isinf(a)) return a == (double)b ? 0.0 : 1e30;
    int e;
    std::frexp((double)b, &e);
    return (double)(std::fabs((long double)a - b) / std::ldexp((long double)1, e - 53));
}

int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(-1.0, 1.0), ex(-300.0, 300.0);
    std::vector<double> x;
    std::vector<float> f;
    std::vector<long long> v;
    for (double t : {0.0, -0.0, 1.0, -1.0, 0.5, 63.999999999999993, 64.0, 1.9999999999999998, -1.9999999999999998, 3e-39, 1.2e-38,
                     3.4028234e38, 3.5e38, 1e300, 1e-300, 1.0 + std::ldexp(1.0, -24), 1.0 + 3 * std::ldexp(1.0, -24),
                     2.0 - std::ldexp(1.0, -25), 5e-324, 1e30, 1e-30})
        x.push_back(t);
    while (x.size() < 400000) {
        const int k = (int)(x.size() % 4);
        x.push_back(k == 0 ? u(g) * 2.0 : k == 1 ? u(g) * 70.0 : k == 2 ? std::ldexp(u(g), (int)ex(g)) : u(g) * 1e-3);
        if (k == 3) {   // a tie between two floats, or next to one
            uint64_t b;
            double t = x.back();
            std::memcpy(&b, &t, 8);
            b = (b & ~0x1fffffffull) | (0x10000000ull + (g() % 3) - 1);
            std::memcpy(&t, &b, 8);
            x.back() = t;
        }
    }
    const int n = (int)x.size();
    for (int i = 0; i < n; i++) {
        const uint32_t b = i < 8 ? (uint32_t[]){0u, 0x80000000u, 1u, 0x007fffffu, 0x00800000u, 0x7f7fffffu, 0x7f800000u, 0xff800000u}[i]
                                 : (uint32_t)(g() & 0xff7fffffu);   // (never NaN)
        float t;
        std::memcpy(&t, &b, 4);
        f.push_back(t);
        v.push_back(i == 0 ? 0 : i == 1 ? 1 : i == 2 ? -1 : i == 3 ? (1LL << 62) : i == 4 ? -(1LL << 62) - 1
                                                        : (long long)g() >> (1 + g() % 62));
    }
    double *dx;
    float* df;
    long long* dv;
    Out* dout;
    std::vector<Out> o(n);
    if (cudaMalloc(&dx, n * 8) || cudaMalloc(&df, n * 4) || cudaMalloc(&dv, n * 8) || cudaMalloc(&dout, n * sizeof(Out)) ||
        cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice) || cudaMemcpy(df, f.data(), n * 4, cudaMemcpyHostToDevice) ||
        cudaMemcpy(dv, v.data(), n * 8, cudaMemcpyHostToDevice))
        return 1;
    k_check<<<(n + 255) / 256, 256>>>(dx, df, dv, n, dout);
    if (cudaMemcpy(o.data(), dout, n * sizeof(Out), cudaMemcpyDeviceToHost)) return 1;
    double wide = 0, nar = 0, root = 0, rcp = 0, expn = 0, fix = 0, sn = 0, cs = 0, back = 0;
    for (int i = 0; i < n; i++) {
        const Out& q = o[i];
        const double w = (double)f[i];
        wide += std::memcmp(&w, &q.wide, 8) != 0;
        nar += std::memcmp(&q.nar, &q.nar0, 4) != 0;
        const double a = std::fabs(x[i]);
        if (a > 1e-300 && a < 1e300) {
            root = std::fmax(root, ulp(q.r, std::sqrt((long double)a)));
            rcp = std::fmax(rcp, ulp(q.y, 1 / std::sqrt((long double)a)));
        }
        const double e = std::fmod(a, 70.0);
        expn = std::fmax(expn, ulp(q.ex, std::exp(-(long double)e)));
        const long double psi = std::fmod(x[i], 2.0);
        fix = std::fmax(fix, (double)std::fabs((long double)q.fix - std::ldexp(psi, 62)));
        sn = std::fmax(sn, (double)std::fabs(std::ldexp((long double)q.sn, -61) - std::sin(psi)));
        cs = std::fmax(cs, (double)std::fabs(std::ldexp((long double)q.cs, -61) - std::cos(psi)));
        back = std::fmax(back, v[i] ? ulp(q.back, std::ldexp((long double)v[i], -61)) : q.back != 0.0);
    }
    std::printf("widen %g\nnarrow %g\nsqrt %g\nrsqrt %g\nexp %g\nfixed %g\nsin %g\ncos %g\nback %g\n", wide, nar, root, rcp,
                expn, fix, std::ldexp(sn, 59), std::ldexp(cs, 59), back);
    return 0;
}
