// Per-cluster kernels: the chimesFF::compute_2B/3B/4B entry points, where the
// caller owns the cluster loop and passes distances, displacement vectors and
// type indices (chimesFF/src/chimesFF.cpp:1644-1775, 1931-2176, 2496-2872).
// One thread (3-/4-body: one or more lanes) per cluster, FP64, any number of
// clusters per launch; outputs are per-cluster (the host adds them into the
// caller's accumulators).
//
// Besides energy, forces and the packed stress, each cluster reports the
// reference's `force_scalar_in` value: for 2B the penalty force scalar over r
// (1.0 without a penalty), for 3B/4B the per-pair force scalars of the LAST
// coefficient of the list, as the reference's loop leaves them.  status bits:
// 1 = the cluster passed the type and cutoff checks, 2 = penalty region
// (badness 1), 4 = below the inner cutoff (badness 2), 8 = a many-body pair below
// its inner cutoff (the reference prints a warning; badness is unchanged),
// 16 = a tabulated term's distance outside its table (the reference exits or
// reads past its table there).
#include <cuda_runtime.h>

#include <algorithm>

#include "ck_common.h"
#include "ck_fixed.cuh"
#include "ck_kernels.h"
#include "ck_math.cuh"
#include "ck_tab.cuh"

namespace ck {

cudaError_t allow_max_smem(const void* kernel);   // ck_force.cu

namespace {

__global__ void k_direct2(const DevParamSet* Pp, int n, const double* dx, const double* dr, const int* typ,
                          double* force, double* stress, double* energy, double* fscal, int* status) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const DevParamSet& P = *Pp;
    for (int k = 0; k < 6; k++) { force[6 * c + k] = 0.0; stress[6 * c + k] = 0.0; }
    energy[c] = 0.0;
    fscal[c] = 0.0;
    status[c] = 0;
    const int t0 = typ[2 * c], t1 = typ[2 * c + 1];
    const PairRec pr = P.pairs[P.pair_map[t0 * P.ntypes + t1]];
    const double r = dx[c];
    const double* d = &dr[3 * c];
    if (r >= pr.rout) return;
    int st = 1;
    double xd, dxdr;
    bool oor;
    morse_x(r, pr.rin, pr.lam, pr.xavg, pr.xdiff, xd, dxdr, oor);
    const double* a = P.c2d + pr.coef_off;
    const double tx = 2.0 * xd;
    double t0c = 1.0, t1c = xd, u0 = 1.0, u1 = tx;
    double S = a[0] * t0c + a[1] * t1c, GD = a[1] * u0;
    for (int k = 2; k <= P.o2; k++) {
        const double t2 = tx * t1c - t0c, u2 = tx * u1 - u0;
        S += a[k] * t2;
        GD += a[k] * k * u1;
        t0c = t1c; t1c = t2; u0 = u1; u1 = u2;
    }
    double G = GD * dxdr;
    if (oor) {
        const double damp = exp((r - pr.rin) / P.inner_smooth);
        S += P.inner_smooth * (damp - 1.0) * G;
        G *= damp;
    }
    double fc, fcd;
    fcut_eval<double>(P, r, pr.rout, fc, fcd);
    double E = fc * S;
    const double dx_inv = r > 0.0 ? 1.0 / r : 1e20;
    double fs = (fc * G + fcd * S) * dx_inv;
    double fs_out = 1.0;
    if (r - P.pen_dist < pr.rin) {
        st |= r < pr.rin ? 4 : 2;
        const double rp = pr.rin + P.pen_dist - r;
        if (rp > 0.0) {
            E += rp * rp * rp * P.pen_scale;
            fs_out = (-3.0 * rp * rp * P.pen_scale) / r;
            fs += fs_out;
        }
    }
    for (int k = 0; k < 3; k++) {
        force[6 * c + k] = fs * d[k];
        force[6 * c + 3 + k] = -fs * d[k];
    }
    stress[6 * c + 0] = -fs * d[0] * d[0];
    stress[6 * c + 1] = -fs * d[0] * d[1];
    stress[6 * c + 2] = -fs * d[0] * d[2];
    stress[6 * c + 3] = -fs * d[1] * d[1];
    stress[6 * c + 4] = -fs * d[1] * d[2];
    stress[6 * c + 5] = -fs * d[2] * d[2];
    energy[c] = E;
    fscal[c] = fs_out;
    status[c] = st;
}

// 3-/4-body clusters of a set with fixed-point streams (ck_fixed.cuh): one warp
// per cluster, blockDim / 32 clusters per block.  The block's pairs are set up one per
// thread (a warp's FP64 instruction costs the same for one lane as for 32),
// the warp forms the cluster's products -- of both sides and their
// derivatives, so that a group of coefficients adds its row's terms at once --
// and its lanes take the stream's groups (4-body: fours of a row's or column's
// coefficients; 3-body: columns) in turn.  A group's sum is small beside the
// whole tuple's: it is kept with fx_zbits more bits (as many as the lane's sums
// leave room for), so that each cluster's own result is as good as one in FP64
// (error 5.4e-16 against 6.4e-16 of the kernel below; 5.2e-15 with sums at the scale of the
// whole one).  The lanes' sums are added in FP64 and
// the forces formed one component per thread.
// Clusters of any types in any order: the streams are read through L1/L2.
//
// Bound: latency (the set-up of a block's pairs by two of its warps, L1 reads of the
// coefficients), the FP64 pipe at 37%, four blocks of eight warps per SM (130 us with
// three, at 73 registers).  Measured, 9001 quadruplets with 4 powers per
// pair: 117 us against 873 for the per-coefficient kernel below (its FP64 pipe at
// 85%).
template <int NB>
struct DirSmem {
    static constexpr int NP = Topo<NB>::NP;
    int R, n3;         // powers per pair; products per side (4-body)
    unsigned char* base;
    __device__ DirSmem(unsigned char* b, int R_) : R(R_), n3(NB == 4 ? R_ * R_ * R_ : 0), base(b) {}
    // per cluster: FxEnt tab[NP][R], double scal[NP][4] (fc, fc', gs, r), fs[NP], sum[8];
    // int flag[NP]; 4-body: FxPair prod[2][4][n3]
    static __host__ __device__ size_t bytes(int R) {
        return (sizeof(FxEnt) * NP * R + sizeof(double) * (5 * NP + 8) + sizeof(int) * 8 +
                (NB == 4 ? sizeof(FxPair) * 8 * R * R * R : 0) + 15) / 16 * 16;
    }
    __device__ unsigned char* at(int c) const { return base + (size_t)c * bytes(R); }
    __device__ FxEnt* tab(int c) const { return reinterpret_cast<FxEnt*>(at(c)); }
    __device__ double* scal(int c) const { return reinterpret_cast<double*>(tab(c) + NP * R); }
    __device__ double* fs(int c) const { return scal(c) + 4 * NP; }
    __device__ double* sum(int c) const { return fs(c) + NP; }
    __device__ int* flag(int c) const { return reinterpret_cast<int*>(sum(c) + 8); }
    __device__ FxPair* prod(int c) const { return reinterpret_cast<FxPair*>(flag(c) + 8); }
};

template <int NB>
__global__ void __launch_bounds__(256, 4) k_directx(const DevParamSet* Pp, int n, const double* dx, const double* dr,
                                                 const int* typ, double* force, double* stress, double* energy,
                                                 double* fscal, int* status) {
    constexpr int NP = Topo<NB>::NP;
    extern __shared__ __align__(16) unsigned char smem[];
    const DevParamSet& P = *Pp;
    const int Rp = NB == 3 ? P.R3 : P.R4;
    const DirSmem<NB> m(smem, Rp);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, CB = blockDim.x >> 5;
    const int c0 = blockIdx.x * CB, nc = min(CB, n - c0);
    auto tuple = [&](int c) -> const TupleRec& {
        int u = 0;
        for (int k = 0; k < NB; k++) u = u * P.ntypes + typ[NB * (c0 + c) + k];
        return (NB == 3 ? P.t3 : P.t4)[u];
    };
    // pairs
    for (int t = threadIdx.x; t < nc * NP; t += blockDim.x) {
        const int c = t / NP, p = t % NP;
        const TupleRec& R = tuple(c);
        const double r = dx[NP * (c0 + c) + p];
        double* q = m.scal(c) + 4 * p;
        q[3] = r;
        m.flag(c)[p] = R.type_id < 0 || r >= R.rout[p] ? kPairFar : (r < R.rin[p] ? kPairOor : 0);
        if (R.type_id < 0 || r >= R.rout[p]) continue;
        // (x and the cutoff with the divisions and library functions of the kernels below)
        FxEnt* tab = m.tab(c) + p * Rp;
        double xd, dxdr, fc, fcd;
        bool oor;
        morse_x(r, R.rin[p], R.lam[p], R.xavg[p], R.xdiff[p], xd, dxdr, oor);
        fcut_eval<double>(P, r, R.rout[p], fc, fcd);
        const int kd = fx_kd(Rp);
        double gs = dxdr * (double)(1 << kd);
        // (D at T's scale: the room that the lane's sums have goes to zb)
        pair_tables_x<0>(P, r, R.rin[p], xd, gs, Rp, kd, fc, fcd,
                         [&](int k, const Fx& a, const Fx& b) { tab[k] = FxEnt{a.h, a.l, b.h, b.l}; });
        if (r != r) fc = fcd = r;   // (a distance that is no number: the cluster's results are none)
        q[0] = fc; q[1] = fcd; q[2] = gs;
    }
    __syncthreads();
    // the warp's cluster: S and the G's
    bool active = w < nc;
    if (active)
        for (int p = 0; p < NP; p++) active = active && !(m.flag(w)[p] & kPairFar);
    if (active) {
        const TupleRec& R = tuple(w);
        const FxEnt* T = m.tab(w);
        auto tv = [](const FxEnt& e) { return Fx{e.x, e.y}; };
        auto dv = [](const FxEnt& e) { return Fx{e.z, e.w}; };
        FxAcc acc[NP + 1];
        // a group's sum at 2^(kFxSum + zb): the lane adds at most 16 of them, or zb <= 3
        const int len = NB == 4 ? 4 : 1 + (Rp + 1) / 2;
        const int groups = max(R.fx_split[4] - R.fx_split[0], R.fx_split[8] - (NB == 4 ? R.fx_split[4] : 0)) / len;
        const int zb = groups <= 16 * 32 ? R.fx_zbits : min(R.fx_zbits, 3);
        auto fine = [zb](const FxAcc& a) {
            constexpr int D = kFxCoef - kFxSum;
            const long long v = zb >= D ? (a.hi << (zb - D)) + (a.mid >> (kFxLimb + D - zb))
                                        : (a.hi + (a.mid >> kFxLimb)) >> (D - zb);
            return fx_limbs(v + (1LL << (kFxLimb - 1)));
        };
        if constexpr (NB == 4) {
            FxPair* prod = m.prod(w);
            const int n3 = m.n3;
            for (int k = lane; k < 2 * n3; k += 32) {
                const int side = k >= n3 ? 1 : 0, i = k - side * n3;
                const FxEnt* t = T + 3 * side * Rp;
                const FxEnt a = t[i / (Rp * Rp)], b = t[Rp + i / Rp % Rp], c = t[2 * Rp + i % Rp];
                const Fx ab = fx_mul(tv(a), tv(b));
                FxPair* o = prod + 4 * side * n3 + i;
                o[0] = fx_store(fx_mul(ab, tv(c)));
                o[n3] = fx_store(fx_mul(fx_mul(tv(b), tv(c)), dv(a)));
                o[2 * n3] = fx_store(fx_mul(fx_mul(tv(a), tv(c)), dv(b)));
                o[3 * n3] = fx_store(fx_mul(ab, dv(c)));
            }
            __syncwarp();
            const FxEnt* ent = P.fx4 + R.fx_off;
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const FxPair *V = prod + 4 * (1 - side) * n3, *X = prod + 4 * side * n3;
                for (int o = R.fx_split[4 * side] + 4 * lane; o < R.fx_split[4 * side + 4]; o += 128) {
                    FxAcc z;
                    int pows = 0;
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const FxEnt q = ent[o + k];
                        z.mac(Fx{q.x, q.y}, fx_load(V[q.z]));
                        pows = q.w;
                    }
                    const int i = ((pows & 31) * Rp + ((pows >> kPowBits) & 31)) * Rp + ((pows >> (2 * kPowBits)) & 31);
                    const Fx zv = fine(z);
                    if (side == 0) acc[0].mac(fx_load(X[i]), zv);
#pragma unroll
                    for (int k = 0; k < 3; k++) acc[1 + 3 * side + k].mac(fx_load(X[(1 + k) * n3 + i]), zv);
                }
            }
        } else {
            const int cl = 1 + (Rp + 1) / 2, ncol = R.fx_split[8] / cl;
            const FxEnt* ent = P.fx3 + R.fx_off;
            for (int k = lane; k < ncol; k += 32) {
                const FxEnt* e = ent + k * cl;
                const FxEnt hd = e[0];
                FxAcc z, zd;
                for (int q = 0; q < Rp; q += 2) {
                    const FxEnt a = e[1 + q / 2], t0 = T[q];
                    z.mac(tv(a), tv(t0));
                    zd.mac(tv(a), dv(t0));
                    if (q + 1 < Rp) {
                        const FxEnt t1 = T[q + 1];
                        z.mac(dv(a), tv(t1));
                        zd.mac(dv(a), dv(t1));
                    }
                }
                const FxEnt b = T[Rp + hd.x], c = T[2 * Rp + hd.y];
                const Fx zv = fine(z), Y = fx_mul(tv(b), tv(c));
                acc[0].mac(Y, zv);
                acc[1].mac(Y, fine(zd));
                acc[2].mac(fx_mul(dv(b), tv(c)), zv);
                acc[3].mac(fx_mul(tv(b), dv(c)), zv);
            }
        }
        // summed over the lanes, folded: lane 4 k ends with sum k
        const double unit = R.fx_amp * ldexp(kFxUnit, -zb);
        double x[8];
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = k <= NP ? (double)acc[k <= NP ? k : 0].sum() : 0.0;
#pragma unroll
        for (int h = 4, off = 16; h >= 1; h >>= 1, off >>= 1) {
            const bool up = lane & off;
#pragma unroll
            for (int k = 0; k < h; k++) {
                const double give = up ? x[k] : x[k + h], keep = up ? x[k + h] : x[k];
                x[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
            }
        }
        x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
        x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
        if ((lane & 3) == 0) m.sum(w)[lane >> 2] = x[0] * unit;
    }
    if (w < nc && lane == 0) m.flag(w)[7] = active;
    __syncthreads();
    // force scalars, and those of the last coefficient
    for (int t = threadIdx.x; t < nc * NP; t += blockDim.x) {
        const int c = t / NP, p = t % NP;
        double f = 0.0, last = 0.0;
        if (m.flag(c)[7]) {
            const TupleRec& R = tuple(c);
            const double* q = m.scal(c);
            double rest = 1.0;
            for (int u = 0; u < NP; u++)
                if (u != p) rest *= q[4 * u];
            rest /= q[4 * p + 3];
            const double S = m.sum(c)[0], G = m.sum(c)[1 + p] * q[4 * p + 2];
            f = rest * (q[4 * p] * G + q[4 * p + 1] * S);
            if (R.ncoef > 0) {
                const int kl = R.coef_off + R.ncoef - 1;
                const uint32_t pw = (NB == 3 ? P.p3 : P.p4)[kl];
                double a = (NB == 3 ? P.c3d : P.c4d)[kl] * rest, tp = 0.0, dp = 0.0;
                for (int u = 0; u < NP; u++) {
                    const FxEnt e = m.tab(c)[u * Rp + ((pw >> (kPowBits * u)) & 31u)];
                    const double tu = (double)(((long long)e.x << kFxLimb) + e.y) * 0x1p-56;
                    if (u != p) a *= tu;
                    else {
                        tp = tu;
                        dp = (double)(((long long)e.z << kFxLimb) + e.w) * 0x1p-56 * q[4 * p + 2];
                    }
                }
                last = a * (q[4 * p] * dp + q[4 * p + 1] * tp);
            }
        }
        m.fs(c)[p] = f;
        fscal[NP * (c0 + c) + p] = last;
    }
    __syncthreads();
    // forces, stress, energy and status, one value per thread
    constexpr int NO = 3 * NB + 8;
    for (int t = threadIdx.x; t < nc * NO; t += blockDim.x) {
        const int c = t / NO, k = t % NO;
        const long long cl = c0 + c;
        const bool on = m.flag(c)[7];
        const double* d = dr + 3 * NP * cl;
        const double* fs = m.fs(c);
        double v = 0.0;
        if (k < 3 * NB) {
            if (on)
                for (int p = 0; p < NP; p++) {
                    const double g = fs[p] * d[3 * p + k % 3];
                    if (Topo<NB>::a(p) == k / 3) v += g;
                    else if (Topo<NB>::b(p) == k / 3) v -= g;
                }
            force[3 * NB * cl + k] = v;
        } else if (k < 3 * NB + 6) {
            const int s = k - 3 * NB, i = s < 3 ? 0 : s < 5 ? 1 : 2, j = s < 3 ? s : s < 5 ? s - 2 : 2;
            if (on)
                for (int p = 0; p < NP; p++) v -= fs[p] * d[3 * p + i] * d[3 * p + j];
            stress[6 * cl + s] = v;
        } else if (k == 3 * NB + 6) {
            if (on) {
                v = m.sum(c)[0];
                for (int p = 0; p < NP; p++) v *= m.scal(c)[4 * p];
            }
            energy[cl] = v;
        } else {
            int st = on ? 1 : 0;
            for (int p = 0; p < NP && on; p++)
                if (m.flag(c)[p] & kPairOor) st |= 8;   // below-rin warning only (badness is a 2B notion)
            status[cl] = st;
        }
    }
}

template <int NB>
bool launch_directx(const DevParamSet* Pd, int Rp, int n, const double* dx, const double* dr, const int* typ,
                    double* force, double* stress, double* energy, double* fscal, int* status, cudaStream_t st) {
    // clusters per block: eight, fewer where they would leave SMs idle or exceed the shared memory
    int cb = std::min(8, std::max(1, n / sm_count()));
    const size_t one = DirSmem<NB>::bytes(Rp);
    while (cb > 1 && cb * one > 96 * 1024) cb--;
    if (one > 200 * 1024) return false;
    auto kern = k_directx<NB>;
    if (cb * one > 48 * 1024) allow_max_smem((const void*)kern);
    count_launch(), kern<<<(n + cb - 1) / cb, 32 * cb, cb * one, st>>>(Pd, n, dx, dr, typ, force, stress, energy, fscal,
                                                                       status);
    return true;
}

// Sets without the streams (a coefficient that is no number, or too many powers
// per pair).  TPC lanes per cluster (a power of two up to 32): the lanes of a cluster
// fill its Chebyshev tables and cutoffs in shared memory (pair p by lane
// p mod TPC), each lane sums every TPC-th coefficient, the group reduces S and
// G with shuffles, and the lane holding the list's last coefficient supplies
// force_scalar_in.  With few clusters (a 4-body batch of a few thousand) one
// lane per cluster leaves most SMs idle; the launcher picks TPC from the
// cluster count.  One-warp blocks; shared memory per cluster
// NP * (2 * (order + 1) + 2) doubles.
template <int NB, int TPC>
__global__ void __launch_bounds__(32) k_directn(const DevParamSet* Pp, int n, const double* dx, const double* dr,
                                                const int* typ, double* force, double* stress, double* energy,
                                                double* fscal, int* status) {
    constexpr int NP = Topo<NB>::NP;
    constexpr unsigned kAll = 0xffffffffu;
    extern __shared__ __align__(16) double dsm[];
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int c = (int)(tid / TPC), gl = (int)(tid % TPC);
    const DevParamSet& P = *Pp;
    const int order = NB == 3 ? P.o3 : P.o4;
    const int op1 = order + 1;
    // this cluster's tables: T[p][0..order], D[p][0..order], then fc[p], fcd[p]
    double* tab = dsm + (long long)(threadIdx.x / TPC) * NP * (2 * op1 + 2);
    double* fcs = tab + 2 * NP * op1;
    double* fcds = fcs + NP;
    bool active = c < n;   // group-uniform; every lane reaches the syncs and shuffles below
    if (active && gl == 0) {
        for (int k = 0; k < 3 * NB; k++) force[3 * NB * c + k] = 0.0;
        for (int k = 0; k < 6; k++) stress[6 * c + k] = 0.0;
        for (int k = 0; k < NP; k++) fscal[NP * c + k] = 0.0;
        energy[c] = 0.0;
        status[c] = 0;
    }
    const TupleRec* R = nullptr;
    const double* r = nullptr;
    if (active) {
        int u = 0;
        for (int k = 0; k < NB; k++) u = u * P.ntypes + typ[NB * c + k];
        R = (NB == 3 ? P.t3 : P.t4) + u;
        r = &dx[NP * c];
        if (R->type_id < 0) active = false;   // excluded cluster type
        else
            for (int p = 0; p < NP; p++)
                if (r[p] >= R->rout[p]) active = false;
    }
    if (active)
        for (int p = gl; p < NP; p += TPC) {
            cheby_table<double>(tab + 2 * p * op1, tab + (2 * p + 1) * op1, r[p], R->rin[p], R->lam[p], R->xavg[p],
                                R->xdiff[p], order, P.inner_smooth, nullptr);
            fcut_eval<double>(P, r[p], R->rout[p], fcs[p], fcds[p]);
        }
    __syncwarp();
    double S = 0.0, G[NP], last[NP], pre[NP + 1], suf[NP + 1];
    for (int p = 0; p < NP; p++) G[p] = last[p] = 0.0;
    pre[NP] = 0.0;
    int st = 1;
    if (active) {
        for (int p = 0; p < NP; p++)
            if (r[p] < R->rin[p]) st |= 8;   // below-rin warning only (badness is a 2B notion)
        pre[0] = 1.0;
        for (int p = 0; p < NP; p++) pre[p + 1] = pre[p] * fcs[p];
        suf[NP] = 1.0;
        for (int p = NP - 1; p >= 0; p--) suf[p] = suf[p + 1] * fcs[p];
        const double* cf = (NB == 3 ? P.c3d : P.c4d) + R->coef_off;
        const uint32_t* pw = (NB == 3 ? P.p3 : P.p4) + R->coef_off;
        const int kl = R->ncoef - 1;
        for (int k = gl; k < R->ncoef; k += TPC) {
            double t[NP], dd[NP];
            for (int p = 0; p < NP; p++) {
                const int q = (pw[k] >> (kPowBits * p)) & 31u;
                t[p] = tab[2 * p * op1 + q];
                dd[p] = tab[(2 * p + 1) * op1 + q];
            }
            double tp[NP + 1], ts[NP + 1];
            tp[0] = 1.0;
            for (int p = 0; p < NP; p++) tp[p + 1] = tp[p] * t[p];
            ts[NP] = 1.0;
            for (int p = NP - 1; p >= 0; p--) ts[p] = ts[p + 1] * t[p];
            S += cf[k] * tp[NP];
            for (int p = 0; p < NP; p++) G[p] += cf[k] * dd[p] * tp[p] * ts[p + 1];
            if (k == kl)
                for (int p = 0; p < NP; p++)
                    last[p] = cf[k] * (fcs[p] * dd[p] + fcds[p] * t[p]) * (pre[p] * suf[p + 1] / r[p]) * tp[p] *
                              ts[p + 1];
        }
    }
    // combine the group's partial sums; the last coefficient's lane holds
    // force_scalar_in, the others hold zeros
#pragma unroll
    for (int off = TPC / 2; off > 0; off >>= 1) {
        S += __shfl_xor_sync(kAll, S, off);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            G[p] += __shfl_xor_sync(kAll, G[p], off);
            last[p] += __shfl_xor_sync(kAll, last[p], off);
        }
    }
    if (!active || gl != 0) return;
    const double* d = &dr[3 * NP * c];
    double vir[6] = {0, 0, 0, 0, 0, 0};
    for (int p = 0; p < NP; p++) {
        const double fsp = pre[p] * suf[p + 1] / r[p] * (fcs[p] * G[p] + fcds[p] * S);
        const double* dp = &d[3 * p];
        const int a = Topo<NB>::a(p), b = Topo<NB>::b(p);
        for (int k = 0; k < 3; k++) {
            force[3 * NB * c + 3 * a + k] += fsp * dp[k];
            force[3 * NB * c + 3 * b + k] -= fsp * dp[k];
        }
        vir[0] -= fsp * dp[0] * dp[0];
        vir[1] -= fsp * dp[0] * dp[1];
        vir[2] -= fsp * dp[0] * dp[2];
        vir[3] -= fsp * dp[1] * dp[1];
        vir[4] -= fsp * dp[1] * dp[2];
        vir[5] -= fsp * dp[2] * dp[2];
    }
    for (int k = 0; k < 6; k++) stress[6 * c + k] = vir[k];
    for (int p = 0; p < NP; p++) fscal[NP * c + p] = last[p];
    energy[c] = pre[NP] * S;
    status[c] = st;
}

template <int NB>
void launch_directn(const DevParamSet* Pd, int order, int n, const double* dx, const double* dr, const int* typ,
                    double* force, double* stress, double* energy, double* fscal, int* status, cudaStream_t st) {
    constexpr int NP = Topo<NB>::NP;
    // lanes per cluster: enough threads for about 16 warps on each of ~152 SMs
    const long long want = 152LL * 16 * 32 / (n > 0 ? n : 1);
    int tpc = 1;
    while (tpc < 32 && 2LL * tpc <= want) tpc *= 2;
    const unsigned grid = (unsigned)(((long long)n * tpc + 31) / 32);
    const size_t smem = sizeof(double) * (size_t)(32 / tpc) * NP * (2 * (order + 1) + 2);
#define CK_DIRECTN(T_)                                                                                    \
    do {                                                                                                  \
        auto kern = k_directn<NB, T_>;                                                                    \
        if (smem > 48 * 1024) allow_max_smem((const void*)kern);                                          \
        count_launch(), kern<<<grid, 32, smem, st>>>(Pd, n, dx, dr, typ, force, stress, energy, fscal, status); \
    } while (0)
    switch (tpc) {
        case 1: CK_DIRECTN(1); break;
        case 2: CK_DIRECTN(2); break;
        case 4: CK_DIRECTN(4); break;
        case 8: CK_DIRECTN(8); break;
        case 16: CK_DIRECTN(16); break;
        default: CK_DIRECTN(32); break;
    }
#undef CK_DIRECTN
}

// compute_2B_tab (chimesFF.cpp:1782-1867): table energy and force scalar;
// force_scalar_in is get_penalty's value (1.0, or the penalty slope inside the
// penalty region), which overwrites the table's scalar at the end.
__global__ void k_direct2tab(const DevParamSet* Pp, int n, const double* dx, const double* dr, const int* typ,
                             double* force, double* stress, double* energy, double* fscal, int* status) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const DevParamSet& P = *Pp;
    for (int k = 0; k < 6; k++) { force[6 * c + k] = 0.0; stress[6 * c + k] = 0.0; }
    energy[c] = 0.0;
    fscal[c] = 0.0;
    status[c] = 0;
    const int pt = P.pair_map[typ[2 * c] * P.ntypes + typ[2 * c + 1]];
    const PairRec pr = P.pairs[pt];
    const double r = dx[c];
    const double* d = &dr[3 * c];
    if (r >= pr.rout) return;
    int st = 1;
    double E, fs;
    if (tab2_lookup(P, pt, r, E, fs) != kTabOk) st |= 16;
    for (int k = 0; k < 3; k++) {
        force[6 * c + k] = __dmul_rn(fs, d[k]);
        force[6 * c + 3 + k] = __dsub_rn(0.0, __dmul_rn(fs, d[k]));
    }
    stress[6 * c + 0] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[0]), d[0]));
    stress[6 * c + 1] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[0]), d[1]));
    stress[6 * c + 2] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[0]), d[2]));
    stress[6 * c + 3] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[1]), d[1]));
    stress[6 * c + 4] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[1]), d[2]));
    stress[6 * c + 5] = __dsub_rn(0.0, __dmul_rn(__dmul_rn(fs, d[2]), d[2]));
    double fs_out = 1.0;
    if (r - P.pen_dist < pr.rin) {
        st |= r < pr.rin ? 4 : 2;
        const double rp = pr.rin + P.pen_dist - r;
        if (rp > 0.0) fs_out = __dmul_rn(__dmul_rn(__dmul_rn(-3.0, rp), rp), P.pen_scale);
    }
    energy[c] = E;
    fscal[c] = fs_out;
    status[c] = st;
}

// compute_3B_tab (chimesFF.cpp:2183-2322): the type and per-pair outer-cutoff
// checks of compute_3B, then the tricubic look-up; force_scalar_in receives the
// three table force scalars.
__global__ void k_direct3tab(const DevParamSet* Pp, int n, const double* dx, const double* dr, const int* typ,
                             double* force, double* stress, double* energy, double* fscal, int* status) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const DevParamSet& P = *Pp;
    for (int k = 0; k < 9; k++) force[9 * c + k] = 0.0;
    for (int k = 0; k < 6; k++) stress[6 * c + k] = 0.0;
    for (int k = 0; k < 3; k++) fscal[3 * c + k] = 0.0;
    energy[c] = 0.0;
    status[c] = 0;
    const int u = (typ[3 * c] * P.ntypes + typ[3 * c + 1]) * P.ntypes + typ[3 * c + 2];
    const TupleRec& R = P.t3[u];
    if (R.type_id < 0) return;
    const double* r = &dx[3 * c];
    for (int p = 0; p < 3; p++)
        if (r[p] >= R.rout[p]) return;
    double v[4];
    int st = 1;
    if (tab3_lookup(P, R.type_id, r[0], r[1], r[2], v) != kTabOk) st |= 16;
    double f[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, vir[6] = {0, 0, 0, 0, 0, 0};
    for (int p = 0; p < 3; p++) {
        const double fsp = v[1 + p];
        const double* d = &dr[9 * c + 3 * p];
        const int a = Topo<3>::a(p), b = Topo<3>::b(p);
        for (int k = 0; k < 3; k++) {
            f[3 * a + k] = __dadd_rn(f[3 * a + k], __dmul_rn(fsp, d[k]));
            f[3 * b + k] = __dsub_rn(f[3 * b + k], __dmul_rn(fsp, d[k]));
        }
        vir[0] = __dsub_rn(vir[0], __dmul_rn(fsp, __dmul_rn(d[0], d[0])));
        vir[1] = __dsub_rn(vir[1], __dmul_rn(fsp, __dmul_rn(d[0], d[1])));
        vir[2] = __dsub_rn(vir[2], __dmul_rn(fsp, __dmul_rn(d[0], d[2])));
        vir[3] = __dsub_rn(vir[3], __dmul_rn(fsp, __dmul_rn(d[1], d[1])));
        vir[4] = __dsub_rn(vir[4], __dmul_rn(fsp, __dmul_rn(d[1], d[2])));
        vir[5] = __dsub_rn(vir[5], __dmul_rn(fsp, __dmul_rn(d[2], d[2])));
    }
    for (int k = 0; k < 9; k++) force[9 * c + k] = f[k];
    for (int k = 0; k < 6; k++) stress[6 * c + k] = vir[k];
    for (int k = 0; k < 3; k++) fscal[3 * c + k] = v[1 + k];
    energy[c] = v[0];
    status[c] = st;
}

}  // namespace

void launch_direct(const DevParamSet* P, int nbody, int order, int n, const double* dx, const double* dr,
                   const int* typ, double* force, double* stress, double* energy, double* fscal, int* status,
                   cudaStream_t st, bool tab, int fx_powers) {
    if (n <= 0) return;
    const unsigned grid = (unsigned)((n + 63) / 64);
    if (tab) {
        if (nbody == 2) count_launch(), k_direct2tab<<<grid, 64, 0, st>>>(P, n, dx, dr, typ, force, stress, energy, fscal, status);
        else count_launch(), k_direct3tab<<<grid, 64, 0, st>>>(P, n, dx, dr, typ, force, stress, energy, fscal, status);
        return;
    }
    if (nbody == 2) count_launch(), k_direct2<<<grid, 64, 0, st>>>(P, n, dx, dr, typ, force, stress, energy, fscal, status);
    else if (fx_powers > 0 && (nbody == 3 ? launch_directx<3>(P, fx_powers, n, dx, dr, typ, force, stress, energy, fscal, status, st)
                                          : launch_directx<4>(P, fx_powers, n, dx, dr, typ, force, stress, energy, fscal, status, st)))
        return;
    else if (nbody == 3) launch_directn<3>(P, order, n, dx, dr, typ, force, stress, energy, fscal, status, st);
    else launch_directn<4>(P, order, n, dx, dr, typ, force, stress, energy, fscal, status, st);
}

}  // namespace ck
