// Device helpers shared by the cluster force kernels (ck_force.cu,
// ck_factored.cu): pair geometry, force scatter to the caller's atoms, the
// per-system energy/virial accumulator and the per-cluster force epilogue.
#pragma once
#include <cuda_runtime.h>

#include "ck_common.h"
#include "ck_math.cuh"

namespace ck {

// Raises a kernel's dynamic shared-memory limit to the device's opt-in maximum,
// once per kernel.  The limit is a per-function attribute shared by every host
// thread, so it is never lowered: threads launching the same kernel with
// different shared-memory sizes (request-server workers) cannot race on it.
// The shared memory a launch actually gets is its own launch argument.
cudaError_t allow_max_smem(const void* kernel);

namespace {

constexpr unsigned kFull = 0xffffffffu;

// Checked build (compiled with -DCK_BOUNDS, libchimescalc_bounds.so): index
// checks on the arrays the cluster kernels index with computed values --
// ghost slots, caller atoms, type tuples, coefficient and factored-entry
// ranges, Chebyshev powers, tensor-core images.  A failed check raises bit 2
// of flags[7] and the access is skipped (the call then returns an error); it
// never traps.  In the normal build the checks compile to nothing.
#ifdef CK_BOUNDS
__device__ __forceinline__ bool ck_bound(const BatchView& B, bool ok) {
    if (!ok) atomicOr(&B.flags[7], 2);
    return ok;
}
#else
__device__ __forceinline__ bool ck_bound(const BatchView&, bool) { return true; }
#endif
// Vector between two images; its squared length.
__device__ __forceinline__ double pair_vec(const BatchView& B, const double* h, int ga, int gb, double* dr) {
    if (!ck_bound(B, ga >= 0 && ga < B.n_ghost_total && gb >= 0 && gb < B.n_ghost_total)) {
        dr[0] = dr[1] = dr[2] = 0.0;
        return 1e300;   // beyond every cutoff: the cluster is dropped
    }
    const double* fa = &B.ghost_fs[3 * (long long)ga];
    const double* fb = &B.ghost_fs[3 * (long long)gb];
    const double dx = fb[0] - fa[0], dy = fb[1] - fa[1], dz = fb[2] - fa[2];
    dr[0] = h[0] * dx + h[1] * dy + h[2] * dz;
    dr[1] = h[3] * dx + h[4] * dy + h[5] * dz;
    dr[2] = h[6] * dx + h[7] * dy + h[8] * dz;
    return dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
}
__device__ __forceinline__ void pair_geom(const BatchView& B, const double* h, int ga, int gb, double* dr, double& r) {
    r = sqrt(pair_vec(B, h, ga, gb, dr));
}

// Ordered type tuple of cluster c: its ghost slots, system, parameter set and tuple index.
template <int NB>
__device__ __forceinline__ const TupleRec* cluster_tuple(const BatchView& B, const int* clusters, long long c,
                                                         int* id, int& s, const DevParamSet*& P, int& u) {
    for (int k = 0; k < NB; k++) {
        id[k] = clusters[(long long)NB * c + k];
        if (!ck_bound(B, id[k] >= 0 && id[k] < B.n_ghost_total)) id[k] = 0;
    }
    s = B.atom_sys[B.ghost_parent[id[0]]];
    P = &B.psets[B.sys[s].pset];
    u = 0;
    for (int k = 0; k < NB; k++) u = u * P->ntypes + B.atom_type[B.ghost_parent[id[k]]];
    int ntup = 1;
    for (int k = 0; k < NB; k++) ntup *= P->ntypes;
    if (!ck_bound(B, u >= 0 && u < ntup)) u = 0;
    return (NB == 3 ? P->t3 : P->t4) + u;
}

// (o: one of the caller's atoms)
__device__ __forceinline__ void add_force_atom(const BatchView& B, int o, double fx, double fy, double fz) {
    if (!ck_bound(B, o >= 0 && o < B.n_in_total)) return;
    atomicAdd(&B.force[3 * (long long)o + 0], fx);
    atomicAdd(&B.force[3 * (long long)o + 1], fy);
    atomicAdd(&B.force[3 * (long long)o + 2], fz);
}
__device__ __forceinline__ void add_force(const BatchView& B, int ghost, double fx, double fy, double fz) {
    add_force_atom(B, B.atom_orig[B.ghost_parent[ghost]], fx, fy, fz);
}

// Per-atom energy and virial of one n-atom interaction, shared equally by its
// atoms (Pair::ev_tally_mb, etc/lmp/etc/pair.cpp); vir in the order
// xx xy xz yy yz zz, stored as xx yy zz xy xz yz.  Only when requested.
// (at: the caller's atoms)
__device__ __forceinline__ void tally_at(const BatchView& B, const int* at, int n, double e, const double* vir) {
    if (!B.eatom && !B.vatom) return;
    const double w = 1.0 / n;
    for (int k = 0; k < n; k++) {
        const long long o = at[k];
        if (B.eatom) atomicAdd(&B.eatom[o], e * w);
        if (B.vatom) {
            double* v = &B.vatom[6 * o];
            atomicAdd(&v[0], vir[0] * w);
            atomicAdd(&v[1], vir[3] * w);
            atomicAdd(&v[2], vir[5] * w);
            atomicAdd(&v[3], vir[1] * w);
            atomicAdd(&v[4], vir[2] * w);
            atomicAdd(&v[5], vir[4] * w);
        }
    }
}

// The same for ghosts or atoms of the list.
__device__ __forceinline__ void tally_atoms(const BatchView& B, const int* ghosts, int n, double e, const double* vir) {
    if (!B.eatom && !B.vatom) return;
    int at[4];
    for (int k = 0; k < n; k++) at[k] = B.atom_orig[B.ghost_parent[ghosts[k]]];
    tally_at(B, at, n, e, vir);
}

// Energy/virial accumulator for one system at a time, per lane.
struct EVAcc {
    int s = -1;
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    __device__ void flush(const BatchView& B) {
        if (s >= 0)
            for (int k = 0; k < 7; k++) atomicAdd(&B.ev[8 * s + k], v[k]);
        s = -1;
        for (int k = 0; k < 7; k++) v[k] = 0;
    }
    __device__ void add(const BatchView& B, int sys, double e, const double* vir) {
        if (sys != s) { flush(B); s = sys; }
        v[0] += e;
        for (int k = 0; k < 6; k++) v[1 + k] += vir[k];
    }
    // end of kernel: one set of atomics per warp when its lanes hold one system
    __device__ void flush_warp(const BatchView& B) {
        const int lane = threadIdx.x & 31;
        const unsigned have = __ballot_sync(kFull, s >= 0);
        if (!have) return;
        const int s0 = __shfl_sync(kFull, s, __ffs(have) - 1);
        if (__all_sync(kFull, s < 0 || s == s0)) {
            for (int k = 0; k < 7; k++) {
                double x = v[k];
                for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(kFull, x, off);
                v[k] = x;
            }
            if (lane == 0)
                for (int k = 0; k < 7; k++) atomicAdd(&B.ev[8 * s0 + k], v[k]);
        } else {
            flush(B);
        }
    }
};

// The same per warp (all 32 lanes call it): lane 4 k holds value k of the sum of
// one system at a time.
struct EVWarp {
    int ws = -1;      // the sum's system (uniform)
    double wv = 0.0;
    __device__ void flush(const BatchView& B) {
        const int lane = threadIdx.x & 31;
        if (ws >= 0 && (lane & 3) == 0 && lane < 28) atomicAdd(&B.ev[8 * ws + (lane >> 2)], wv);
        ws = -1;
        wv = 0.0;
    }
    // One interaction's energy and virial per lane (valid lanes), summed over
    // the warp per system -- the lanes of a warp mostly hold one, or few; more than
    // kRounds add theirs one by one.  The seven sums are folded together (a
    // lane keeps half of its values and hands over the rest at each step: 9
    // additions, where seven butterflies take 35; GB300 issues an FP64 addition
    // per 16 cycles and SM), so each costs 10 FP64 instructions.
    static constexpr int kRounds = 6;
    __device__ void add(const BatchView& B, int sys, double e, const double* vir, bool valid) {
        const int lane = threadIdx.x & 31;
        unsigned have = __ballot_sync(kFull, valid);
        for (int round = 0; have && round < kRounds; round++) {
            const int s0 = __shfl_sync(kFull, sys, __ffs(have) - 1);
            const bool mine = valid && sys == s0;
            have &= ~__ballot_sync(kFull, mine);
            double x[8];
            x[0] = mine ? e : 0.0;
#pragma unroll
            for (int k = 0; k < 6; k++) x[1 + k] = mine ? vir[k] : 0.0;
            x[7] = 0.0;
#pragma unroll
            for (int n = 4, off = 16; n >= 1; n >>= 1, off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int k = 0; k < n; k++) {
                    const double give = up ? x[k] : x[k + n], keep = up ? x[k + n] : x[k];
                    x[k] = keep + __shfl_xor_sync(kFull, give, off);
                }
            }
            x[0] += __shfl_xor_sync(kFull, x[0], 2);
            x[0] += __shfl_xor_sync(kFull, x[0], 1);
            if (s0 != ws) {
                flush(B);
                ws = s0;
            }
            wv += x[0];
            if (mine) valid = false;
        }
        if (valid) {
            atomicAdd(&B.ev[8 * sys], e);
            for (int k = 0; k < 6; k++) atomicAdd(&B.ev[8 * sys + 1 + k], vir[k]);
        }
    }
};

// Chebyshev tables and cutoff of pair p of a tuple (set_cheby_polys,
// chimesFF.h:542-628; get_fcut, chimesFF.h:347-386) with the tuple's
// precomputed reciprocals in place of the divisions; ex = exp(-r / lambda).
__device__ __forceinline__ PairTab tuple_pair(const TupleRec& R, int p) {
    return PairTab{R.rin[p], R.rout[p], R.xavg[p], R.xdiff[p], R.inv_lam[p], R.inv_xdiff[p], R.fc_th[p], R.fc_inv[p]};
}

template <typename CT>
__device__ __forceinline__ void pair_setup(const DevParamSet& P, const PairTab& Q, double r, double ex, CT* T, CT* D,
                                           int stride, int nT, CT& fc, CT& fcd, int* flags) {
    const double rin = Q.rin;
    const bool oor = less_pos(r, rin);
    const double e = oor ? exp_neg(rin * Q.inv_lam) : ex;
    const double xd = (e - Q.xavg) * Q.inv_xdiff;
    const double dxdr = -e * Q.inv_lam * Q.inv_xdiff;
    cheby_fill_strided<CT>(T, D, stride, nT, xd, dxdr, oor, r, rin, P.inner_smooth, flags);
    const double finv = Q.fc_inv;
    if (!P.tersoff) {
        const CT f0 = CT(1.0) - to_ct<CT>(r) * to_ct<CT>(finv);
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (CT(-3.0) * to_ct<CT>(finv));
    } else {
        const double th = Q.fc_th;
        if (less_pos(r, th)) { fc = CT(1); fcd = CT(0); }
        else if (!less_pos(r, Q.rout) && r > Q.rout) { fc = CT(0); fcd = CT(0); }
        else {
            const CT f0 = to_ct<CT>(r - th) * to_ct<CT>(finv) * CT(kPi) + CT(kPi / 2.0);
            CT sn, cs;
            csincos<CT>(f0, &sn, &cs);
            fc = CT(0.5) + CT(0.5) * sn;
            fcd = CT(0.5) * cs * (CT(kPi) * to_ct<CT>(finv));
        }
    }
}

__device__ __forceinline__ void virial_add(double* vir, double f, const double* d) {
    vir[0] -= f * d[0] * d[0];
    vir[1] -= f * d[0] * d[1];
    vir[2] -= f * d[0] * d[2];
    vir[3] -= f * d[1] * d[1];
    vir[4] -= f * d[1] * d[2];
    vir[5] -= f * d[2] * d[2];
}

// compute_2B (chimesFF.cpp:1644-1775) of one pair below its outer cutoff:
// energy E (Chebyshev sum with T_{pow+1}, cutoff, penalty) and the force
// scalar fs (F_i += fs dr, F_j -= fs dr, virial -= fs dr (x) dr).  flags:
// device diagnostics (badness max, penalty hits, below-rin count).
template <typename CT>
__device__ __forceinline__ void pair_2b(const DevParamSet& P, const PairRec& pr, double dist, int* flags, double& E,
                                        double& fs) {
    // the Morse map with the pair type's reciprocals (no FP64 divisions:
    // GB300 issues FP64 at a small fraction of the FP32 rate, and a division
    // is several FP64 instructions)
    const bool oor = dist < pr.rin;
    const double rr = oor ? pr.rin : dist;
    const double ex = exp(-rr * pr.inv_lam);
    const double xd = (ex - pr.xavg) * pr.inv_xdiff;
    const double dxdr = -ex * pr.inv_lam * pr.inv_xdiff;
    const CT* a = coef2<CT>(P) + pr.coef_off;   // dense a_n, n = 0..o2
    const CT x = CT(xd), tx = CT(2) * x;
    CT t0c = CT(1), t1c = x, u0 = CT(1), u1 = tx;
    CT S = a[0] * t0c + a[1] * t1c;
    CT GD = a[1] * u0;                     // sum a_n n U_{n-1}
    for (int n = 2; n <= P.o2; n++) {
        const CT t2 = tx * t1c - t0c;
        const CT u2 = tx * u1 - u0;
        S += a[n] * t2;
        GD += a[n] * CT(n) * u1;
        t0c = t1c; t1c = t2; u0 = u1; u1 = u2;
    }
    double Sd = double(S), Gd = double(GD) * dxdr;
    if (oor) {
        atomicAdd(&flags[4], 1);
        const double damp = exp((dist - pr.rin) / P.inner_smooth);
        Sd += P.inner_smooth * (damp - 1.0) * Gd;
        Gd *= damp;
    }
    double fc, fcd;
    if (!P.tersoff) {
        const double f0 = 1.0 - dist * pr.fc_inv;
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (-3.0 * pr.fc_inv);
    } else if (dist < pr.fc_th) {
        fc = 1.0;
        fcd = 0.0;
    } else if (dist > pr.rout) {
        fc = 0.0;
        fcd = 0.0;
    } else {
        const double f0 = (dist - pr.fc_th) * pr.fc_inv * kPi + kPi / 2.0;
        double sn, cs;
        sincos(f0, &sn, &cs);
        fc = 0.5 + 0.5 * sn;
        fcd = 0.5 * cs * (kPi * pr.fc_inv);
    }
    E = fc * Sd;
    const double dx_inv = dist > 0.0 ? 1.0 / dist : 1e20;
    fs = (fc * Gd + fcd * Sd) * dx_inv;
    // get_penalty (chimesFF.h:388-419)
    if (dist - P.pen_dist < pr.rin) {
        const double rp = pr.rin + P.pen_dist - dist;
        atomicMax(&flags[2], dist < pr.rin ? 2 : 1);
        if (rp > 0.0) {
            atomicAdd(&flags[3], 1);
            E += rp * rp * rp * P.pen_scale;
            fs += (-3.0 * rp * rp * P.pen_scale) / dist;
        }
    }
}

// Forces, virial and energy of one 3- or 4-body cluster from its contraction
// sums (compute_3B/4B, chimesFF.cpp:2068-2169 and the 4-body counterpart):
//   f_p = (prod_{q!=p} fc_q / r_p) (fc_p G_p + fc'_p S),  E = prod fc * S.
template <int NB>
__device__ __forceinline__ void cluster_epilogue(const BatchView& B, const int* id, int sys,
                                                 const double (*dr)[4], const double* fc, const double* fcd,
                                                 double S, const double* G, EVAcc& acc) {
    constexpr int NP = Topo<NB>::NP;
    double pre[NP + 1], suf[NP + 1];
    pre[0] = 1.0;
    for (int p = 0; p < NP; p++) pre[p + 1] = pre[p] * fc[p];
    suf[NP] = 1.0;
    for (int p = NP - 1; p >= 0; p--) suf[p] = suf[p + 1] * fc[p];
    double f[NB][3];
    for (int k = 0; k < NB; k++) f[k][0] = f[k][1] = f[k][2] = 0.0;
    double vir[6] = {0, 0, 0, 0, 0, 0};
    for (int p = 0; p < NP; p++) {
        const double fsp = pre[p] * suf[p + 1] / dr[p][3] * (fc[p] * G[p] + fcd[p] * S);
        const int a = Topo<NB>::a(p), b = Topo<NB>::b(p);
        for (int k = 0; k < 3; k++) {
            f[a][k] += fsp * dr[p][k];
            f[b][k] -= fsp * dr[p][k];
        }
        virial_add(vir, fsp, dr[p]);
    }
    int at[NB];
    for (int k = 0; k < NB; k++) at[k] = B.atom_orig[B.ghost_parent[id[k]]];
    for (int k = 0; k < NB; k++) add_force_atom(B, at[k], f[k][0], f[k][1], f[k][2]);
    acc.add(B, sys, pre[NP] * S, vir);
    tally_at(B, at, NB, pre[NP] * S, vir);
}

// The same for the mixed form, in FP32: the cluster's force scalars, forces
// and virial derive from the FP32 contraction sums, so they are formed in
// FP32 (GB300's FP64 pipe issues one warp instruction per 16 cycles per SM,
// and this epilogue was most of a mixed cluster kernel's FP64 work); the
// per-atom forces (FP64 atomics) and the system's energy and virial (FP64)
// are accumulated in FP64.  dr: the pairs' vectors, rinv: 1 / distance.
// The cluster's energy and virial are returned for the caller's (warp-wide)
// accumulation.  at: the cluster's atoms among the caller's.
template <int NB>
__device__ __forceinline__ void cluster_epilogue_f32(const BatchView& B, const int* at, const float (*dr)[3],
                                                     const float* rinv, const float* fc, const float* fcd, float S,
                                                     const float* G, double& e_out, double* vir_out) {
    constexpr int NP = Topo<NB>::NP;
    float pre[NP + 1], suf[NP + 1];
    pre[0] = 1.0f;
#pragma unroll
    for (int p = 0; p < NP; p++) pre[p + 1] = pre[p] * fc[p];
    suf[NP] = 1.0f;
#pragma unroll
    for (int p = NP - 1; p >= 0; p--) suf[p] = suf[p + 1] * fc[p];
    float f[NB][3];
#pragma unroll
    for (int k = 0; k < NB; k++) f[k][0] = f[k][1] = f[k][2] = 0.0f;
    float v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const float fsp = pre[p] * suf[p + 1] * rinv[p] * (fc[p] * G[p] + fcd[p] * S);
        const int a = Topo<NB>::a(p), b = Topo<NB>::b(p);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            f[a][k] += fsp * dr[p][k];
            f[b][k] -= fsp * dr[p][k];
        }
        v[0] -= fsp * dr[p][0] * dr[p][0];
        v[1] -= fsp * dr[p][0] * dr[p][1];
        v[2] -= fsp * dr[p][0] * dr[p][2];
        v[3] -= fsp * dr[p][1] * dr[p][1];
        v[4] -= fsp * dr[p][1] * dr[p][2];
        v[5] -= fsp * dr[p][2] * dr[p][2];
    }
#pragma unroll
    for (int k = 0; k < NB; k++) add_force_atom(B, at[k], widen(f[k][0]), widen(f[k][1]), widen(f[k][2]));
    for (int k = 0; k < 6; k++) vir_out[k] = widen(v[k]);
    e_out = widen(pre[NP] * S);
    tally_at(B, at, NB, e_out, vir_out);
}

}  // namespace
}  // namespace ck
