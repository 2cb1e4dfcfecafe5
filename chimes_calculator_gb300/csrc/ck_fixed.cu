// The FP64 form of the pair stage and of the 3-body and 4-body contraction, in
// 64-bit fixed point (arithmetic in ck_fixed.cuh, coefficient streams in
// ck_common.h).
//
// For the clusters of one ordered type tuple, with X_I the products of the row
// pairs' T (3-body: T_ij; 4-body: T_ij T_ik T_il) and Y_J those of the column
// pairs (3-body: T_ik T_jk; 4-body: T_jk T_jl T_kl):
//   z_I = sum_J a_IJ Y_J, w_J = sum_I a_IJ X_I,  S = sum_I X_I z_I,
//   G_p = sum_I (dX_I/dT_p) dT_p z_I (row pairs), sum_J (dY_J/dT_p) dT_p w_J (column pairs)
// -- the sums of compute_3B / compute_4B (chimesFF.cpp:1931-2176, 2496-2872) in
// another association order, two multiply-adds per coefficient.
//
// A block of NW warps takes 32 clusters of one tuple (the buckets' padding), a
// lane of every warp the same cluster: all lanes of a warp read the same
// coefficients (one broadcast), and the warps share the cluster's tables and
// split the coefficients (NW contiguous parts of about equal work), so that
// few clusters still fill the GPU without lanes that read different records.
// Everything is linear in the parts' sums (exact integers); warp 0 adds them
// and forms the force scalars.
//
// Pair-entry form (ENT; list-build path, when every tuple uses the same cutoffs
// for a given pair type): all pairs of a cluster are entries of some atom's
// list (BatchView::all_pairs).  k_pairs_x computes per entry, once, the
// geometry, the 2-body term, the cutoffs and the tables of both body orders;
// the cluster kernels only gather them and add each pair's force scalar to its
// entry (3 or 6 atomics and about 20 or 45 FP64 operations a cluster, where the
// set-up and epilogue per cluster took 300 or 800); k_pair_forces then
// turns each entry's scalar into forces and virial, once per entry and not once
// per cluster.  Otherwise (caller's neighbour lists, per-tuple cutoffs) a
// cluster's pairs are set up and its forces scattered in the cluster kernel.
//
// Measured (GB300, 384 configurations of 8-512 atoms, 12/10/4, 1.81 M triplets
// and 358 k quadruplets): 3-body 1.48 ms and 4-body 0.86 ms, against 5.91 and
// 3.12 ms for the FP64 factored kernels that this form replaced and 3.27 and
// 1.63 ms with the pairs set up per cluster.  (With the bits of single clusters,
// ck_fixed.cuh, the stages take 1.47 and 1.00 ms against 1.53 and 0.99 before: the
// 3-body sums need no shift now, the 4-body ones a variable one.)  Bound by the integer
// multiply-adds (about half of the pipe's rate) and the latency that 16 warps
// per SM leave exposed.
#include <cuda_runtime.h>

#include <cstdint>

#include "ck_common.h"
#include "ck_fixed.cuh"
#include "ck_force_common.cuh"
#include "ck_kernels.h"
#include "ck_math.cuh"

namespace ck {

namespace {

constexpr int kFxTile = 32;   // clusters per block

__device__ __forceinline__ FxEnt fx_quad(const Fx& t, const Fx& d) { return FxEnt{t.h, t.l, d.h, d.l}; }
__device__ __forceinline__ Fx quad_t(const FxEnt* q) { return fx_load(*reinterpret_cast<const FxPair*>(q)); }

// Per-lane energy accumulator for one system at a time.
struct EAcc {
    int s = -1;
    double v = 0.0;
    __device__ void flush(const BatchView& B) {
        if (s >= 0) atomicAdd(&B.ev[8 * s], v);
        s = -1;
        v = 0.0;
    }
    __device__ void add(const BatchView& B, int sys, double e) {
        if (sys != s) { flush(B); s = sys; }
        v += e;
    }
    // warp-collective, one interaction per valid lane: lane 0 takes the warp's
    // sum per system (see EVAcc::add_warp)
    __device__ void add_warp(const BatchView& B, int sys, double e, bool valid) {
        unsigned have = __ballot_sync(kFull, valid);
        for (int round = 0; have && round < 4; round++) {
            const int s0 = __shfl_sync(kFull, sys, __ffs(have) - 1);
            const bool mine = valid && sys == s0;
            have &= ~__ballot_sync(kFull, mine);
            double x = mine ? e : 0.0;
            for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(kFull, x, off);
            if ((threadIdx.x & 31) == 0) add(B, s0, x);
            if (mine) valid = false;
        }
        if (valid) add(B, sys, e);
    }
    // end of kernel: one atomic per warp when the warp holds one system
    __device__ void flush_warp(const BatchView& B) {
        const unsigned have = __ballot_sync(kFull, s >= 0);
        if (!have) return;
        const int s0 = __shfl_sync(kFull, s, __ffs(have) - 1);
        if (__all_sync(kFull, s < 0 || s == s0)) {
            double x = s >= 0 ? v : 0.0;
            for (int off = 16; off; off >>= 1) x += __shfl_xor_sync(kFull, x, off);
            if ((threadIdx.x & 31) == 0) atomicAdd(&B.ev[8 * s0], x);
        } else {
            flush(B);
        }
    }
};

// ---------------------------------------------------------------------------
// Per list entry: geometry, 1-body and 2-body terms, cutoffs and tables
// ---------------------------------------------------------------------------
__device__ __forceinline__ void put_pair(const DevParamSet& P, const PairTab& Q, double r, double rinv, double ex,
                                         int R, FxEnt* tab, double* scal) {
    double fc, fcd, gs;
    pair_setup_x(P, Q, r, ex, R, fx_kd(R), fc, fcd, gs, [&](int n, const Fx& t, const Fx& d) { tab[n] = fx_quad(t, d); });
    const int flags = (!less_pos(r, Q.rout) ? kPairFar : 0) | (less_pos(r, Q.rin) ? kPairOor : 0);
    reinterpret_cast<double2*>(scal)[0] = make_double2(fc, fc * gs * rinv);
    reinterpret_cast<double2*>(scal)[1] = make_double2(fcd * rinv, __hiloint2double(0, flags));
}

// The mixed form's pair-table cache: the values the cluster kernel would compute
// for a pair ij, ik or il, once per entry.
__device__ __forceinline__ void put_pair_f(const DevParamSet& P, const PairTab& Q, const double* dr, double r, double ex,
                                           int R, int rs, float* tab, double* g) {
    float fc, fcd;
    pair_setup<float>(P, Q, r, ex, tab, tab + rs, 1, R, fc, fcd, nullptr);
    for (int n = R; n < rs; n++) tab[n] = tab[rs + n] = 0.0f;
    PairCache& c = *reinterpret_cast<PairCache*>(g);
    c.d[0] = dr[0]; c.d[1] = dr[1]; c.d[2] = dr[2]; c.r = r;
    c.df[0] = narrow(dr[0]); c.df[1] = narrow(dr[1]); c.df[2] = narrow(dr[2]); c.rinv = 1.0f / narrow(r);
    c.fc = fc; c.fcd = fcd;
    c.flags = (!less_pos(r, Q.rout) ? kPairFar : 0) | (less_pos(r, Q.rin) ? kPairOor : 0);
    c.pad = 0.0f;
}

// Bound by the FP64 pipe (68%: geometry, the maps, forces; polynomial sums,
// exponential, sines, conversions and comparisons are integer arithmetic).  Measured:
// 5.23 M entries mixed 1.19 ms with the tables of both body orders (1.37 with FP64
// conversions and comparisons) and 0.40 ms for their forces, against 1.84 ms for
// a 2-body kernel and 0.59 ms for a pass over the 3-body tables alone.  rs3, rs4:
// stride of the tables of a body order, 0 for none.  (Entries one by one: with an atom's entries spread
// over eight lanes instead, 384 configurations took 941 us and not 456, the
// lanes' rounds being one long dependent chain each.)
template <bool MIXED>
__global__ void __launch_bounds__(128) k_pairs_x(BatchView B, const int* l2_owner, int rs3, int rs4) {
    const long long n2 = list_total(B);
    EAcc acc, acc1;   // 2-body, 1-body (an atom and an entry of the same number are mostly of different systems)
    const long long ntot = n2 > B.n_atoms_total ? n2 : B.n_atoms_total;
    // one contiguous range of entries per block, so that the energy changes system seldom
    const long long per = ((ntot + gridDim.x - 1) / gridDim.x + blockDim.x - 1) / blockDim.x * blockDim.x;
    const long long e_end = min(ntot, per * (blockIdx.x + 1));
    for (long long e = per * blockIdx.x + threadIdx.x; e < e_end; e += blockDim.x) {
        if (e < B.n_atoms_total) {   // compute_1B (chimesFF.cpp:1636-1641)
            const int s = B.atom_sys[e];
            acc1.add(B, s, B.psets[B.sys[s].pset].eoff[B.atom_type[e]]);
        }
        if (e >= n2) continue;
        const int a = l2_owner[e];
        const int s = B.atom_sys[a];
        const SysDesc& d = B.sys[s];
        const DevParamSet& P = B.psets[d.pset];
        const int gj = B.l2_ghost[e];
        int pt = P.pair_map[B.atom_type[a] * P.ntypes + B.atom_type[B.ghost_parent[gj]]];
        if (!ck_bound(B, pt >= 0 && pt < P.npairs)) pt = 0;
        const PairRec& pr = P.pairs[pt];
        double dr[3], r, rinv;
        sqrt_rcp(pair_vec(B, d.h, B.atom_self[a], gj, dr), r, rinv);
        const double ex = exp_neg(r * pr.inv_lam);
        double E = 0.0, fs = 0.0;
        if (less_pos(r, pr.rout)) {
            if (pr.fx_amp != 0.0) pair_2b_x(P, pr, r, rinv, ex, B.flags, E, fs);
            else pair_2b<double>(P, pr, r, B.flags, E, fs);
            acc.add(B, s, E);
        }
        reinterpret_cast<double2*>(B.pe + 4 * e)[0] = make_double2(dr[0], dr[1]);
        reinterpret_cast<double2*>(B.pe + 4 * e)[1] = make_double2(dr[2], fs);
        // (FP64: a pair jk of some cluster can lie at the cutoff itself, to rounding, in this list)
        const unsigned w = MIXED ? reinterpret_cast<const unsigned*>(B.l2_vec)[4 * e + 3] : 0u;
        if (rs3 > 0 && d.has3 && (MIXED ? (w & kL2In3) != 0 : less_pos(r, d.c3 + 1e-6))) {
            if (MIXED) put_pair_f(P, P.pt3[pt], dr, r, ex, P.R3, rs3, reinterpret_cast<float*>(B.pct3) + e * 2 * rs3, B.pcd3 + 8 * e);
            else put_pair(P, P.pt3[pt], r, rinv, ex, P.R3, reinterpret_cast<FxEnt*>(B.pct3) + e * rs3, B.pcd3 + 4 * e);
        }
        if (rs4 > 0 && d.has4 && (MIXED ? (w & kL2In4) != 0 : less_pos(r, d.c4 + 1e-6))) {
            if (MIXED) put_pair_f(P, P.pt4[pt], dr, r, ex, P.R4, rs4, reinterpret_cast<float*>(B.pct4) + e * 2 * rs4, B.pcd4 + 8 * e);
            else put_pair(P, P.pt4[pt], r, rinv, ex, P.R4, reinterpret_cast<FxEnt*>(B.pct4) + e * rs4, B.pcd4 + 4 * e);
        }
    }
    acc.flush_warp(B);
    acc1.flush_warp(B);
}

// Forces and virial of every list entry from its summed force scalar: eight
// lanes per atom, its entries in turn; the atom's own force is summed over the
// lanes, the neighbours' go out as atomics.
__global__ void __launch_bounds__(256) k_pair_forces(BatchView B) {
    const int gl = threadIdx.x & 7;
    const long long ngrp = (long long)gridDim.x * (blockDim.x / 8);
    const long long per = (B.n_atoms_total + ngrp - 1) / ngrp;
    const long long a0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 8 * per;
    EVAcc acc;
    for (long long k = 0; k < per; k++) {   // (all lanes of a warp make every round)
        const long long a = a0 + k;
        const bool have = a < B.n_atoms_total;
        long long b0 = 0, b1 = 0;
        if (have) list_range(B, a, b0, b1);
        double f[3] = {0.0, 0.0, 0.0};
        if (have) {
            const int s = B.atom_sys[a];
            if (s != acc.s) { acc.flush(B); acc.s = s; }
        }
        for (long long e = b0 + gl; e < b1; e += 8) {
            const double2 p = reinterpret_cast<const double2*>(B.pe + 4 * e)[0];
            const double2 q = reinterpret_cast<const double2*>(B.pe + 4 * e)[1];
            const double fs = q.y;
            if (__double_as_longlong(fs) << 1 == 0) continue;
            const double d[3] = {p.x, p.y, q.x}, g[3] = {fs * p.x, fs * p.y, fs * q.x};
            for (int c = 0; c < 3; c++) f[c] += g[c];
            add_force(B, B.l2_ghost[e], -g[0], -g[1], -g[2]);
            acc.v[1] -= g[0] * d[0];
            acc.v[2] -= g[0] * d[1];
            acc.v[3] -= g[0] * d[2];
            acc.v[4] -= g[1] * d[1];
            acc.v[5] -= g[1] * d[2];
            acc.v[6] -= g[2] * d[2];
        }
        for (int off = 4; off; off >>= 1)
            for (int c = 0; c < 3; c++) f[c] += __shfl_xor_sync(kFull, f[c], off);
        if (have && gl == 0) add_force(B, B.atom_self[a], f[0], f[1], f[2]);
    }
    acc.flush_warp(B);
}

// ---------------------------------------------------------------------------
// Set-up and finish of a tile
// ---------------------------------------------------------------------------
// Shared memory of a block (all of it dynamic: allow_max_smem's limit leaves
// no room for static arrays): the claimed tile, then interleaved
// [entry][cluster]
//   ENT:  double miss[NM * 4]         fc, fc gs / r, fc'/r, flags of pairs that no list holds
//   else: double geo[NP * 4], fc[NP], fcd[NP], gs[NP]
//   long long part[NW][NP + 1]        the warps' S and G
//   FxEnt  tab[NT * rs]               T and dT limbs (3-body ENT: pairs ik, jk; else all pairs)
template <int NB, int NW, bool ENT>
struct FxSmem {
    static constexpr int NP = Topo<NB>::NP;
    static constexpr int KC = NB - 1;                       // pairs of the first atom
    static constexpr int P0 = NB == 3 && ENT ? 1 : 0;       // first pair with a table here
    static constexpr int ND = ENT ? (NP - KC) * 4 : NP * 7;
    long long* tile;
    double* d;
    long long* part;
    FxEnt* tab;
    unsigned char* rest;
    __device__ FxSmem(unsigned char* smem, int rs) {
        tile = reinterpret_cast<long long*>(smem);
        d = reinterpret_cast<double*>(smem + 16);
        part = reinterpret_cast<long long*>(d + ND * kFxTile);
        tab = reinterpret_cast<FxEnt*>(part + NW * (NP + 1) * kFxTile);
        rest = reinterpret_cast<unsigned char*>(tab + (NP - P0) * rs * kFxTile);
    }
    __device__ FxEnt* table(int p, int rs) const { return tab + (p - P0) * rs * kFxTile; }
    static size_t bytes(int rs) {
        return 16 + sizeof(double) * (size_t)(ND + NW * (NP + 1)) * kFxTile +
               sizeof(FxEnt) * (size_t)(NP - P0) * rs * kFxTile;
    }
};

// ENT, cold path: a pair that its list does not hold (within rounding of the
// search radius): its tables and scalars from the atoms themselves.
template <int NB>
__device__ __noinline__ void missing_pair(const BatchView& B, const DevParamSet& P, const TupleRec& R, int p,
                                          const int* id, FxEnt* tab, double* scal) {
    const int s = B.atom_sys[B.ghost_parent[id[0]]];
    double dr[3], r, fc, fcd, gs;
    pair_geom(B, B.sys[s].h, id[Topo<NB>::a(p)], id[Topo<NB>::b(p)], dr, r);
    const int Rp = NB == 3 ? P.R3 : P.R4;
    const PairTab Q = tuple_pair(R, p);
    pair_setup_x(P, Q, r, exp_neg(r * Q.inv_lam), Rp, fx_kd(Rp), fc, fcd, gs,
                 [&](int n, const Fx& t, const Fx& d) { tab[n * kFxTile] = fx_quad(t, d); });
    scal[0] = fc;
    scal[kFxTile] = fc * gs / r;
    scal[2 * kFxTile] = fcd / r;
    scal[3 * kFxTile] = __hiloint2double(0, (!less_pos(r, Q.rout) ? kPairFar : 0) | (less_pos(r, Q.rin) ? kPairOor : 0));
}
__device__ __noinline__ void missing_force(const BatchView& B, int ga, int gb, int s, double fs) {
    double dr[3], r, vir[6] = {0, 0, 0, 0, 0, 0};
    pair_geom(B, B.sys[s].h, ga, gb, dr, r);
    add_force(B, ga, fs * dr[0], fs * dr[1], fs * dr[2]);
    add_force(B, gb, -fs * dr[0], -fs * dr[1], -fs * dr[2]);
    virial_add(vir, fs, dr);
    for (int k = 0; k < 6; k++) atomicAdd(&B.ev[8 * s + 1 + k], vir[k]);
}

// Tables of this lane's cluster c into shared memory, spread over the warps.
// ENT: gathered from the list entries ent[] (lanes without a cluster take entry
// 0; which clusters are evaluated is known at the finish).  Else computed;
// returns whether the cluster is evaluated (compute_3B/4B's early-outs).
template <int NB, int NW, bool ENT>
__device__ __forceinline__ bool fx_setup(const BatchView& B, const int* clusters, int c, const DevParamSet& P,
                                         const TupleRec& R, int rs, const FxSmem<NB, NW, ENT>& m, int* ent) {
    using M = FxSmem<NB, NW, ENT>;
    constexpr int NP = M::NP, KC = M::KC;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int Rp = NB == 3 ? P.R3 : P.R4;
    bool active = c >= 0;
    if constexpr (ENT) {
        const int* ce = NB == 3 ? B.c3e : B.c4e;
        const FxEnt* pct = reinterpret_cast<const FxEnt*>(NB == 3 ? B.pct3 : B.pct4);
#pragma unroll
        for (int p = 0; p < NP; p++) ent[p] = active ? ce[(long long)NP * c + p] : 0;
        // a warp takes every NW-th power of each pair, four loads in flight
#pragma unroll
        for (int p = M::P0; p < NP; p++) {
            const FxEnt* src = pct + (long long)(ent[p] < 0 ? 0 : ent[p]) * rs;
            FxEnt* dst = m.table(p, rs) + lane;
            for (int n0 = w; n0 < Rp; n0 += 4 * NW) {
                FxEnt t[4];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (n0 + k * NW < Rp) t[k] = src[n0 + k * NW];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (n0 + k * NW < Rp) dst[(n0 + k * NW) * kFxTile] = t[k];
            }
        }
        if (KC < NP) __syncthreads();   // (a missing pair's tables replace what was copied for it)
#pragma unroll
        for (int p = KC; p < NP; p++)
            if (ent[p] < 0 && w == 0) {
                int id[NB];
                for (int k = 0; k < NB; k++) id[k] = clusters[(long long)NB * c + k];
                missing_pair<NB>(B, P, R, p, id, m.table(p, rs) + lane, m.d + (p - KC) * 4 * kFxTile + lane);
            }
        __syncthreads();
    } else {
        double* geo = m.d;
        if (active) {
            int id[NB];
            for (int k = 0; k < NB; k++) id[k] = clusters[(long long)NB * c + k];
            const double* h = B.sys[B.atom_sys[B.ghost_parent[id[0]]]].h;
            for (int p = w; p < NP; p += NW) {
                double dr[3], r;
                pair_geom(B, h, id[Topo<NB>::a(p)], id[Topo<NB>::b(p)], dr, r);
                for (int k = 0; k < 3; k++) geo[(4 * p + k) * kFxTile + lane] = dr[k];
                geo[(4 * p + 3) * kFxTile + lane] = r;
            }
        }
        __syncthreads();
        if (active)
            for (int p = 0; p < NP; p++)
                if (geo[(4 * p + 3) * kFxTile + lane] >= R.rout[p]) active = false;
        if (active)
            for (int p = w; p < NP; p += NW) {
                FxEnt* tab = m.table(p, rs) + lane;
                const double r = geo[(4 * p + 3) * kFxTile + lane];
                const PairTab Q = tuple_pair(R, p);
                if (r < Q.rin) atomicAdd(&B.flags[4], 1);
                double fc, fcd, gs;
                pair_setup_x(P, Q, r, exp_neg(r * Q.inv_lam), Rp, fx_kd(Rp), fc, fcd, gs,
                             [&](int n, const Fx& t, const Fx& d) { tab[n * kFxTile] = fx_quad(t, d); });
                geo[(4 * NP + p) * kFxTile + lane] = fc;
                geo[(5 * NP + p) * kFxTile + lane] = fcd;
                geo[(6 * NP + p) * kFxTile + lane] = gs;
            }
        __syncthreads();
    }
    return active;
}

// The warps' parts of S and the G's (at 2^(kFxSum + ez)), added and turned into force scalars (ENT,
// added to the pairs' entries) or forces by warp 0.
//   f_p = (prod_{q != p} fc_q / r_p) (fc_p G_p + fc'_p S), E = prod fc S
template <int NB, int NW, bool ENT, typename Acc>
__device__ __forceinline__ void fx_finish(const BatchView& B, const int* clusters, int c,
                                          const FxSmem<NB, NW, ENT>& m, const TupleRec& R, bool active,
                                          const int* ent, const long long* own, const int* ez, Acc& acc) {
    constexpr int NP = Topo<NB>::NP;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (NW > 1) {
        for (int k = 0; k <= NP; k++) m.part[(w * (NP + 1) + k) * kFxTile + lane] = own[k];
        __syncthreads();
        if (w > 0) return;
    }
    double S, G[NP];
    for (int k = 0; k <= NP; k++) {
        long long v = own[k];
        for (int u = 1; u < NW; u++) v += m.part[(u * (NP + 1) + k) * kFxTile + lane];
        (k == 0 ? S : G[k - 1]) = from_fixed(v, -ez[k]);
    }
    const double unit = R.fx_amp * kFxUnit;
    int s = 0;
    if (active) s = B.atom_sys[B.ghost_parent[clusters[(long long)NB * c]]];
    if constexpr (ENT) {
        constexpr int KC = NB - 1;
        const double* pcd = NB == 3 ? B.pcd3 : B.pcd4;
        double fc[NP], ga[NP], ca[NP];
        int flags = 0, oor = 0;
#pragma unroll
        for (int p = 0; p < NP; p++) {
            double fl;
            if (p >= KC && ent[p] < 0) {
                const double* q = m.d + (p - KC) * 4 * kFxTile + lane;
                fc[p] = q[0]; ga[p] = q[kFxTile]; ca[p] = q[2 * kFxTile]; fl = q[3 * kFxTile];
            } else {
                const double2* q = reinterpret_cast<const double2*>(pcd + 4 * (long long)ent[p]);
                const double2 x = q[0], y = q[1];
                fc[p] = x.x; ga[p] = x.y; ca[p] = y.x; fl = y.y;
            }
            const int f = __double2loint(fl);
            flags |= f;
            oor += f & kPairOor ? 1 : 0;
        }
        active = active && !(flags & kPairFar);   // compute_3B/4B's early-outs
        double E = 0.0;
        if (active) {
            if (oor) atomicAdd(&B.flags[4], oor);
            double rest[NP];   // unit times the other pairs' cutoffs
            if constexpr (NB == 3) {
                const double u0 = unit * fc[0];
                rest[0] = unit * fc[1] * fc[2];
                rest[1] = u0 * fc[2];
                rest[2] = u0 * fc[1];
            } else {
                double suf = 1.0, pre = unit;
#pragma unroll
                for (int p = NP - 1; p > 0; p--) { rest[p] = suf; suf *= fc[p]; }
                rest[0] = suf * unit;
#pragma unroll
                for (int p = 1; p < NP; p++) { pre *= fc[p - 1]; rest[p] *= pre; }
            }
            E = rest[NP - 1] * fc[NP - 1] * S;
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const double fs = rest[p] * (ga[p] * G[p] + ca[p] * S);
                if (p >= KC && ent[p] < 0) {
                    const int* id = clusters + (long long)NB * c;
                    missing_force(B, id[Topo<NB>::a(p)], id[Topo<NB>::b(p)], s, fs);
                } else {
                    atomicAdd(&B.pe[4 * (long long)ent[p] + 3], fs);
                }
            }
        }
        acc.add_warp(B, s, E, active);
    } else if (active) {
        const double* geo = m.d;
        double dr[NP][4], fc[NP], fcd[NP];
        int id[NB];
        for (int k = 0; k < NB; k++) id[k] = clusters[(long long)NB * c + k];
        for (int p = 0; p < NP; p++) {
            for (int k = 0; k < 4; k++) dr[p][k] = geo[(4 * p + k) * kFxTile + lane];
            fc[p] = geo[(4 * NP + p) * kFxTile + lane];
            fcd[p] = geo[(5 * NP + p) * kFxTile + lane];
            G[p] *= unit * geo[(6 * NP + p) * kFxTile + lane];
        }
        cluster_epilogue<NB>(B, id, s, dr, fc, fcd, S * unit, G, acc);
    }
}

// Claims the block's next tile (thread 0) and returns it to all threads; also
// the barrier between two tiles' uses of the shared memory.
__device__ __forceinline__ long long fx_claim(unsigned long long* head, long long* slot) {
    if (threadIdx.x == 0) *slot = (long long)atomicAdd(head, 1ull);
    __syncthreads();
    const long long t = *slot;
    __syncthreads();
    return t;
}

template <bool ENT>
struct AccOf {
    using type = EVAcc;
};
template <>
struct AccOf<true> {
    using type = EAcc;
};

// ---------------------------------------------------------------------------
// 3-body.  X = T_ij and the row sums z stay in registers (RX powers, unrolled;
// a column's mask says which groups of two it has), Y_J is formed per column,
// and the column sums w_J are folded over q_jk within a run of q_ik.
// ---------------------------------------------------------------------------
// 16 warps per SM (128 registers): 384 configurations 1.70 -> 1.61 ms for the
// stage; all groups' loads ahead of the masked sums and not inside them, and
// plain masks against unmasked sums over zeros, measured the same.
template <int RX, int NW, bool ENT>
__global__ void __launch_bounds__(32 * NW, RX <= 10 ? 16 / NW : 1) k_forcex3(BatchView B, const int* clusters, const int* perm,
                                                     const long long* perm_n, long long perm_cap, int rs) {
    extern __shared__ __align__(16) unsigned char smem[];
    const FxSmem<3, NW, ENT> m(smem, rs);
    FxEnt* strm = reinterpret_cast<FxEnt*>(m.rest);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ntiles = min(*perm_n, perm_cap) / kFxTile;
    int loaded = -1;
    const DevParamSet* loaded_set = nullptr;
    typename AccOf<ENT>::type acc;
    for (;;) {
        const long long tile = fx_claim(&B.queue[0], m.tile);
        if (tile >= ntiles) break;
        const long long base = tile * kFxTile;
        const int c0 = perm[base];
        if (c0 < 0) continue;   // uniform: a tile never starts in a bucket's padding
        int id0[3], s0, u, ent[3];
        const DevParamSet* P;
        const TupleRec* R = cluster_tuple<3>(B, clusters, c0, id0, s0, P, u);
        constexpr int CL = 1 + RX / 2;   // a column here: header, then every group
        const int cl = 1 + (P->R3 + 1) / 2;   // and as stored
        int ncol = R->fx_split[8] / cl;
        if (!ck_bound(B, R->fx_off >= 0 && R->fx_off + (long long)R->fx_split[8] <= P->n_fx3)) ncol = 0;
        if (R->fx_off != loaded || P != loaded_set) {
            for (int q = threadIdx.x; q < ncol * CL; q += 32 * NW) {
                const int col = q / CL, k = q % CL;
                strm[q] = k < cl ? P->fx3[R->fx_off + col * cl + k] : FxEnt{0, 0, 0, 0};
            }
            loaded = R->fx_off;
            loaded_set = P;
        }
        const int c = perm[base + lane];
        const bool active = fx_setup<3, NW, ENT>(B, clusters, c, *P, *R, rs, m, ent);
        const int Rp = P->R3;
        const FxEnt* t0 = ENT ? reinterpret_cast<const FxEnt*>(B.pct3) + (long long)ent[0] * rs : m.table(0, rs) + lane;
        constexpr int st0 = ENT ? 1 : kFxTile;
        const FxEnt *t1 = m.table(1, rs) + lane, *t2 = m.table(2, rs) + lane;
        Fx X[RX];
        FxRec z[RX];
#pragma unroll
        for (int q = 0; q < RX; q++) X[q] = q < Rp ? quad_t(t0 + q * st0) : Fx{0, 0};
        FxAcc g1, g2, ca, cb;
        FxEnt tb{0, 0, 0, 0};
        int qb = -1;
        int o = ncol ? R->fx_split[8 * w / NW] / cl * CL : 0;
        const int o1 = ncol ? R->fx_split[8 * (w + 1) / NW] / cl * CL : 0;
        for (; o < o1; o += 1 + RX / 2) {
            const FxEnt hd = strm[o];
            FxEnt a[RX / 2];
#pragma unroll
            for (int g = 0; g < RX / 2; g++) a[g] = strm[o + 1 + g];
            const FxEnt tc = t2[hd.y * kFxTile];
            if (hd.x != qb) {   // uniform: a new run of q_ik
                g1.mac(Fx{tb.z, tb.w}, ca.value());
                g2.mac(Fx{tb.x, tb.y}, cb.value());
                ca = FxAcc();
                cb = FxAcc();
                tb = t1[hd.x * kFxTile];
                qb = hd.x;
            }
            const Fx Y = fx_mul(Fx{tb.x, tb.y}, Fx{tc.x, tc.y});
            FxRec wj;
#pragma unroll
            for (int g = 0; g < RX / 2; g++)
                if (hd.z & (1 << g)) {   // uniform
                    wj.mac(Fx{a[g].x, a[g].y}, X[2 * g]);
                    wj.mac(Fx{a[g].z, a[g].w}, X[2 * g + 1]);
                    z[2 * g].mac(Fx{a[g].x, a[g].y}, Y);
                    z[2 * g + 1].mac(Fx{a[g].z, a[g].w}, Y);
                }
            const Fx wv = wj.value();
            ca.mac(Fx{tc.x, tc.y}, wv);
            cb.mac(Fx{tc.z, tc.w}, wv);
        }
        g1.mac(Fx{tb.z, tb.w}, ca.value());
        g2.mac(Fx{tb.x, tb.y}, cb.value());
        FxAcc S, g0;
#pragma unroll
        for (int q = 0; q < RX; q++)
            if (q < Rp) {
                const FxEnt t = t0[q * st0];
                const Fx zv = z[q].value();
                S.mac(Fx{t.x, t.y}, zv);
                g0.mac(Fx{t.z, t.w}, zv);
            }
        const long long own[4] = {S.sum(), g0.sum(), g1.sum(), g2.sum()};
        constexpr int ez[4] = {kFxZ3, kFxZ3 + kFxDer, kFxZ3 + kFxDer, kFxZ3 + kFxDer};
        fx_finish<3, NW, ENT>(B, clusters, c, m, *R, active, ent, own, ez, acc);
    }
    if (w == 0) acc.flush_warp(B);
}

// ---------------------------------------------------------------------------
// 4-body
// ---------------------------------------------------------------------------
// One side: the records [o, o1) of its stream, V the other side's products, t
// the side's three pair tables.  The record sums are folded over the last
// pair's power, then the middle one's, then the first one's, as their records
// are sorted: out[0] = sum_I X_I z_I, out[1..3] = the three pairs' gradients.
__device__ __forceinline__ void fx_side(const FxEnt* __restrict__ ent, int o, int o1, const FxPair* V, const FxEnt* t,
                                        int rs, int fz, long long* out) {
    const FxEnt *t1 = t + rs * kFxTile, *t2 = t1 + rs * kFxTile;
    const FxCut cr(fx_zget(fz, kFxZr));
    FxAcc S, g0, g1, g2, ra, rb, rP, rQ, rR;
    int q0 = -1, q1 = -1;
    auto fold1 = [&]() {
        if (q1 < 0) return;
        const Fx a = ra.value(fx_zget(fz, kFxZr) - fx_zget(fz, kFxZra)),
                 b = rb.value(fx_zget(fz, kFxZr) + kFxDer - fx_zget(fz, kFxZrb));
        const FxEnt v = t1[q1 * kFxTile];
        rP.mac(Fx{v.x, v.y}, a);
        rQ.mac(Fx{v.z, v.w}, a);
        rR.mac(Fx{v.x, v.y}, b);
        ra = FxAcc();
        rb = FxAcc();
    };
    auto fold0 = [&]() {
        if (q0 < 0) return;
        const Fx p = rP.value(fx_zget(fz, kFxZra) - fx_zget(fz, kFxZP));
        const FxEnt v = t[q0 * kFxTile];
        S.mac(Fx{v.x, v.y}, p);
        g0.mac(Fx{v.z, v.w}, p);
        g1.mac(Fx{v.x, v.y}, rQ.value(fx_zget(fz, kFxZra) + kFxDer - fx_zget(fz, kFxZQ)));
        g2.mac(Fx{v.x, v.y}, rR.value(fx_zget(fz, kFxZrb) - fx_zget(fz, kFxZR)));
        rP = FxAcc();
        rQ = FxAcc();
        rR = FxAcc();
    };
    FxRec z(cr);
    FxEnt q[4], n[4];
#pragma unroll
    for (int k = 0; k < 4; k++) q[k] = ent[o + k];   // (a side without entries reads its neighbour's: in bounds)
    while (o < o1) {
        o += 4;
        if (o < o1) {
#pragma unroll
            for (int k = 0; k < 4; k++) n[k] = ent[o + k];   // the next four in flight
        }
#pragma unroll
        for (int k = 0; k < 4; k++) z.mac(Fx{q[k].x, q[k].y}, fx_load(V[q[k].z * kFxTile]));
        const int pows = q[3].w;
        if (pows >= 0) {   // uniform: the record's end
            const int r0 = pows & 31, r1 = (pows >> kPowBits) & 31, r2 = (pows >> (2 * kPowBits)) & 31;
            if (r0 != q0 || r1 != q1) {
                fold1();
                if (r0 != q0) fold0();
                q0 = r0;
                q1 = r1;
            }
            const Fx zv = z.value(cr);
            const FxEnt v = t2[r2 * kFxTile];
            ra.mac(Fx{v.x, v.y}, zv);
            rb.mac(Fx{v.z, v.w}, zv);
            z = FxRec(cr);
        }
#pragma unroll
        for (int k = 0; k < 4; k++) q[k] = n[k];
    }
    fold1();
    fold0();
    out[0] = S.sum();
    out[1] = g0.sum();
    out[2] = g1.sum();
    out[3] = g2.sum();
}

// With one warp it takes the rows, then the columns; with more, half of the
// warps take the rows and half the columns.
template <int NW, bool ENT>
__global__ void __launch_bounds__(32 * NW, NW > 1 ? (ENT ? 16 : 12) / NW : 1) k_forcex4(BatchView B, const int* clusters, const int* perm,
                                                     const long long* perm_n, long long perm_cap, int rs) {
    extern __shared__ __align__(16) unsigned char smem[];
    const FxSmem<4, NW, ENT> m(smem, rs);
    FxPair* X = reinterpret_cast<FxPair*>(m.rest);
    FxPair* Y = X + rs * rs * rs * kFxTile;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ntiles = min(*perm_n, perm_cap) / kFxTile;
    typename AccOf<ENT>::type acc;
    for (;;) {
        const long long tile = fx_claim(&B.queue[1], m.tile);
        if (tile >= ntiles) break;
        const long long base = tile * kFxTile;
        const int c0 = perm[base];
        if (c0 < 0) continue;   // uniform
        int id0[4], s0, u, ent6[6];
        const DevParamSet* P;
        const TupleRec* R = cluster_tuple<4>(B, clusters, c0, id0, s0, P, u);
        const int c = perm[base + lane];
        const bool active = fx_setup<4, NW, ENT>(B, clusters, c, *P, *R, rs, m, ent6);
        const int Rp = P->R4;
        const FxEnt* T = m.tab + lane;
        // the products X_I, Y_J: the first two pairs' product per (q0, q1), spread over the warps
        for (int k = w; k < 2 * Rp * Rp; k += NW) {
            const int side = k >= Rp * Rp ? 1 : 0, q01 = k - side * Rp * Rp;
            const FxEnt* t = T + 3 * side * rs * kFxTile;
            const Fx v = fx_mul(quad_t(t + (q01 / Rp) * kFxTile), quad_t(t + (rs + q01 % Rp) * kFxTile));
            FxPair* dst = (side ? Y : X) + q01 * Rp * kFxTile + lane;
            for (int q = 0; q < Rp; q++) dst[q * kFxTile] = fx_store(fx_mul(v, quad_t(t + (2 * rs + q) * kFxTile)));
        }
        __syncthreads();
        const bool ok = ck_bound(B, R->fx_off >= 0 && R->fx_off + (long long)R->fx_split[8] <= P->n_fx4);
        const FxEnt* ent = P->fx4 + R->fx_off;
        const int* fz = R->fx_z;
        long long own[7] = {0, 0, 0, 0, 0, 0, 0};
        if (NW == 1) {
            long long b[4];
            fx_side(ent, ok ? R->fx_split[0] : 0, ok ? R->fx_split[4] : 0, Y + lane, T, rs, fz[0], own);
            fx_side(ent, ok ? R->fx_split[4] : 0, ok ? R->fx_split[8] : 0, X + lane, T + 3 * rs * kFxTile, rs, fz[1], b);
            for (int k = 1; k < 4; k++) own[3 + k] = b[k];
        } else {
            constexpr int H = NW > 1 ? NW / 2 : 1;   // warps per side
            const int side = w / H, k0 = 4 * side + 4 * (w % H) / H, k1 = 4 * side + 4 * (w % H + 1) / H;
            long long a[4];
            fx_side(ent, ok ? R->fx_split[k0] : 0, ok ? R->fx_split[k1] : 0, (side ? X : Y) + lane,
                    T + 3 * side * rs * kFxTile, rs, fz[side], a);
            own[0] = side ? 0 : a[0];
            for (int k = 1; k < 4; k++) {
                own[k] = side ? 0 : a[k];
                own[3 + k] = side ? a[k] : 0;
            }
        }
        int ez[7];
        ez[0] = fx_zget(fz[0], kFxZP);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            ez[1 + 3 * k] = fx_zget(fz[k], kFxZP) + kFxDer;
            ez[2 + 3 * k] = fx_zget(fz[k], kFxZQ);
            ez[3 + 3 * k] = fx_zget(fz[k], kFxZR);
        }
        fx_finish<4, NW, ENT>(B, clusters, c, m, *R, active, ent6, own, ez, acc);
    }
    if (w == 0) acc.flush_warp(B);
}

unsigned fx_grid(const void* kern, int threads, size_t smem, long long tiles) {
    allow_max_smem(kern);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem);
    const long long want = (long long)sm_count() * (occ > 0 ? occ : 1);
    return (unsigned)(want < tiles ? want : tiles);
}

template <int RX, int NW, bool ENT>
void launch_x3(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    const int rs = L.rf3;
    const size_t smem = FxSmem<3, NW, ENT>::bytes(rs) + sizeof(FxEnt) * (size_t)L.xs3 * (1 + RX / 2);
    auto kern = k_forcex3<RX, NW, ENT>;
    const unsigned grid = fx_grid((const void*)kern, 32 * NW, smem, (B.perm3_cap + kFxTile - 1) / kFxTile);
    count_launch(), kern<<<grid, 32 * NW, smem, st>>>(B, B.c3, B.perm3, B.bk_start + B.nbk3, B.perm3_cap, rs);
}

template <int NW, bool ENT>
void launch_x3_nw(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (L.rf3 <= 4) launch_x3<4, NW, ENT>(B, L, st);
    else if (L.rf3 <= 8) launch_x3<8, NW, ENT>(B, L, st);
    else if (L.rf3 <= 10) launch_x3<10, NW, ENT>(B, L, st);
    else launch_x3<12, NW, ENT>(B, L, st);
}

template <int NW, bool ENT>
void launch_x4_nw(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    const int rs = L.rf4;
    const size_t smem = FxSmem<4, NW, ENT>::bytes(rs) + sizeof(FxPair) * (size_t)2 * rs * rs * rs * kFxTile;
    auto kern = k_forcex4<NW, ENT>;
    const unsigned grid = fx_grid((const void*)kern, 32 * NW, smem, (B.perm4_cap + kFxTile - 1) / kFxTile);
    count_launch(), kern<<<grid, 32 * NW, smem, st>>>(B, B.c4, B.perm4, B.bk_start + B.nbk3 + 1 + B.nbk4,
                                                       B.perm4_cap, rs);
}

template <bool ENT>
void launch_x3_ent(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    switch (L.xw3) {
        case 1: launch_x3_nw<1, ENT>(B, L, st); break;
        case 2: launch_x3_nw<2, ENT>(B, L, st); break;
        case 4: launch_x3_nw<4, ENT>(B, L, st); break;
        default: launch_x3_nw<8, ENT>(B, L, st); break;
    }
}

template <bool ENT>
void launch_x4_ent(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    switch (L.xw4) {
        case 1: launch_x4_nw<1, ENT>(B, L, st); break;
        case 2: launch_x4_nw<2, ENT>(B, L, st); break;
        case 4: launch_x4_nw<4, ENT>(B, L, st); break;
        default: launch_x4_nw<8, ENT>(B, L, st); break;
    }
}

}  // namespace

void launch_pairs(const BatchView& B, const int* l2_owner, const ForceLaunch& L, cudaStream_t st) {
    const long long ntot = B.n2_cap > B.n_atoms_total ? B.n2_cap : B.n_atoms_total;
    if (ntot <= 0) return;
    const long long want = (long long)sm_count() * 12, need = (ntot + 127) / 128;
    const unsigned grid = (unsigned)(want < need ? want : need);
    if (L.precision == kMixed) {
        count_launch(), k_pairs_x<true><<<grid, 128, 0, st>>>(B, l2_owner, B.use_pc3 ? L.rf3 : 0, B.use_pc4 ? L.rf4 : 0);
    } else {
        const bool ent = B.all_pairs;
        count_launch(), k_pairs_x<false><<<grid, 128, 0, st>>>(B, l2_owner, ent && B.nbk3 > 0 ? L.rf3 : 0,
                                                             ent && B.nbk4 > 0 ? L.rf4 : 0);
    }
}

void launch_pair_forces(const BatchView& B, cudaStream_t st) {
    if (B.n_atoms_total <= 0) return;
    const long long want = (long long)sm_count() * 6, need = (B.n_atoms_total + 31) / 32;
    count_launch(), k_pair_forces<<<(unsigned)(want < need ? want : need), 256, 0, st>>>(B);
}

void launch_force3x(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm3_cap <= 0 || B.nbk3 <= 0 || L.rf3 <= 0) return;
    if (B.all_pairs) launch_x3_ent<true>(B, L, st);
    else launch_x3_ent<false>(B, L, st);
}

void launch_force4x(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm4_cap <= 0 || B.nbk4 <= 0 || L.rf4 <= 0) return;
    if (B.all_pairs) launch_x4_ent<true>(B, L, st);
    else launch_x4_ent<false>(B, L, st);
}

}  // namespace ck
