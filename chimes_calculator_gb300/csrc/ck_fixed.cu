// 3-body and 4-body contraction of the FP64 form in 64-bit fixed point
// (arithmetic in ck_fixed.cuh, coefficient streams in ck_common.h).
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
// Everything is linear in the parts' sums; warp 0 adds them and forms the
// forces in FP64.
//
// Measured (GB300, 384 configurations of 8-512 atoms, 12/10/4, 1.81 M triplets
// and 358 k quadruplets; against the factored FP64 kernels this replaces):
// 3-body 5.91 -> 3.27 ms, 4-body 3.12 -> 1.63 ms; 1024 atoms 12/8/4: 131 -> 80
// and 132 -> 117 us.  The contraction no longer bounds them; the FP64 set-up of
// the pairs that the cache does not hold, the FP64 epilogue and the latency
// of both do.
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

__device__ __forceinline__ PairTab tuple_pair_x(const TupleRec& R, int p) {
    return PairTab{R.rin[p], R.rout[p], R.xavg[p], R.xdiff[p], R.inv_lam[p], R.inv_xdiff[p], R.fc_th[p], R.fc_inv[p]};
}

// Pair-table cache of the FP64 form: for every list entry closer than the
// body order's largest outer cutoff, the pair's geometry, cutoff and tables
// with the pair type's constants, once per entry instead of once per cluster.
// pcd[e][8] = dr0 dr1 dr2 r fc fc' oor gs; pct[e][2 rs] = T, then dT limbs.
template <int NB>
__global__ void __launch_bounds__(256) k_pair_tables_x(BatchView B, const int* l2_owner, int rs) {
    const long long n2 = min(B.l2_off[B.n_atoms_total], B.n2_cap);
    double* pcd = NB == 3 ? B.pcd3 : B.pcd4;
    FxPair* pct = reinterpret_cast<FxPair*>(NB == 3 ? B.pct3 : B.pct4);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n2; e += stride) {
        const int r = l2_owner[e];
        const SysDesc& d = B.sys[B.atom_sys[r]];
        if (!(NB == 3 ? d.has3 : d.has4) || B.l2_dist[e] >= (NB == 3 ? d.c3 : d.c4)) continue;
        const DevParamSet& P = B.psets[d.pset];
        const int gi = B.atom_self[r], gj = B.l2_ghost[e];
        double dr[3], rr;
        pair_geom(B, d.h, gi, gj, dr, rr);
        const int pt = P.pair_map[B.atom_type[r] * P.ntypes + B.atom_type[B.ghost_parent[gj]]];
        const PairTab& Q = (NB == 3 ? P.pt3 : P.pt4)[pt];
        const int Rp = NB == 3 ? P.R3 : P.R4;
        double fc, fcd, gs;
        FxPair* T = pct + (size_t)e * 2 * rs;
        pair_setup_x(P, Q, rr, T, T + rs, 1, Rp, fx_kd(Rp), fc, fcd, gs, nullptr);
        double* g = pcd + 8 * e;
        g[0] = dr[0]; g[1] = dr[1]; g[2] = dr[2]; g[3] = rr;
        g[4] = fc; g[5] = fcd; g[6] = rr < Q.rin ? 1.0 : 0.0; g[7] = gs;
    }
}

// Shared memory of a block (all of it dynamic: allow_max_smem's limit leaves
// no room for static arrays), the claimed tile, then interleaved [entry][cluster]:
//   double geo[NP * 4], fc[NP], fcd[NP], gs[NP], part[NW][NP + 1]
//   FxPair   T[NP * rs], D[NP * rs]
template <int NB, int NW>
struct FxSmem {
    static constexpr int NP = Topo<NB>::NP;
    long long* tile;
    double *geo, *fc, *fcd, *gs, *part;
    FxPair *T, *D, *rest;
    __device__ FxSmem(unsigned char* smem, int rs) {
        tile = reinterpret_cast<long long*>(smem);
        geo = reinterpret_cast<double*>(smem + 16);
        fc = geo + NP * 4 * kFxTile;
        fcd = fc + NP * kFxTile;
        gs = fcd + NP * kFxTile;
        part = gs + NP * kFxTile;
        T = reinterpret_cast<FxPair*>(part + NW * (NP + 1) * kFxTile);
        D = T + NP * rs * kFxTile;
        rest = D + NP * rs * kFxTile;
    }
    static size_t bytes(int rs) {
        return 16 + sizeof(double) * (size_t)(NP * 7 + NW * (NP + 1)) * kFxTile + sizeof(FxPair) * (size_t)2 * NP * rs * kFxTile;
    }
};

// Geometry, cutoffs and tables of this lane's cluster c, its pairs spread over
// the block's warps; pairs ij, ik[, il] from the cache when there is one.
// Returns whether the cluster is evaluated (compute_3B/4B's early-outs).
template <int NB, int NW>
__device__ __forceinline__ bool fx_setup(const BatchView& B, const int* clusters, int c, const DevParamSet& P,
                                         const TupleRec& R, int rs, const FxSmem<NB, NW>& m, int* id, int& s) {
    constexpr int NP = Topo<NB>::NP, KC = NB - 1;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool use_pc = NB == 3 ? B.use_pc3 : B.use_pc4;
    const int* ce = NB == 3 ? B.c3e : B.c4e;
    const double* pcd = NB == 3 ? B.pcd3 : B.pcd4;
    const FxPair* pct = reinterpret_cast<const FxPair*>(NB == 3 ? B.pct3 : B.pct4);
    const int Rp = NB == 3 ? P.R3 : P.R4;
    bool active = c >= 0;
    s = 0;
    if (active) {
        for (int k = 0; k < NB; k++) id[k] = clusters[(long long)NB * c + k];
        s = B.atom_sys[B.ghost_parent[id[0]]];
        const double* h = B.sys[s].h;
        for (int sl = w; sl < NP; sl += NW) {
            // with the cache the evaluated pairs come first, spread over the warps
            const int p = use_pc ? (sl < NP - KC ? KC + sl : sl - (NP - KC)) : sl;
            double dr[3], r;
            if (use_pc && p < KC) {
                const double* g = pcd + 8 * (long long)ce[(long long)KC * c + p];
                dr[0] = g[0]; dr[1] = g[1]; dr[2] = g[2]; r = g[3];
            } else {
                pair_geom(B, h, id[Topo<NB>::a(p)], id[Topo<NB>::b(p)], dr, r);
            }
            m.geo[(4 * p + 0) * kFxTile + lane] = dr[0];
            m.geo[(4 * p + 1) * kFxTile + lane] = dr[1];
            m.geo[(4 * p + 2) * kFxTile + lane] = dr[2];
            m.geo[(4 * p + 3) * kFxTile + lane] = r;
        }
    }
    __syncthreads();
    if (active)
        for (int p = 0; p < NP; p++)
            if (m.geo[(4 * p + 3) * kFxTile + lane] >= R.rout[p]) active = false;
    if (active)
        for (int sl = w; sl < NP; sl += NW) {
            const int p = use_pc ? (sl < NP - KC ? KC + sl : sl - (NP - KC)) : sl;
            FxPair* T = m.T + p * rs * kFxTile + lane;
            FxPair* D = m.D + p * rs * kFxTile + lane;
            double fc, fcd, gs;
            if (use_pc && p < KC) {
                const long long ent = ce[(long long)KC * c + p];
                const double* g = pcd + 8 * ent;
                const FxPair* tab = pct + ent * 2 * rs;
                for (int n = 0; n < Rp; n++) {
                    T[n * kFxTile] = tab[n];
                    D[n * kFxTile] = tab[rs + n];
                }
                fc = g[4];
                fcd = g[5];
                gs = g[7];
                if (g[6] != 0.0) atomicAdd(&B.flags[4], 1);
            } else {
                pair_setup_x(P, tuple_pair_x(R, p), m.geo[(4 * p + 3) * kFxTile + lane], T, D, kFxTile, Rp, fx_kd(Rp),
                             fc, fcd, gs, B.flags);
            }
            m.fc[p * kFxTile + lane] = fc;
            m.fcd[p * kFxTile + lane] = fcd;
            m.gs[p * kFxTile + lane] = gs;
        }
    __syncthreads();
    return active;
}

// The warps' parts of S and the G's, added and turned into forces by warp 0.
template <int NB, int NW>
__device__ __forceinline__ void fx_finish(const BatchView& B, const FxSmem<NB, NW>& m, const TupleRec& R, bool active,
                                          const int* id, int s, EVAcc& acc) {
    constexpr int NP = Topo<NB>::NP;
    const int lane = threadIdx.x & 31;
    if (NW > 1) __syncthreads();
    if (threadIdx.x < 32 && active) {
        double S = 0.0, dr[NP][4], fc[NP], fcd[NP], G[NP];
        for (int w = 0; w < NW; w++) S += m.part[w * (NP + 1) * kFxTile + lane];
        for (int p = 0; p < NP; p++) {
            double g = 0.0;
            for (int w = 0; w < NW; w++) g += m.part[(w * (NP + 1) + 1 + p) * kFxTile + lane];
            G[p] = g * m.gs[p * kFxTile + lane] * R.fx_amp;
            for (int k = 0; k < 4; k++) dr[p][k] = m.geo[(4 * p + k) * kFxTile + lane];
            fc[p] = m.fc[p * kFxTile + lane];
            fcd[p] = m.fcd[p * kFxTile + lane];
        }
        cluster_epilogue<NB>(B, id, s, dr, fc, fcd, S * R.fx_amp, G, acc);
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

// 3-body.  X = T_ij and the row sums z stay in registers (RX powers, unrolled;
// a column's mask says which of them it has), Y_J is formed per column, and
// the column sums w_J are folded over q_jk within a run of q_ik.
template <int RX, int NW>
__global__ void __launch_bounds__(32 * NW) k_forcex3(BatchView B, const int* clusters, const int* perm,
                                                     const long long* perm_n, long long perm_cap, int rs) {
    extern __shared__ __align__(16) unsigned char smem[];
    const FxSmem<3, NW> m(smem, rs);
    FxEnt* strm = reinterpret_cast<FxEnt*>(m.rest);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ntiles = min(*perm_n, perm_cap) / kFxTile;
    int loaded = -1;
    const DevParamSet* loaded_set = nullptr;
    EVAcc acc;
    for (;;) {
        const long long tile = fx_claim(&B.queue[0], m.tile);
        if (tile >= ntiles) break;
        const long long base = tile * kFxTile;
        const int c0 = perm[base];
        if (c0 < 0) continue;   // uniform: a tile never starts in a bucket's padding
        int id[3], s, u;
        const DevParamSet* P;
        const TupleRec* R = cluster_tuple<3>(B, clusters, c0, id, s, P, u);
        int len = R->fx_split[8];
        if (!ck_bound(B, R->fx_off >= 0 && R->fx_off + (long long)len <= P->n_fx3)) len = 0;
        if (R->fx_off != loaded || P != loaded_set) {
            for (int q = threadIdx.x; q < len; q += 32 * NW) strm[q] = P->fx3[R->fx_off + q];
            loaded = R->fx_off;
            loaded_set = P;
        }
        const bool active = fx_setup<3, NW>(B, clusters, perm[base + lane], *P, *R, rs, m, id, s);
        const int Rp = P->R3;
        const FxPair *T0 = m.T + lane, *T1 = T0 + rs * kFxTile, *T2 = T1 + rs * kFxTile;
        const FxPair *D0 = m.D + lane, *D1 = D0 + rs * kFxTile, *D2 = D1 + rs * kFxTile;
        Fx X[RX];
        FxAcc z[RX];
#pragma unroll
        for (int q = 0; q < RX; q++) X[q] = q < Rp ? fx_load(T0[q * kFxTile]) : Fx{0, 0};
        FxAcc g1, g2, ca, cb;
        Fx tb{0, 0}, db{0, 0};
        int qb = -1;
        int o = len ? R->fx_split[8 * w / NW] : 0;
        const int o1 = len ? R->fx_split[8 * (w + 1) / NW] : 0;
        FxEnt hd = strm[o];   // (the buffer has room for a header past the stream)
        while (o < o1) {
            const int b = hd.x, c = hd.y, mask = hd.z;
            const FxEnt* q4 = strm + o + 1;
            o += 1 + __popc(mask);
            hd = strm[o];
            if (b != qb) {   // uniform: a new run of q_ik
                g1.mac(db, ca.value<0>());
                g2.mac(tb, cb.value<0>());
                ca = FxAcc();
                cb = FxAcc();
                tb = fx_load(T1[b * kFxTile]);
                db = fx_load(D1[b * kFxTile]);
                qb = b;
            }
            const Fx tc = fx_load(T2[c * kFxTile]), dc = fx_load(D2[c * kFxTile]);
            const Fx Y = fx_mul(tb, tc);
            FxAcc wj;
#pragma unroll
            for (int g = 0; g < RX / 2; g++)
                if (mask & (1 << g)) {   // uniform
                    const FxEnt a = *q4++;
                    wj.mac(Fx{a.x, a.y}, X[2 * g]);
                    wj.mac(Fx{a.z, a.w}, X[2 * g + 1]);
                    z[2 * g].mac(Fx{a.x, a.y}, Y);
                    z[2 * g + 1].mac(Fx{a.z, a.w}, Y);
                }
            const Fx wv = wj.value<kFxDown>();
            ca.mac(tc, wv);
            cb.mac(dc, wv);
        }
        g1.mac(db, ca.value<0>());
        g2.mac(tb, cb.value<0>());
        FxAcc S, g0;
#pragma unroll
        for (int q = 0; q < RX; q++)
            if (q < Rp) {
                const Fx zv = z[q].template value<kFxDown>();
                S.mac(X[q], zv);
                g0.mac(fx_load(D0[q * kFxTile]), zv);
            }
        double* part = m.part + w * 4 * kFxTile + lane;
        part[0 * kFxTile] = S.real(kFxUnit);
        part[1 * kFxTile] = g0.real(kFxUnit);
        part[2 * kFxTile] = g1.real(kFxUnit);
        part[3 * kFxTile] = g2.real(kFxUnit);
        fx_finish<3, NW>(B, m, *R, active, id, s, acc);
    }
    if (w == 0) acc.flush_warp(B);
}

// One side of the 4-body contraction: the entries [o, o1) of its stream, V the
// other side's products, t / d the side's three pair tables.  The record sums
// are folded over the last pair's power, then the middle one's, then the
// first one's, as their records are sorted: out[0] = sum_I X_I z_I, out[1..3]
// = the three pairs' gradients.
__device__ __forceinline__ void fx_side(const FxEnt* __restrict__ ent, int o, int o1, const FxPair* V, const FxPair* t,
                                        const FxPair* d, int rs, double* out) {
    const FxPair *t1 = t + rs * kFxTile, *t2 = t1 + rs * kFxTile, *d1 = d + rs * kFxTile, *d2 = d1 + rs * kFxTile;
    FxAcc S, g0, g1, g2, ra, rb, rP, rQ, rR;
    int q0 = -1, q1 = -1;
    auto fold1 = [&]() {
        if (q1 < 0) return;
        const Fx a = ra.value<0>(), b = rb.value<0>(), tv = fx_load(t1[q1 * kFxTile]);
        rP.mac(tv, a);
        rQ.mac(fx_load(d1[q1 * kFxTile]), a);
        rR.mac(tv, b);
        ra = FxAcc();
        rb = FxAcc();
    };
    auto fold0 = [&]() {
        if (q0 < 0) return;
        const Fx p = rP.value<0>(), tv = fx_load(t[q0 * kFxTile]);
        S.mac(tv, p);
        g0.mac(fx_load(d[q0 * kFxTile]), p);
        g1.mac(tv, rQ.value<0>());
        g2.mac(tv, rR.value<0>());
        rP = FxAcc();
        rQ = FxAcc();
        rR = FxAcc();
    };
    while (o < o1) {
        const FxEnt hd = ent[o++];
        FxAcc z;
        for (const int end = o + 4 * hd.x; o < end; o += 4) {
            FxEnt q[4];
#pragma unroll
            for (int k = 0; k < 4; k++) q[k] = ent[o + k];
#pragma unroll
            for (int k = 0; k < 4; k++) z.mac(Fx{q[k].x, q[k].y}, fx_load(V[q[k].z * kFxTile]));
        }
        const int r0 = hd.y & 31, r1 = (hd.y >> kPowBits) & 31, r2 = (hd.y >> (2 * kPowBits)) & 31;
        if (r0 != q0 || r1 != q1) {   // uniform
            fold1();
            if (r0 != q0) fold0();
            q0 = r0;
            q1 = r1;
        }
        const Fx zv = z.value<kFxDown>();
        ra.mac(fx_load(t2[r2 * kFxTile]), zv);
        rb.mac(fx_load(d2[r2 * kFxTile]), zv);
    }
    fold1();
    fold0();
    out[0] = S.real(kFxUnit);
    out[1] = g0.real(kFxUnit);
    out[2] = g1.real(kFxUnit);
    out[3] = g2.real(kFxUnit);
}

// 4-body.  With one warp it takes the rows, then the columns; with more, half
// of the warps take the rows and half the columns.
template <int NW>
__global__ void __launch_bounds__(32 * NW) k_forcex4(BatchView B, const int* clusters, const int* perm,
                                                     const long long* perm_n, long long perm_cap, int rs) {
    extern __shared__ __align__(16) unsigned char smem[];
    const FxSmem<4, NW> m(smem, rs);
    FxPair* X = m.rest;
    FxPair* Y = X + rs * rs * rs * kFxTile;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long ntiles = min(*perm_n, perm_cap) / kFxTile;
    EVAcc acc;
    for (;;) {
        const long long tile = fx_claim(&B.queue[1], m.tile);
        if (tile >= ntiles) break;
        const long long base = tile * kFxTile;
        const int c0 = perm[base];
        if (c0 < 0) continue;   // uniform
        int id[4], s, u;
        const DevParamSet* P;
        const TupleRec* R = cluster_tuple<4>(B, clusters, c0, id, s, P, u);
        const bool active = fx_setup<4, NW>(B, clusters, perm[base + lane], *P, *R, rs, m, id, s);
        const int Rp = P->R4;
        const FxPair *T = m.T + lane, *D = m.D + lane;
        // the products X_I, Y_J: the first two pairs' product per (q0, q1), spread over the warps
        for (int k = w; k < 2 * Rp * Rp; k += NW) {
            const int side = k >= Rp * Rp ? 1 : 0, q01 = k - side * Rp * Rp;
            const FxPair* t = T + 3 * side * rs * kFxTile;
            const Fx v = fx_mul(fx_load(t[(q01 / Rp) * kFxTile]), fx_load(t[(rs + q01 % Rp) * kFxTile]));
            FxPair* dst = (side ? Y : X) + q01 * Rp * kFxTile + lane;
            for (int q = 0; q < Rp; q++) dst[q * kFxTile] = fx_store(fx_mul(v, fx_load(t[(2 * rs + q) * kFxTile])));
        }
        __syncthreads();
        const bool ok = ck_bound(B, R->fx_off >= 0 && R->fx_off + (long long)R->fx_split[8] <= P->n_fx4);
        const FxEnt* ent = P->fx4 + R->fx_off;
        double* part = m.part + w * 7 * kFxTile + lane;
        if (NW == 1) {
            double a[4], b[4];
            fx_side(ent, ok ? R->fx_split[0] : 0, ok ? R->fx_split[4] : 0, Y + lane, T, D, rs, a);
            fx_side(ent, ok ? R->fx_split[4] : 0, ok ? R->fx_split[8] : 0, X + lane, T + 3 * rs * kFxTile,
                    D + 3 * rs * kFxTile, rs, b);
            for (int k = 0; k < 4; k++) part[k * kFxTile] = a[k];
            for (int k = 1; k < 4; k++) part[(3 + k) * kFxTile] = b[k];
        } else {
            constexpr int H = NW > 1 ? NW / 2 : 1;   // warps per side
            const int side = w / H, k0 = 4 * side + 4 * (w % H) / H, k1 = 4 * side + 4 * (w % H + 1) / H;
            double a[4];
            fx_side(ent, ok ? R->fx_split[k0] : 0, ok ? R->fx_split[k1] : 0, (side ? X : Y) + lane,
                    T + 3 * side * rs * kFxTile, D + 3 * side * rs * kFxTile, rs, a);
            part[0] = side ? 0.0 : a[0];
            for (int k = 1; k < 4; k++) {
                part[k * kFxTile] = side ? 0.0 : a[k];
                part[(3 + k) * kFxTile] = side ? a[k] : 0.0;
            }
        }
        fx_finish<4, NW>(B, m, *R, active, id, s, acc);
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

template <int RX, int NW>
void launch_x3(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    const int rs = L.rf3;
    const size_t smem = FxSmem<3, NW>::bytes(rs) + sizeof(FxEnt) * (size_t)(L.xs3 + 1);
    auto kern = k_forcex3<RX, NW>;
    const unsigned grid = fx_grid((const void*)kern, 32 * NW, smem, (B.perm3_cap + kFxTile - 1) / kFxTile);
    count_launch(), kern<<<grid, 32 * NW, smem, st>>>(B, B.c3, B.perm3, B.bk_start + B.nbk3, B.perm3_cap, rs);
}

template <int NW>
void launch_x3_nw(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (L.rf3 <= 4) launch_x3<4, NW>(B, L, st);
    else if (L.rf3 <= 8) launch_x3<8, NW>(B, L, st);
    else if (L.rf3 <= 10) launch_x3<10, NW>(B, L, st);
    else launch_x3<12, NW>(B, L, st);
}

template <int NW>
void launch_x4_nw(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    const int rs = L.rf4;
    const size_t smem = FxSmem<4, NW>::bytes(rs) + sizeof(FxPair) * (size_t)2 * rs * rs * rs * kFxTile;
    auto kern = k_forcex4<NW>;
    const unsigned grid = fx_grid((const void*)kern, 32 * NW, smem, (B.perm4_cap + kFxTile - 1) / kFxTile);
    count_launch(), kern<<<grid, 32 * NW, smem, st>>>(B, B.c4, B.perm4, B.bk_start + B.nbk3 + 1 + B.nbk4,
                                                       B.perm4_cap, rs);
}

}  // namespace

void launch_pair_tables_x(const BatchView& B, const int* l2_owner, int nbody, const ForceLaunch& L, cudaStream_t st) {
    if (!(nbody == 3 ? B.use_pc3 : B.use_pc4) || B.n2_cap <= 0) return;
    const long long want = (long long)sm_count() * 8, need = (B.n2_cap + 255) / 256;
    const unsigned grid = (unsigned)(want < need ? want : need);
    if (nbody == 3) count_launch(), k_pair_tables_x<3><<<grid, 256, 0, st>>>(B, l2_owner, L.rf3);
    else count_launch(), k_pair_tables_x<4><<<grid, 256, 0, st>>>(B, l2_owner, L.rf4);
}

void launch_force3x(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm3_cap <= 0 || B.nbk3 <= 0 || L.rf3 <= 0) return;
    switch (L.ftpc3) {
        case 1: launch_x3_nw<1>(B, L, st); break;
        case 2: launch_x3_nw<2>(B, L, st); break;
        case 4: launch_x3_nw<4>(B, L, st); break;
        default: launch_x3_nw<8>(B, L, st); break;
    }
}

void launch_force4x(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm4_cap <= 0 || B.nbk4 <= 0 || L.rf4 <= 0) return;
    switch (L.ftpc4) {
        case 1: launch_x4_nw<1>(B, L, st); break;
        case 2: launch_x4_nw<2>(B, L, st); break;
        case 4: launch_x4_nw<4>(B, L, st); break;
        default: launch_x4_nw<8>(B, L, st); break;
    }
}

}  // namespace ck
