// Cluster fingerprints: the FINGERPRINT build of the reference (records of
// the clusters its LAMMPS pair style evaluates, etc/lmp/src/pair_chimes.cpp:
// 525-536, 620-662, 700-741, 775-810, chimesFF.cpp:1694-1702, 2013-2021,
// 2603-2612) and its cluster-distance histograms
// (chimesFF/src/FP/multi_calc_histogram.cpp).
//
// Records: after a pair-style evaluation, the clusters of one body order that
// pass compute_nB's type and cutoff checks and the recording order rule
// (2-body: i < j, 3-/4-body: strictly increasing tags), as distances and type
// indices, compacted in the pair style's loop order (flag, scan, fill).
//
// Histogram: each record's distances go through the Morse map of its own
// cutoffs (read_flat_clusters) and are sorted; every pair of records (i from
// set 1, j from set 2; j > i when both are the same set) contributes its
// Euclidean distance to a histogram of nbin bins over [0, maxd).  The pair
// loop is O(n1*n2) and runs here as tiles of 256 x 256 records: set-2 tiles
// staged in shared memory (broadcast reads), each thread owning two set-1
// records; counts go to a histogram column per lane in shared memory (bin-major, so a
// warp's 32 columns sit on 32 different banks), by atomics that the block's warps
// share: no load to wait for, and room for more blocks than a column per thread.
// Distances are computed in FP32 with a rigorous bound on the error of the
// distance; a pair whose bin the bound certifies is counted directly, the
// rest (about 1e-4 of them) are recomputed in FP64 with the reference's
// operations, and those that the difference between the device's exponential and the
// host's could move to another bin by the host, so the counts equal the tool's.
//
// Bound: instruction issue.  The two records of a thread go through packed FP32
// instructions together, and the bound is one on the distance in units of bins (a
// constant per record and a relative part) and not on its square against both
// edges: 20 instructions a pair against 45, and a fifth as many pairs to repeat in
// FP64.  Measured, 40001 triplets with themselves, 100 bins: 0.58 ms against 1.86
// (0.63 with the FP64 repeats inlined and counted by the pair loop).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "ck_common.h"
#include "ck_engine.h"
#include "ck_force_common.cuh"
#include "ck_fingerprint.h"
#include "ck_kernels.h"

namespace ck {

namespace {

constexpr int kFpTileJ = 256;   // set-2 records per shared-memory tile
constexpr int kFpRows = 2;      // set-1 records per thread
constexpr int kFpStep = 4;      // set-2 records in flight per thread

// One staged set-2 record, every value twice (packed operands): edges, -margin.
template <int P>
struct __align__(16) FpRec {
    float2 e[P];
    float2 m;
};

// packed FP32 (two values per 64-bit register)
__device__ __forceinline__ unsigned long long fp_pack(float a, float b) {
    return (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a);
}
__device__ __forceinline__ float fp_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float fp_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ unsigned long long fp_add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fp_add2_rm(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fp_mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fp_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float fp_rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP64 bin of one pair, with the tool's operations (dist_struct += pow(a - b, 2) in
// order, sqrt, floor(dist / binw), the dist == maxd rule) on the device's edges; -1 when
// the distance falls past the last bin, kFpTie when eta, the bound on what the
// device's edges differ by from the host's (in units of bins), leaves the bin open.
constexpr int kFpTie = -2;
// What the FP64 bin of a pair needs of the call.
struct FpCall {
    const double *d1, *d2;   // edges of both sets
    double binw, maxd;
    int nbin;
    float inv_w, eta_q;
    int* flags;
};
// The FP32 distance and its error, u = 2^-24, N = |a| + |b| (norms of the
// records): with a, b and each difference rounded,
//   |s32 - s| <= 2 u N sqrt(s) + (2 + P) u s (+ second order),
// so |sqrt(s32) - sqrt(s)| <= 2 u N + (2 + P) u sqrt(s) -- the second-order part
// included once sqrt(s) >= 4 u N, which the test below implies -- and
// t = (s32 / w) rsqrt(s32) adds 2^-21.9 t at most.  In units of bins:
//   |t - dist / w| <= 4 u N / w + 2^-20 t
// A pair is counted in floor(t) when t's fraction is farther than that from 0
// and 1 (the floor by a round-down add at 1.5 * 2^23: no conversion
// instructions); otherwise, and for s = 0, in its exact FP64 bin.
constexpr float kFpMargin = 4.0f * 5.9604645e-8f * 1.001f;   // per unit of norm and bin width
constexpr float kFpRel = 9.5367432e-7f;                      // 2^-20
constexpr float kFpMagic = 12582912.0f;                      // 1.5 * 2^23: adding it rounds to an integer
constexpr int kFpMagicBits = 0x4B400000;

// The tool's edges come from the host's exp, the device's from its own: each within
// one unit in the last place of exp(-d / lambda), so that an edge x = (exp - avg) /
// diff differs by at most 2^-50 (|x| + |avg / diff|), a distance by the norms of
// both records' differences.  In units of bins, with records' margins m and
// q = 2^-50 * 2 sqrt(P) max |avg / diff| / w (0: the edges are the host's):
//   eta = 2^-50 (m_a + m_b) / kFpMargin + q
// A pair whose bin that leaves open -- an edge is nearer than some 1e-14 of a bin --
// is listed, and the host bins it.
constexpr float kFpEtaMargin = 0x1.03p-50f / (4.0f * 5.9604645e-8f);   // (rounded up)
struct FpPair {
    long long i, j;
};
constexpr int kFpTies = 1 << 16;   // pairs listed (more: the host makes all edges)
constexpr int kFpFlags = 4;        // words before them: a distance past the last bin; pairs to list
// Tiles a block takes in one launch: each adds at most kFpTileJ per record of four
// warps' threads to one of the block's 32-bit counts.
constexpr int kFpBlockTiles = 1 << 20;
static_assert((long long)kFpBlockTiles * kFpTileJ * kFpRows * 4 < 1LL << 32, "counts of a lane's column");

// Counts records i and j in FP64, where the FP32 candidate is not certified (margins:
// the sum of theirs; hist: the lane's column).  Called and not inlined: its registers
// would cost the pair loop a block per SM.
template <int P>
__device__ __noinline__ void fp_exact(const FpCall& C, long long i, long long j, float margins, unsigned int* hist) {
    double ds = 0.0;
    for (int p = 0; p < P; p++) {
        const double d = __dsub_rn(C.d1[i * P + p], C.d2[j * P + p]);
        ds = __dadd_rn(ds, __dmul_rn(d, d));
    }
    const float eta = C.eta_q > 0.0f ? kFpEtaMargin * margins + C.eta_q : 0.0f;
    // a candidate, confirmed in FP64 when ds lies inside its squared edges by far
    // more than the roundings of sqrt and the division, and more than eta, twice (an
    // edge above zero is one bin or more)
    int bin = (int)(sqrtf((float)ds) * C.inv_w);
    const double lo = bin * C.binw, hi = lo + C.binw;
    if (!(bin >= 0 && bin < C.nbin && eta < 3e-10f && ds >= lo * lo * (1.0 + 1e-9) && ds <= hi * hi * (1.0 - 1e-9))) {
        // the tool's operations
        const double dist = __dadd_rn(__dsqrt_rn(ds), 0.0);
        const double t = __ddiv_rn(dist, C.binw), k = rint(t);
        if (eta > 0.0f && k >= 1.0 && !(fabs(t - k) > (double)eta + 0x1p-50 * t)) {
            const int n = atomicAdd(&C.flags[1], 1);
            if (n < kFpTies) reinterpret_cast<FpPair*>(C.flags + kFpFlags)[n] = FpPair{i, j};
            return;
        }
        bin = (int)floor(t);
        if (dist == C.maxd) bin = bin - 1;
        if (bin < 0 || bin >= C.nbin) {
            atomicOr(&C.flags[0], 1);   // (the call fails)
            return;
        }
    }
    atomicAdd(&hist[bin * 32], 1u);
}

// e, m: records' edges and margins (kFpMargin norm / w, rounded up).
template <int P>
__global__ void __launch_bounds__(128, P == 1 ? 7 : P == 3 ? 6 : 5)
    k_fp_hist(const float* __restrict__ e1, const float* __restrict__ m1, long long n1, const float* __restrict__ e2,
              const float* __restrict__ m2, long long n2, int same, long long t_begin, long long t_end,
              long long n_jtile, unsigned long long* counts, const __grid_constant__ FpCall C) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int T = blockDim.x;
    const int tid = threadIdx.x, lane = tid & 31, nbin = C.nbin;
    FpRec<P>* tile = reinterpret_cast<FpRec<P>*>(smem);
    unsigned int* hist = reinterpret_cast<unsigned int*>(tile + kFpTileJ);       // [nbin + 1][32]
    for (int b = tid; b < nbin * 32; b += T) hist[b] = 0u;
    const float inv_wf = C.inv_w;
    const int rows = T * kFpRows;
    const unsigned long long inv2 = fp_pack(inv_wf, inv_wf), magic2 = fp_pack(kFpMagic, kFpMagic),
                             unmagic2 = fp_pack(-kFpMagic, -kFpMagic), half2 = fp_pack(-0.5f, -0.5f),
                             rel2 = fp_pack(-kFpRel, -kFpRel), neg2 = fp_pack(-1.0f, -1.0f);
    for (long long t = t_begin + blockIdx.x; t < t_end; t += gridDim.x) {
        const long long it = t / n_jtile, jt = t % n_jtile;
        const long long i0 = it * rows, j0 = jt * kFpTileJ;
        // a tile whose every j is <= every i holds no pair j > i
        if (same && j0 + kFpTileJ - 1 <= i0) continue;
        const int jn = (int)min((long long)kFpTileJ, n2 - j0);
        __syncthreads();
        for (int k = tid; k < jn; k += T) {
            FpRec<P> r;
            for (int p = 0; p < P; p++) {
                const float v = -e2[(j0 + k) * P + p];
                r.e[p] = make_float2(v, v);
            }
            const float v = -m2[j0 + k];
            r.m = make_float2(v, v);
            tile[k] = r;
        }
        __syncthreads();
        const long long ia = i0 + tid, ib = ia + T;
        if (ia >= n1) continue;
        const bool two = ib < n1;   // (else the second row repeats the first and counts nothing)
        unsigned long long a[P];
        for (int p = 0; p < P; p++) a[p] = fp_pack(e1[ia * P + p], e1[(two ? ib : ia) * P + p]);
        const unsigned long long lim2 = fp_pack(0.5f - m1[ia], 0.5f - m1[two ? ib : ia]);
        // from k on both rows take every record; before it, where both records are of
        // the same set, only the first row does
        const int ka = same ? (int)max(0LL, min((long long)jn, ia + 1 - j0)) : 0;
        const int kb = !two ? jn : same ? (int)max(0LL, min((long long)jn, ib + 1 - j0)) : 0;
        // record k against both rows: candidate bins, and whether the bound certifies them
        auto candidates = [&](int k, int& ba, int& bb, bool& oka, bool& okb) {
            const FpRec<P>& r = tile[k];
            unsigned long long s = 0ull;
#pragma unroll
            for (int p = 0; p < P; p++) {
                const unsigned long long d = fp_add2(a[p], reinterpret_cast<const unsigned long long*>(r.e)[p]);
                s = p == 0 ? fp_mul2(d, d) : fp_fma2(d, d, s);
            }
            const unsigned long long q = fp_mul2(fp_mul2(s, inv2), fp_pack(fp_rsqrt_approx(fp_lo(s)), fp_rsqrt_approx(fp_hi(s))));
            const unsigned long long mag = fp_add2_rm(q, magic2);           // magic + floor(dist / w)
            const unsigned long long kf = fp_add2(mag, unmagic2);
            const unsigned long long h = fp_add2(fp_fma2(kf, neg2, q), half2);   // fraction - 1/2
            const unsigned long long lim = fp_fma2(q, rel2, fp_add2(lim2, *reinterpret_cast<const unsigned long long*>(&r.m)));
            ba = (int)(unsigned)mag - kFpMagicBits;
            bb = (int)(unsigned)(mag >> 32) - kFpMagicBits;
            oka = fabsf(fp_lo(h)) < fp_lo(lim) && (unsigned)ba < (unsigned)nbin;
            okb = fabsf(fp_hi(h)) < fp_hi(lim) && (unsigned)bb < (unsigned)nbin;
        };
        // bit u of `open`: the first row with record k + u, bit kFpStep + u: the second
        auto exact = [&](int k, unsigned open) {
            while (open) {
                const int q = __ffs(open) - 1, u = q % kFpStep;
                open &= open - 1;
                const long long i = q < kFpStep ? ia : ib;
                fp_exact<P>(C, i, j0 + k + u, m1[i] - tile[k + u].m.x, hist + lane);
            }
        };
        for (int k = ka; k < kb; k++) {
            int ba, bb;
            bool oka, okb;
            candidates(k, ba, bb, oka, okb);
            if (oka) atomicAdd(&hist[ba * 32 + lane], 1u);
            else exact(k, 1u);
        }
        int k = kb;
        for (; k + kFpStep <= jn; k += kFpStep) {   // a few records' chains together
            int ba[kFpStep], bb[kFpStep];
            bool oka[kFpStep], okb[kFpStep];
            unsigned open = 0;
#pragma unroll
            for (int u = 0; u < kFpStep; u++) {
                candidates(k + u, ba[u], bb[u], oka[u], okb[u]);
                open |= (oka[u] ? 0u : 1u << u) | (okb[u] ? 0u : 1u << (kFpStep + u));
                ba[u] = oka[u] ? ba[u] : nbin;   // (a column past the bins: an atomic without a branch)
                bb[u] = okb[u] ? bb[u] : nbin;
            }
#pragma unroll
            for (int u = 0; u < kFpStep; u++) {
                atomicAdd(&hist[ba[u] * 32 + lane], 1u);
                atomicAdd(&hist[bb[u] * 32 + lane], 1u);
            }
            if (open) exact(k, open);
        }
        for (; k < jn; k++) {
            int ba, bb;
            bool oka, okb;
            candidates(k, ba, bb, oka, okb);
            if (oka) atomicAdd(&hist[ba * 32 + lane], 1u);
            if (okb) atomicAdd(&hist[bb * 32 + lane], 1u);
            if (!oka || !okb) exact(k, (oka ? 0u : 1u) | (okb ? 0u : 1u << kFpStep));
        }
    }
    __syncthreads();
    for (int b = tid; b < nbin; b += T) {
        unsigned long long sum = 0;
        for (int t2 = 0; t2 < 32; t2++) sum += hist[b * 32 + t2];
        if (sum) atomicAdd(&counts[b], sum);
    }
}

// Edges of a record: the transform of read_flat_clusters (multi_calc_histogram.cpp:
// 26-123) with the cluster's own cutoffs, sorted, in FP64 and FP32, and its margin.
// (Host code before: 2.0 ms of exponentials and sorting for 40001 triplets.)
template <int P>
__global__ void k_fp_edges(const DevParamSet* Pp, long long n, const double* d, const int* t, double inv_w,
                           double* e, float* ef, float* m) {
    constexpr int NB = P == 1 ? 2 : P == 3 ? 3 : 4;
    const DevParamSet& D = *Pp;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += stride) {
        int u = 0;
        for (int k = 0; k < NB; k++) u = u * D.ntypes + t[c * NB + k];
        double x[P], s = 0.0;
#pragma unroll
        for (int p = 0; p < P; p++) {
            double lam, avg, diff;
            if constexpr (P == 1) {
                const PairRec& R = D.pairs[D.pair_map[u]];
                lam = R.lam; avg = R.xavg; diff = R.xdiff;
            } else {
                const TupleRec& R = (NB == 3 ? D.t3 : D.t4)[u];
                lam = R.lam[p]; avg = R.xavg[p]; diff = R.xdiff[p];
            }
            x[p] = (exp(-d[c * P + p] / lam) - avg) / diff;
            s += x[p] * x[p];
        }
#pragma unroll
        for (int q = 1; q < P; q++)
#pragma unroll
            for (int p = P - 1; p >= q; p--) {
                const double lo = x[p] < x[p - 1] ? x[p] : x[p - 1], hi = x[p] < x[p - 1] ? x[p - 1] : x[p];
                x[p - 1] = lo;
                x[p] = hi;
            }
        for (int p = 0; p < P; p++) {
            e[c * P + p] = x[p];
            ef[c * P + p] = (float)x[p];
        }
        m[c] = (float)(sqrt(s) * inv_w * (1.0 + 1e-6)) * kFpMargin;
    }
}

// ---- fingerprint records of the pair-style path ---------------------------
__device__ __forceinline__ double fp_dist(const double* x, int i, int j) {
    const double d0 = __dsub_rn(x[3 * (long long)j + 0], x[3 * (long long)i + 0]);
    const double d1 = __dsub_rn(x[3 * (long long)j + 1], x[3 * (long long)i + 1]);
    const double d2 = __dsub_rn(x[3 * (long long)j + 2], x[3 * (long long)i + 2]);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
}

// 2-body: list entries (i, j) with tag[j] > tag[i] (the pair loop), i < j
// (valid_order) and r below the pair type's outer cutoff (compute_2B).
template <bool FILL>
__global__ void k_nl_fp2(BatchView B, NeighView N, int* flag, const long long* off, double* d, int* t) {
    const DevParamSet& P = B.psets[B.sys[0].pset];
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < N.nent; e += stride) {
        const int i = N.ilist[N.owner[e]];
        const int j = N.neigh[e];
        bool ok = N.tag[j] > N.tag[i] && i < j;
        double r = 0.0;
        if (ok) {
            r = fp_dist(B.ghost_fs, i, j);
            ok = r < P.pairs[P.pair_map[B.atom_type[i] * P.ntypes + B.atom_type[j]]].rout;
        }
        if (!FILL) {
            flag[e] = ok ? 1 : 0;
        } else if (ok) {
            const long long o = off[e];
            d[o] = r;
            t[2 * o] = B.atom_type[i];
            t[2 * o + 1] = B.atom_type[j];
        }
    }
}

// 3-/4-body: listed clusters with strictly increasing tags (valid_order),
// a type that is not excluded and every pair below its outer cutoff.
template <int NB, bool FILL>
__global__ void k_nl_fpn(BatchView B, NeighView N, long long n, int* flag, const long long* off, double* d, int* t) {
    constexpr int NP = NB * (NB - 1) / 2;
    const DevParamSet& P = B.psets[B.sys[0].pset];
    const int* cl = NB == 3 ? B.c3 : B.c4;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += stride) {
        int id[NB];
        for (int k = 0; k < NB; k++) id[k] = cl[(long long)NB * q + k];
        bool ok = true;
        if (NB == 3) ok = N.tag[id[0]] < N.tag[id[1]] && N.tag[id[0]] < N.tag[id[2]] && N.tag[id[1]] < N.tag[id[2]];
        else ok = N.tag[id[0]] < N.tag[id[1]] && N.tag[id[1]] < N.tag[id[2]] && N.tag[id[2]] < N.tag[id[3]];
        double r[NP];
        int u = 0;
        for (int k = 0; k < NB; k++) u = u * P.ntypes + B.atom_type[id[k]];
        const TupleRec& R = (NB == 3 ? P.t3 : P.t4)[u];
        if (ok) ok = R.type_id >= 0;
        if (ok)
            for (int p = 0; p < NP; p++) {
                r[p] = fp_dist(B.ghost_fs, id[Topo<NB>::a(p)], id[Topo<NB>::b(p)]);
                if (r[p] >= R.rout[p]) ok = false;
            }
        if (!FILL) {
            flag[q] = ok ? 1 : 0;
        } else if (ok) {
            const long long o = off[q];
            for (int p = 0; p < NP; p++) d[o * NP + p] = r[p];
            for (int k = 0; k < NB; k++) t[o * NB + k] = B.atom_type[id[k]];
        }
    }
}

unsigned fp_grid(long long n) {
    long long g = (n + 255) / 256;
    if (g < 1) g = 1;
    const long long cap = (long long)sm_count() * 8;
    return (unsigned)(g < cap ? g : cap);
}

}  // namespace

void launch_nl_fp(const BatchView& B, const NeighView& N, int nbody, long long n, bool fill, int* flag,
                  const long long* off, double* d, int* t, cudaStream_t st) {
    if (n <= 0) return;
    const unsigned g = fp_grid(n);
    if (nbody == 2) {
        if (fill) count_launch(), k_nl_fp2<true><<<g, 256, 0, st>>>(B, N, flag, off, d, t);
        else count_launch(), k_nl_fp2<false><<<g, 256, 0, st>>>(B, N, flag, off, d, t);
    } else if (nbody == 3) {
        if (fill) count_launch(), k_nl_fpn<3, true><<<g, 256, 0, st>>>(B, N, n, flag, off, d, t);
        else count_launch(), k_nl_fpn<3, false><<<g, 256, 0, st>>>(B, N, n, flag, off, d, t);
    } else {
        if (fill) count_launch(), k_nl_fpn<4, true><<<g, 256, 0, st>>>(B, N, n, flag, off, d, t);
        else count_launch(), k_nl_fpn<4, false><<<g, 256, 0, st>>>(B, N, n, flag, off, d, t);
    }
}

// ---------------------------------------------------------------------------
// Histogram driver
// ---------------------------------------------------------------------------
namespace {

// transform of read_flat_clusters (multi_calc_histogram.cpp:112-123), host FP64
double fp_transform(double rcin, double rcout, double lambda, double rij) {
    double x_min = std::exp(-1 * rcin / lambda);
    double x_max = std::exp(-1 * rcout / lambda);
    double x_avg = 0.5 * (x_max + x_min);
    double x_diff = 0.5 * (x_max - x_min);
    x_diff *= -1.0;
    return (std::exp(-1 * rij / lambda) - x_avg) / x_diff;
}

// Sorted transformed edges of record c (the cluster's own cutoffs, pair lambdas by
// the atoms' pair type), read_flat_clusters (:26-107).
void fp_host_edges(const Engine& eng, int slot, int nbody, long long c, const double* d, const int* t, double* e) {
    const HostParams& P = eng.params(slot);
    const int nt = P.ntypes, np = nbody * (nbody - 1) / 2;
    const int* ty = t + c * nbody;
    if (nbody == 2) {
        const int p = P.pair_map[ty[0] * nt + ty[1]];
        e[0] = fp_transform(P.rin[p], P.rout[p], P.lam[p], d[c]);
        return;
    }
    int u = 0;
    for (int k = 0; k < nbody; k++) u = u * nt + ty[k];
    const TupleRec& R = eng.tuples(slot, nbody)[u];
    for (int p = 0; p < np; p++) e[p] = fp_transform(R.rin[p], R.rout[p], R.lam[p], d[c * np + p]);
    std::sort(e, e + np);
}

// The bin of two records' edges as the tool computes it (dist_struct, floor(dist /
// binw), the dist == maxd rule); -1 past the last one.
int fp_host_bin(const double* a, const double* b, int np, double binw, double maxd, int nbin) {
    double ds = 0.0;
    for (int p = 0; p < np; p++) ds += (a[p] - b[p]) * (a[p] - b[p]);
    const double dist = std::sqrt(ds);
    int bin = (int)std::floor(dist / binw);
    if (dist == maxd) bin = bin - 1;
    return bin < 0 || bin >= nbin ? -1 : bin;
}

// max |avg / diff| of a set's maps (see kFpEtaMargin)
double fp_shift(const Engine& eng, int slot, int nbody) {
    const HostParams& P = eng.params(slot);
    double q = 0.0;
    auto take = [&](double rin, double rout, double lam) {
        const double lo = std::exp(-1 * rin / lam), hi = std::exp(-1 * rout / lam);
        const double v = std::fabs((hi + lo) / (hi - lo));
        q = v > q || v != v ? v : q;
    };
    if (nbody == 2)
        for (int p = 0; p < P.npairs; p++) take(P.rin[p], P.rout[p], P.lam[p]);
    else
        for (const TupleRec& R : eng.tuples(slot, nbody))
            for (int p = 0; R.type_id >= 0 && p < nbody * (nbody - 1) / 2; p++) take(R.rin[p], R.rout[p], R.lam[p]);
    return q;
}

// Every record has known types and a cluster type that is not excluded.
Status fp_check(const Engine& eng, int slot, int nbody, long long n, const int* t, std::string& err) {
    const int nt = eng.params(slot).ntypes;
    for (long long c = 0; c < n; c++) {
        int u = 0;
        for (int k = 0; k < nbody; k++) {
            const int ty = t[c * nbody + k];
            if (ty < 0 || ty >= nt) {
                err = "fingerprint record " + std::to_string(c) + ": type index out of range";
                return kErrInput;
            }
            u = u * nt + ty;
        }
        if (nbody > 2 && eng.tuples(slot, nbody)[u].type_id < 0) {
            err = "fingerprint record " + std::to_string(c) + ": excluded cluster type";
            return kErrInput;
        }
    }
    return kOk;
}

}  // namespace

Status fp_histogram(Engine& eng, int slot, int nbody, long long n1, const double* d1, const int* t1, long long n2,
                    const double* d2, const int* t2, bool same, int nbin, long long* counts, long long* nsamples,
                    std::string& err) {
    Status st = eng.init_device(err);
    if (st != kOk) return st;
    if (slot < 0 || slot >= eng.n_param_sets()) {
        err = "parameter set not loaded";
        return kErrState;
    }
    if (nbody < 2 || nbody > 4 || nbin < 1 || n1 < 0 || n2 < 0) {
        err = "fingerprint histogram: nbody 2..4, nbin >= 1, non-negative record counts";
        return kErrInput;
    }
    const HostParams& P = eng.params(slot);
    if ((nbody == 3 && P.o3 <= 0) || (nbody == 4 && P.o4 <= 0)) {
        err = "the parameter set has no " + std::to_string(nbody) + "-body terms";
        return kErrInput;
    }
    for (int b = 0; b < nbin; b++) counts[b] = 0;
    *nsamples = 0;
    const int np = nbody * (nbody - 1) / 2;
    if ((st = fp_check(eng, slot, nbody, n1, t1, err)) != kOk) return st;
    if (same) n2 = n1;
    else if ((st = fp_check(eng, slot, nbody, n2, t2, err)) != kOk) return st;
    // one process of gen_flat_hists: nothing is counted unless the first set
    // has at least two records (its task range must have end > start)
    if (n1 <= 1 || n2 <= 0) return kOk;
    const double maxd = nbody == 2 ? 3.0 : (nbody == 3 ? std::sqrt(12.0) + 1.0 : std::sqrt(24.0) + 1.0);
    const double binw = maxd / nbin;
    constexpr int T = 128;
    const size_t rec = nbody == 2 ? sizeof(FpRec<1>) : nbody == 3 ? sizeof(FpRec<3>) : sizeof(FpRec<6>);
    const size_t smem = (size_t)(nbin + 1) * 32 * 4 + rec * kFpTileJ;
    // (a limit above the one it names, as it always was)
    if ((size_t)nbin * 32 * 4 + (nbody == 2 ? 8 : nbody == 3 ? 16 : 32) * (size_t)kFpTileJ > 200 * 1024) {
        err = "fingerprint histogram: nbin too large for the shared-memory histogram (at most 1280 bins)";
        return kErrInput;
    }
    const cudaStream_t s = eng.stream();
#define FP_TRY(call)                                                                   \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            err = std::string("CUDA error: ") + cudaGetErrorString(e_) + " at " #call; \
            return kErrCuda;                                                           \
        }                                                                              \
    } while (0)
    // the engine's workspace: per set the distances (then the edges), types, FP32
    // edges and margins; the counts and the flag
    auto up16 = [](size_t b) { return (b + 15) / 16 * 16; };
    auto set_bytes = [&](long long n) {
        return up16(sizeof(double) * n * np) * 2 + up16(sizeof(int) * n * nbody) + up16(sizeof(float) * n * np) +
               up16(sizeof(float) * n);
    };
    const size_t b1 = set_bytes(n1), b2 = same ? 0 : set_bytes(n2), bc = up16(sizeof(unsigned long long) * nbin);
    unsigned char* ws = nullptr;
    FP_TRY(eng.workspace(b1 + b2 + bc + sizeof(int) * kFpFlags + sizeof(FpPair) * kFpTies, ws));
    struct Set {
        double* d;
        float *e, *m;
    };
    const int Pn = np;
    auto edges = [&](unsigned char* p, long long n, const double* d, const int* ty, Set& out) -> cudaError_t {
        double* raw = reinterpret_cast<double*>(p);
        out.d = reinterpret_cast<double*>(p + up16(sizeof(double) * n * np));
        int* dt = reinterpret_cast<int*>(p + 2 * up16(sizeof(double) * n * np));
        out.e = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(dt) + up16(sizeof(int) * n * nbody));
        out.m = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(out.e) + up16(sizeof(float) * n * np));
        cudaError_t e = cudaMemcpyAsync(raw, d, sizeof(double) * n * np, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dt, ty, sizeof(int) * n * nbody, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        const unsigned g = (unsigned)std::min<long long>((n + 127) / 128, 8LL * sm_count());
        const DevParamSet* D = eng.device_params() + slot;
        if (Pn == 1) count_launch(), k_fp_edges<1><<<g, 128, 0, s>>>(D, n, raw, dt, 1.0 / binw, out.d, out.e, out.m);
        else if (Pn == 3) count_launch(), k_fp_edges<3><<<g, 128, 0, s>>>(D, n, raw, dt, 1.0 / binw, out.d, out.e, out.m);
        else count_launch(), k_fp_edges<6><<<g, 128, 0, s>>>(D, n, raw, dt, 1.0 / binw, out.d, out.e, out.m);
        return cudaGetLastError();
    };
    Set s1, s2;
    FP_TRY(edges(ws, n1, d1, t1, s1));
    s2 = s1;
    if (!same) FP_TRY(edges(ws + b1, n2, d2, t2, s2));
    unsigned long long* dcounts = reinterpret_cast<unsigned long long*>(ws + b1 + b2);
    int* dflags = reinterpret_cast<int*>(ws + b1 + b2 + bc);
    const long long n_it = (n1 + (long long)T * kFpRows - 1) / ((long long)T * kFpRows),
                    n_jt = (n2 + kFpTileJ - 1) / kFpTileJ;
    const void* kern = nbody == 2 ? (const void*)k_fp_hist<1> : nbody == 3 ? (const void*)k_fp_hist<3>
                                                                           : (const void*)k_fp_hist<6>;
    if (smem > 48 * 1024) allow_max_smem(kern);
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, T, smem);
    long long grid = (long long)sm_count() * (occ > 0 ? occ : 1);
    if (grid > n_it * n_jt) grid = n_it * n_jt;
    const int sm = same ? 1 : 0;
    std::vector<unsigned long long> hc(nbin);
    int hflag[2] = {0, 0};   // a distance past the last bin; pairs to list
    // q: kFpEtaMargin's, 0 with the host's edges
    auto histogram = [&](float q) -> cudaError_t {
        cudaError_t e = cudaMemsetAsync(dcounts, 0, bc + sizeof(int) * kFpFlags, s);
        if (e != cudaSuccess) return e;
        const long long ntiles = n_it * n_jt, step = grid * kFpBlockTiles;
        const FpCall C{s1.d, s2.d, binw, maxd, nbin, (float)(1.0 / binw), q, dflags};
        for (long long t0 = 0; t0 < ntiles; t0 += step) {
            const long long t1 = std::min(ntiles, t0 + step);
            count_launch();
            if (nbody == 2)
                k_fp_hist<1><<<(unsigned)grid, T, smem, s>>>(s1.e, s1.m, n1, s2.e, s2.m, n2, sm, t0, t1, n_jt, dcounts, C);
            else if (nbody == 3)
                k_fp_hist<3><<<(unsigned)grid, T, smem, s>>>(s1.e, s1.m, n1, s2.e, s2.m, n2, sm, t0, t1, n_jt, dcounts, C);
            else
                k_fp_hist<6><<<(unsigned)grid, T, smem, s>>>(s1.e, s1.m, n1, s2.e, s2.m, n2, sm, t0, t1, n_jt, dcounts, C);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        e = cudaMemcpyAsync(hc.data(), dcounts, sizeof(unsigned long long) * nbin, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(hflag, dflags, sizeof(hflag), cudaMemcpyDeviceToHost, s);
        return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    };
    const float shift = 0x1.03p-50f * 2.0f * (float)(std::sqrt((double)np) * fp_shift(eng, slot, nbody) / binw);
    if (std::isfinite(shift)) FP_TRY(histogram(shift));
    if (!std::isfinite(shift) || hflag[1] > kFpTies) {
        auto host_edges = [&](long long n, const double* d, const int* t, const Set& out) -> cudaError_t {
            std::vector<double> e((size_t)n * np);
            for (long long c = 0; c < n; c++) fp_host_edges(eng, slot, nbody, c, d, t, &e[(size_t)c * np]);
            return cudaMemcpy(out.d, e.data(), sizeof(double) * e.size(), cudaMemcpyHostToDevice);
        };
        FP_TRY(cudaStreamSynchronize(s));
        FP_TRY(host_edges(n1, d1, t1, s1));
        if (!same) FP_TRY(host_edges(n2, d2, t2, s2));
        FP_TRY(histogram(0.0f));
    } else if (hflag[1] > 0) {
        std::vector<FpPair> tie(hflag[1]);
        FP_TRY(cudaMemcpy(tie.data(), dflags + kFpFlags, sizeof(FpPair) * tie.size(), cudaMemcpyDeviceToHost));
        for (const FpPair& q : tie) {
            double a[6], b[6];
            fp_host_edges(eng, slot, nbody, q.i, d1, t1, a);
            fp_host_edges(eng, slot, nbody, q.j, same ? d1 : d2, same ? t1 : t2, b);
            const int bin = fp_host_bin(a, b, np, binw, maxd, nbin);
            if (bin < 0) hflag[0] = 1;
            else hc[bin]++;
        }
    }
#undef FP_TRY
    if (hflag[0]) {
        err = "ERROR: computed bin larger than nbins (a cluster distance lies past the histogram range)";
        return kErrInput;
    }
    long long tot = 0;
    for (int b = 0; b < nbin; b++) {
        counts[b] = (long long)hc[b];
        tot += counts[b];
    }
    *nsamples = tot;
    return kOk;
}

}  // namespace ck
