// Tensor-core 3-body contraction (mixed form) on the fifth-generation tensor
// cores: tcgen05.mma with TF32 operands in shared memory and FP32
// accumulators in tensor memory (TMEM).
//
// For the clusters of one ordered type tuple, with R powers per pair and the
// tuple's coefficients as a dense matrix A[q_ij][J], J = q_ik * R + q_jk
// (the factored form's row and column indices, ck_common.h FactRow):
//   W  = X  . A,   X[c][q]  = T_ij(c)[q]        (energy and column gradients)
//   W' = dX . A,   dX[c][q] = dT_ij/dr(c)[q]    (row gradient)
// one MMA chain each per 128 clusters (M = 128, K = R padded to 8 or 16, N =
// R^2 padded to 16).  Each cluster's thread then reduces its TMEM row:
//   V[b] = sum_c W[b,c] T_jk[c],  V2[b] = sum_c W[b,c] dT_jk[c],
//   V'[b] = sum_c W'[b,c] T_jk[c]
//   S = sum_b V[b] T_ik[b],   G_ij = sum_b V'[b] T_ik[b],
//   G_ik = sum_b V[b] dT_ik[b],   G_jk = sum_b V2[b] T_ik[b]
// which are the sums of compute_3B (chimesFF/src/chimesFF.cpp:2068-2169) in
// another association order.
//
// Precision: TF32 keeps 10 mantissa bits, so both operands are split into
// three TF32 parts (high h, middle m, low l: each the TF32 rounding of what
// the previous ones leave) and W = Xh.Ah + Xh.Am + Xm.Ah + Xh.Al + Xl.Ah +
// Xm.Am (six MMAs per product; the dropped terms are ~2^-33 relative), with
// FP32 accumulation: the FP32 contraction's accuracy.  (With two parts and
// three MMAs the error is ~2^-21 per product, 3e-6 of the stress of the
// reference's HN3 force field.)  Distances (minimum image) and the Morse
// exponential stay in FP64; the Chebyshev recursion, cutoff and the
// cluster's force scalars, forces and virial are FP32 (they derive from the
// FP32 sums); the per-atom force, energy and virial accumulation is FP64.
// GB300 issues one FP64 warp instruction per 16 cycles per SM: with the
// pair-table cache (k_pairs_x) the geometry, exponential and tables of the
// pairs ij and ik -- list entries of the cluster's first atom -- are read
// instead of recomputed per cluster.
//
// Work: persistent CTAs of 128 threads (one cluster per thread) take
// 128-cluster tiles from an atomic queue over the clusters bucketed by
// (parameter set, tuple) and padded to 128 slots, so a tile has one tuple.
// Per tile: the tuple's coefficient image (B operand) is copied to shared
// memory when the bucket changes; each thread writes its T_ij row (K-major,
// no-swizzle core-matrix layout), one thread issues the MMAs and commits them
// to an mbarrier, and while they run the threads set up pair jk; every thread
// waits with a bounded poll and reduces its row of W in 16-column chunks.  The
// dT_ij/dr row then goes through the same operand buffer and TMEM columns for W',
// while the ik tables are read and the sums with W formed.
//
// Bound: latency of the gathers and of the chains through the MMAs, with the FP64
// pipe (pair jk, virial sums) at 39%.  So four CTAs per SM (16 warps): one
// operand buffer and 128 TMEM columns each, 128 registers a thread, tables read
// when they are needed rather than held.  Measured: 1.47 M triplets of 32768
// atoms 556 -> 338 us, 9.15 M of 2000 configurations 3.30 -> 1.95 ms (320 us and
// 1.82 ms with conversions and comparisons off the FP64 pipe), against two CTAs
// that hold both rows, both accumulators and all tables at once.
// A wait that runs out sets flags[7] and the CTA stops after freeing its TMEM.
#include <cuda_runtime.h>

#include <cstdint>

#include "ck_common.h"
#include "ck_force_common.cuh"
#include "ck_kernels.h"
#include "ck_math.cuh"

namespace ck {

namespace {

constexpr int kTcTile = 128;              // clusters per tile (MMA M)
constexpr uint32_t kTcCols = 128;         // TMEM columns per CTA: W, then W'
constexpr int kTc3Ctas = 4;               // 3-body CTAs per SM (registers, shared memory, 4 x 128 of 512 columns)
constexpr int kTcSpin = 1 << 22;          // bounded mbarrier wait: polls (~0.15 s with the back-off)
constexpr size_t kTcMinSmem = 46 * 1024;  // keeps four CTAs per SM (TMEM)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of tcgen05.mma: start address, leading
// byte offset (between core matrices adjacent in K), stride byte offset
// (between core matrices adjacent in M/N), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

__device__ __forceinline__ float tf32_hi(float x) {
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, int accumulate) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = __uint_as_float(r[q]);
}

// Chebyshev tables T[0..R), dT/dr[0..R) and cutoff of one pair, in registers
// (the arithmetic of pair_setup / cheby_fill_strided, ck_factored.cu and
// ck_math.cuh, unrolled for a compile-time R).
template <int R>
__device__ __forceinline__ void pair_regs(const DevParamSet& P, const TupleRec& Q, int p, double r, float (&T)[R],
                                          float (&D)[R], float& fc, float& fcd, int* flags) {
    const double rin = Q.rin[p];
    const bool oor = less_pos(r, rin);
    const double rr = oor ? rin : r;
    const double e = exp_neg(rr * Q.inv_lam[p]);
    const double xd = (e - Q.xavg[p]) * Q.inv_xdiff[p];
    const double dxdr = -e * Q.inv_lam[p] * Q.inv_xdiff[p];
    const float x = narrow(xd), tx = 2.0f * x, g = narrow(dxdr);
    float k = 0.0f, dm = 1.0f;
    if (oor) {
        if (flags) atomicAdd(&flags[4], 1);
        const double damp = exp((r - rin) / P.inner_smooth);
        k = float(P.inner_smooth * (damp - 1.0));
        dm = float(damp);
    }
    T[0] = 1.0f;
    D[0] = 0.0f;
    float t0 = 1.0f, t1 = x, u0 = 1.0f, u1 = tx;
    if (R > 1) {
        const float d1 = g * u0;
        T[1] = oor ? t1 + k * d1 : t1;
        D[1] = oor ? d1 * dm : d1;
    }
#pragma unroll
    for (int n = 2; n < R; n++) {
        const float t2 = tx * t1 - t0;
        const float u2 = tx * u1 - u0;
        const float dn = float(n) * g * u1;
        T[n] = oor ? t2 + k * dn : t2;
        D[n] = oor ? dn * dm : dn;
        t0 = t1; t1 = t2; u0 = u1; u1 = u2;
    }
    const double finv = Q.fc_inv[p];
    if (!P.tersoff) {
        const float f0 = 1.0f - narrow(r) * narrow(finv);
        fc = f0 * f0 * f0;
        fcd = f0 * f0 * (-3.0f * narrow(finv));
    } else {
        const double th = Q.fc_th[p];
        if (less_pos(r, th)) { fc = 1.0f; fcd = 0.0f; }
        else if (!less_pos(r, Q.rout[p]) && r > Q.rout[p]) { fc = 0.0f; fcd = 0.0f; }
        else {
            const float f0 = narrow(r - th) * narrow(finv) * float(kPi) + float(kPi / 2.0);
            float sn, cs;
            sincosf(f0, &sn, &cs);
            fc = 0.5f + 0.5f * sn;
            fcd = 0.5f * cs * (float(kPi) * narrow(finv));
        }
    }
}

// One row of an A operand's three part images (K-major, no swizzle; part t
// at img + t * AFL): row m's KP values at core-matrix rows, split into TF32
// high / middle / low parts (zero past R, or all zero).
template <int R, int KP>
__device__ __forceinline__ void put_row(float* img, int m, const float (&v)[R], bool on) {
    constexpr int SBOF = KP * 8;   // floats between row blocks (KP/4 core matrices of 32 floats)
    constexpr int AFL = 128 * KP;  // floats per part image
    float* r0 = img + (m >> 3) * SBOF + (m & 7) * 4;
#pragma unroll
    for (int j = 0; j < KP / 4; j++) {
        float h[4], md[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int k = 4 * j + q;
            const float x = (on && k < R) ? v[k < R ? k : 0] : 0.0f;
            h[q] = tf32_hi(x);
            const float rest = x - h[q];
            md[q] = tf32_hi(rest);
            l[q] = rest - md[q];
        }
        *reinterpret_cast<float4*>(r0 + j * 32) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(r0 + AFL + j * 32) = make_float4(md[0], md[1], md[2], md[3]);
        *reinterpret_cast<float4*>(r0 + 2 * AFL + j * 32) = make_float4(l[0], l[1], l[2], l[3]);
    }
}

// R floats of a pair table (T, or dT/dr that follows it), with the widest loads
// that its place allows: tables start at multiples of 2 R floats.
template <int R, int OFF>
__device__ __forceinline__ void load_tab(const float* tab, float (&v)[R]) {
    if constexpr (R % 2 == 0) {
        constexpr int A = OFF % 4;   // 0 or 2: where the first float lies in its 16 bytes
        if constexpr (A == 2) {
            const float2 q = *reinterpret_cast<const float2*>(tab + OFF);
            v[0] = q.x; v[1] = q.y;
        }
#pragma unroll
        for (int k = A; k + 4 <= R; k += 4) {
            const float4 q = *reinterpret_cast<const float4*>(tab + OFF + k);
            v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
        }
        if constexpr ((R - A) % 4 == 2) {
            const float2 q = *reinterpret_cast<const float2*>(tab + OFF + R - 2);
            v[R - 2] = q.x; v[R - 1] = q.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = tab[OFF + k];
    }
}

// Bounded wait for an mbarrier phase (non-blocking polls, then a back-off).
__device__ __forceinline__ bool mma_wait(uint32_t bar, uint32_t phase) {
    uint32_t done = 0;
    for (int it = 0; it < kTcSpin && !done; it++) {
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (!done && it > 256) __nanosleep(32);
    }
    return done != 0;
}

// The six part products of one operand image with the coefficient image,
// committed to the mbarrier.  Part pairs (operand part, coefficient part),
// smallest first so that the accumulator is small while the small terms go in
// (the tensor core's accumulation rounds each addition at the accumulator's
// magnitude): m.m, h.l, l.h, h.m, m.h, then h.h
template <int KP, int NP>
__device__ __forceinline__ void tc3_mma(uint32_t tmem, uint32_t as, uint32_t bs, uint32_t idesc, uint32_t bar) {
    constexpr uint32_t LBO = 128, SBO = KP * 32;               // bytes: next core matrix in K; next 8 rows
    constexpr uint32_t AB = kTcTile * KP * 4, BB = NP * KP * 4;   // bytes per part image
    constexpr int pa[6] = {1, 0, 2, 0, 1, 0}, pb[6] = {1, 2, 0, 1, 0, 0};
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int t = 0; t < 6; t++) {
#pragma unroll
        for (int ks = 0; ks < KP / 8; ks++) {
            const uint32_t o = ks * 256;   // two core matrices along K per step
            mma_tf32(tmem, umma_desc(as + pa[t] * AB + o, LBO, SBO), umma_desc(bs + pb[t] * BB + o, LBO, SBO), idesc,
                     ks > 0 || t > 0);
        }
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// PC: pairs ij and ik from the pair-table cache.
template <int R, bool PC>
__global__ void __launch_bounds__(128, PC ? kTc3Ctas : 2)
    k_forcetc3(BatchView B, const int* clusters, const int* perm, const long long* perm_n, long long perm_cap) {
    constexpr int KP = tc3_kpad(R);                     // K padded to whole MMA steps (8 for TF32)
    constexpr int NP = tc3_npad(R);                     // N padded to 16
    constexpr int AFL = kTcTile * KP;                   // floats per A part image
    constexpr int BFL = NP * KP;                        // floats per B part image
    static_assert(kTc3Parts == 3, "the MMA sequence pairs three parts");
    static_assert(NP <= (int)kTcCols, "W in one CTA's TMEM columns");
    extern __shared__ __align__(1024) unsigned char smem[];
    float* As = reinterpret_cast<float*>(smem);         // T_ij, then dT_ij/dr: parts h, m, l
    float* Bs = As + 3 * AFL;                           // coefficient parts
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ long long s_tile, s_next;
    __shared__ int s_fail;

    const int tid = threadIdx.x, warp = tid >> 5;
    const long long n = min(*perm_n, perm_cap);
    const long long ntiles = n / kTcTile;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(kTcCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s_fail = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar)));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem, bar = smem_u32(&s_bar);
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NP >> 3) << 17) |
                           ((uint32_t)(kTcTile >> 4) << 24);
    uint32_t phase = 0;
    bool ok = true;                                     // no wait of this thread has run out
    EVWarp acc;

    // Tiles: first a contiguous block per CTA (consecutive tiles share the
    // tuple's coefficient image, so the image is seldom reloaded, and the
    // pair-cache entries and positions of the same atoms), then the last
    // eighth claimed one at a time so that the CTAs finish together.  Claimed
    // one ahead, so that each thread can prefetch its next cluster's data into
    // L2 while the current tile's MMAs run.
    const long long per = ntiles * 7 / 8 / gridDim.x;
    long long own = (long long)blockIdx.x * per;        // thread 0's next tile of its block
    const long long own_end = own + per, shared0 = per * gridDim.x;
    auto claim = [&]() -> long long {
        return own < own_end ? own++ : shared0 + (long long)atomicAdd(&B.queue[0], 1ull);
    };
    if (tid == 0) s_next = claim();
    const DevParamSet* P = nullptr;
    const TupleRec* Rt = nullptr;
    long long bend = 0;                                 // end of the bucket whose tuple and image are loaded
    int c = -1;                                         // this thread's cluster (loaded a tile ahead)
    bool ahead = false;
    for (;;) {
        if (tid == 0) {
            s_tile = *(volatile int*)&s_fail ? ntiles : s_next;
            s_next = s_next < ntiles ? claim() : ntiles;
        }
        __syncthreads();
        const long long tile = s_tile;
        const long long next = s_next;
        if (tile >= ntiles) break;
        const long long base = tile * kTcTile;
        if (!ahead) c = perm[base + tid];
        if (base >= bend) {   // another bucket: its tuple, and the tuple's coefficient image at this width
            const int c0 = perm[base];                  // (a tile never starts in a bucket's padding)
            int id0[3], s0, u0;
            Rt = cluster_tuple<3>(B, clusters, c0 < 0 ? 0 : c0, id0, s0, P, u0);
            bend = B.bk_start[B.bk_key3[c0 < 0 ? 0 : c0] + 1];
            const long long img = Rt->tc_off + tc3_offset(P->R3, R);
            const bool img_ok = ck_bound(B, Rt->tc_off >= 0 && img + (long long)kTc3Parts * BFL <= P->n_tc3);
            const float4* src = reinterpret_cast<const float4*>(P->tc3 + (img_ok ? img : 0));
            float4* dst = reinterpret_cast<float4*>(Bs);
            for (int q = tid; q < kTc3Parts * BFL / 4; q += kTcTile) dst[q] = src[q];
        }
        bool active = c >= 0;
        int at[3] = {0, 0, 0}, s = 0;
        float drf[3][3], rinv[3], fcf[3], fcdf[3];
        float T2[R], D2[R], T1[PC ? 1 : R], D1[PC ? 1 : R], D0[PC ? 1 : R];
        int e0 = 0, e1 = 0;
        const float* pct = reinterpret_cast<const float*>(B.pct3);
        const PairCache* pcd = reinterpret_cast<const PairCache*>(B.pcd3);
#pragma unroll
        for (int q = 0; q < R; q++) T2[q] = D2[q] = 0.0f;
        if constexpr (PC) {
            float T0[R];
#pragma unroll
            for (int q = 0; q < R; q++) T0[q] = 0.0f;
            if (active) {
                const int2 ee = *reinterpret_cast<const int2*>(B.c3e + 2LL * c);
                e0 = ee.x; e1 = ee.y;
                load_tab<R, 0>(pct + (long long)e0 * 2 * R, T0);
            }
            put_row<R, KP>(As, tid, T0, active);
        } else {
            // geometry, cutoff early-outs and tables of the three pairs
            float T0[R];
            double rr[3] = {0, 0, 0};
#pragma unroll
            for (int q = 0; q < R; q++) T0[q] = D0[q] = T1[q] = D1[q] = 0.0f;
            if (active) {
                int id[3];
                for (int k = 0; k < 3; k++) {
                    id[k] = clusters[3LL * c + k];
                    at[k] = B.atom_orig[B.ghost_parent[id[k]]];
                }
                s = B.atom_sys[B.ghost_parent[id[0]]];
#pragma unroll
                for (int p = 0; p < 3; p++) {
                    double d[3];
                    pair_geom(B, B.sys[s].h, id[Topo<3>::a(p)], id[Topo<3>::b(p)], d, rr[p]);
                    drf[p][0] = float(d[0]); drf[p][1] = float(d[1]); drf[p][2] = float(d[2]);
                    rinv[p] = 1.0f / float(rr[p]);
                    if (rr[p] >= Rt->rout[p]) active = false;   // compute_3B's early-outs
                }
            }
            if (active) {   // (powers above the set's own R3 multiply zero coefficients)
                pair_regs<R>(*P, *Rt, 0, rr[0], T0, D0, fcf[0], fcdf[0], B.flags);
                pair_regs<R>(*P, *Rt, 1, rr[1], T1, D1, fcf[1], fcdf[1], B.flags);
                pair_regs<R>(*P, *Rt, 2, rr[2], T2, D2, fcf[2], fcdf[2], B.flags);
            }
            put_row<R, KP>(As, tid, T0, active);
        }
        // generic-proxy writes of the operands -> visible to the tensor core
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) tc3_mma<KP, NP>(tmem, smem_u32(As), smem_u32(Bs), idesc, bar);
        ahead = next < ntiles;
        const int cn = ahead ? perm[next * kTcTile + tid] : -1;
        if constexpr (PC) {
            // while the MMAs run: pair jk
            if (active) {
                const int fl0 = pcd[e0].flags, fl1 = pcd[e1].flags;
                int id[3];
                for (int k = 0; k < 3; k++) {
                    id[k] = clusters[3LL * c + k];
                    if (!ck_bound(B, id[k] >= 0 && id[k] < B.n_ghost_total)) id[k] = 0;
                    const int a = B.ghost_parent[id[k]];
                    if (k == 0) s = B.atom_sys[a];
                    at[k] = B.atom_orig[a];
                }
                double d[3], r;
                pair_geom(B, B.sys[s].h, id[1], id[2], d, r);
                active = !((fl0 | fl1) & kPairFar) && less_pos(r, Rt->rout[2]);   // compute_3B's early-outs
                if (active) {
                    const int oor = (fl0 & kPairOor ? 1 : 0) + (fl1 & kPairOor ? 1 : 0);
                    if (oor) atomicAdd(&B.flags[4], oor);
                    pair_regs<R>(*P, *Rt, 2, r, T2, D2, fcf[2], fcdf[2], B.flags);
                    drf[2][0] = narrow(d[0]); drf[2][1] = narrow(d[1]); drf[2][2] = narrow(d[2]);
                    rinv[2] = 1.0f / narrow(r);
                }
            }
        }
        ok = ok && mma_wait(bar, phase);
        phase ^= 1u;
        if (!ok) s_fail = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // this thread's TMEM row (lane = tid): W at columns [0, NP)
        float V[R], V2[R];
#pragma unroll
        for (int b = 0; b < R; b++) V[b] = V2[b] = 0.0f;
        const uint32_t row = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int q = 0; q < NP / 16; q++) {
            float w[16];
            tmem_ld16(row + 16 * q, w);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int u = 0; u < 16; u++) {
                const int j = 16 * q + u;
                if (j < R * R) {
                    const int b = j / R, cc = j % R;
                    V[b] += w[u] * T2[cc];
                    V2[b] += w[u] * D2[cc];
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        // the row gradient: dT_ij/dr through the same operand image and columns
        if constexpr (PC) {
            float D[R];
#pragma unroll
            for (int q = 0; q < R; q++) D[q] = 0.0f;
            if (active) load_tab<R, R>(pct + (long long)e0 * 2 * R, D);
            put_row<R, KP>(As, tid, D, active);
        } else {
            put_row<R, KP>(As, tid, D0, active);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) tc3_mma<KP, NP>(tmem, smem_u32(As), smem_u32(Bs), idesc, bar);
        float S = 0.0f, G0 = 0.0f, G1 = 0.0f, G2 = 0.0f;
        float U1[R];   // T_ik
#pragma unroll
        for (int q = 0; q < R; q++) U1[q] = 0.0f;
        if constexpr (PC) {
            if (cn >= 0) {   // the next tile's entries into L2
                const int2 ee = *reinterpret_cast<const int2*>(B.c3e + 2LL * cn);
                const int* ids = clusters + 3LL * cn;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(B.ghost_fs + 3LL * ids[1]));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(B.ghost_fs + 3LL * ids[2]));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pcd + ee.x));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pcd + ee.y));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pct + (long long)ee.x * 2 * R));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pct + (long long)ee.x * 2 * R + R + R - 1));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pct + (long long)ee.y * 2 * R));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(pct + (long long)ee.y * 2 * R + R + R - 1));
            }
            if (active) {
                const float* tab = pct + (long long)e1 * 2 * R;
                float D[R];
                load_tab<R, 0>(tab, U1);
                load_tab<R, R>(tab, D);
#pragma unroll
                for (int b = 0; b < R; b++) {
                    S += V[b] * U1[b];
                    G1 += V[b] * D[b];
                    G2 += V2[b] * U1[b];
                }
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const float4* g = reinterpret_cast<const float4*>(pcd + (p == 0 ? e0 : e1));
                    const float4 u = g[2];   // (whole words: a gather costs L1 as much for one as for four)
                    const float2 v = *reinterpret_cast<const float2*>(g + 3);
                    drf[p][0] = u.x; drf[p][1] = u.y; drf[p][2] = u.z;
                    rinv[p] = u.w;
                    fcf[p] = v.x;
                    fcdf[p] = v.y;
                }
            }
        } else {
#pragma unroll
            for (int b = 0; b < R; b++) {
                U1[b] = T1[b];
                S += V[b] * T1[b];
                G1 += V[b] * D1[b];
                G2 += V2[b] * T1[b];
            }
        }
        ok = ok && mma_wait(bar, phase);
        phase ^= 1u;
        if (!ok) s_fail = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float Vp[R];
#pragma unroll
        for (int b = 0; b < R; b++) Vp[b] = 0.0f;
#pragma unroll
        for (int q = 0; q < NP / 16; q++) {
            float w[16];
            tmem_ld16(row + 16 * q, w);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int u = 0; u < 16; u++) {
                const int j = 16 * q + u;
                if (j < R * R) Vp[j / R] += w[u] * T2[j % R];
            }
        }
        // (the next tile's MMAs rewrite the columns after the barrier that follows)
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        double e_c = 0.0, vir_c[6] = {0, 0, 0, 0, 0, 0};
        if (active) {
#pragma unroll
            for (int b = 0; b < R; b++) G0 += Vp[b] * U1[b];
            const float G[3] = {G0, G1, G2};
            cluster_epilogue_f32<3>(B, at, drf, rinv, fcf, fcdf, S, G, e_c, vir_c);
        }
        acc.add(B, s, e_c, vir_c, active);
        c = cn;
    }
    acc.flush(B);
    if (!ok) atomicOr(&B.flags[7], 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols));
}

template <int R, bool PC>
void launch_tc_rp(const BatchView& B, cudaStream_t st) {
    constexpr int KP = tc3_kpad(R);
    constexpr int NP = tc3_npad(R);
    size_t smem = sizeof(float) * kTc3Parts * ((size_t)kTcTile * KP + (size_t)NP * KP);
    if (smem < kTcMinSmem) smem = kTcMinSmem;
    auto kern = k_forcetc3<R, PC>;
    // the kernel's own dynamic size (its static shared memory counts against
    // the opt-in maximum, so the largest value is not accepted here); every
    // launch of a width asks for the same size, so concurrent callers agree
    cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const long long tiles = B.perm3_cap / kTcTile;
    long long want = (long long)(PC ? kTc3Ctas : 2) * sm_count();
    const unsigned grid = (unsigned)(want < tiles ? want : (tiles > 0 ? tiles : 1));
    const long long* pn = B.bk_start + B.nbk3;
    count_launch(), kern<<<grid, kTcTile, smem, st>>>(B, B.c3, B.perm3, pn, B.perm3_cap);
}
template <int R>
void launch_tc_r(const BatchView& B, cudaStream_t st) {
    if (B.use_pc3) launch_tc_rp<R, true>(B, st);
    else launch_tc_rp<R, false>(B, st);
}


// ---------------------------------------------------------------------------
// Tensor-core 4-body contraction (mixed form).  With R powers per pair a
// tuple's coefficients form a dense matrix A[I][J], I = (q_ij, q_ik, q_il) and
// J = (q_jk, q_jl, q_kl) (R^3 each).  For a cluster, X_I = T_ij T_ik T_il and
// Y_J = T_jk T_jl T_kl: S = X.A.Y, and the pair gradients are
//   G_ij = dX_ij.A.Y, G_ik = dX_ik.A.Y, G_il = dX_il.A.Y  (dX_p: T_p -> dT_p/dr)
//   G_jk, G_jl, G_kl = W.dY_p with W = X.A.
// A tile is 32 clusters of one tuple and the MMA's 128 rows are the four row
// vectors X, dX_ij, dX_ik, dX_il of each (row 32 v + c: warp v builds variant
// v of cluster c and reads its TMEM row back), so one M = 128, N = R^3 MMA
// chain gives W, W_ij, W_ik, W_il for all 32 clusters; each row is then
// contracted with the cluster's column tables, and warp 0 forms the forces.
// Operands in three TF32 parts as in the 3-body kernel: the five small part
// products (smallest first) and the large one go into two accumulators that
// are summed in FP32.
//
// One CTA of three groups of 128 threads per SM: the groups share the tuple's
// coefficient image (49 KB at R = 4) and each works on its own tile, with its
// own barrier, mbarrier, operand buffer (49 KB) and 2 x 64 TMEM columns, so that one
// group's waits are covered by the others.  The A operand goes through the
// group's buffer in halves along K (R = 4; four groups with quarters sum the
// small products in another order, 4e-10 off).  With the pair-table cache a thread
// loads its variant's tables of ij, ik and il, and warps 1-3 set up jk, jl and
// kl while the first MMAs run.  What
// warp 0 reads for the forces is kept for two tiles, so that the other warps
// go on to the next one.  Bound: latency of the chain tables - operand - MMAs -
// TMEM at 12 warps an SM, the FP64 pipe at 23%.  Measured: 292 k quadruplets of
// 32768 atoms 530 -> 276 us, 1.83 M of 2000 configurations 3.3 -> 1.69 ms, against two
// CTAs of 128 threads with six pairs set up per cluster.
constexpr int kTc4Tile = 32;              // clusters per tile
constexpr size_t kTc4MinSmem = 184 * 1024;   // no room for another tensor-core CTA on the SM (TMEM)

// A group's shared memory besides its operand buffer; NT pairs, the last ones.
template <int R, int NT>
struct Tc4Group {
    float tab[NT][2 * R][kTc4Tile];       // T, then dT/dr
    struct {
        float dr[NT][3][kTc4Tile], rinv[NT][kTc4Tile], fc[NT][kTc4Tile], fcd[NT][kTc4Tile];
        int fl[NT][kTc4Tile];             // kPairFar, kPairOor
        float res[7][kTc4Tile];           // S, G_0 .. G_5
    } epi[2];
};

template <int R>
struct Tc4Shape {
    static constexpr int N3 = R * R * R;
    static constexpr int KP = tc4_kpad(N3);             // K padded to whole MMA steps
    static constexpr int NP = tc4_npad(N3);             // N padded to 16
    static constexpr int KH = KP > 32 ? KP / 2 : KP;    // K per pass through the operand buffer
    static constexpr int AFL = 128 * KH;                // floats per A part image (one pass)
    static constexpr int BFL = NP * KP;                 // floats per B part image
};

__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }

// tiles in flight per CTA, as many as the shared memory holds (one CTA per SM)
CK_HD constexpr int tc4_groups(bool pc) { return pc ? 3 : 2; }

template <int R, bool PC>
__global__ void __launch_bounds__(128 * tc4_groups(PC), 1)
    k_forcetc4(BatchView B, const int* clusters, const int* perm, const long long* perm_n, long long perm_cap) {
    using Sh = Tc4Shape<R>;
    constexpr int N3 = Sh::N3, KP = Sh::KP, NP = Sh::NP, KH = Sh::KH, AFL = Sh::AFL, BFL = Sh::BFL;
    constexpr int NH = KP / KH;
    constexpr int NG = tc4_groups(PC);
    constexpr int NT = PC ? 3 : 6, P0 = 6 - NT;         // pairs set up here: P0 .. 5
    constexpr uint32_t LBO = 128, SBOA = KH * 32, SBOB = KP * 32;   // bytes: next core matrix in K; next 8 rows
    // TMEM: the large (h.h) and the small part products in separate
    // accumulators, summed in FP32 at the end (each accumulates its own terms
    // in order of size within a pass)
    constexpr uint32_t DCOL = NP <= 32 ? 32 : (NP <= 64 ? 64 : 128);
    constexpr uint32_t COLS = 2 * DCOL;
    constexpr uint32_t ALLOC = COLS * NG <= 128 ? 128 : (COLS * NG <= 256 ? 256 : 512);
    static_assert(COLS * NG <= ALLOC, "the groups' accumulators in one SM's TMEM");
    constexpr int C = kTc4Tile;
    static_assert(kTc3Parts == 3, "the MMA sequence below pairs three parts");
    extern __shared__ __align__(1024) unsigned char smem[];
    float* Bs = reinterpret_cast<float*>(smem);         // coefficient parts
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar[NG];
    __shared__ long long s_lo, s_hi;
    __shared__ int s_fail;

    const int tid = threadIdx.x, grp = tid >> 7, gt = tid & 127, warp = gt >> 5, c = tid & 31;
    float* As = Bs + 3 * BFL + grp * 3 * AFL;           // rows X / dX parts h, m, l
    auto& sm = reinterpret_cast<Tc4Group<R, NT>*>(Bs + 3 * BFL + NG * 3 * AFL)[grp];
    const long long n = min(*perm_n, perm_cap);
    const long long ntiles = n / C;
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(ALLOC));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s_fail = 0;
        for (int k = 0; k < NG; k++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_bar[k])));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem + grp * COLS, bar = smem_u32(&s_bar[grp]);
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NP >> 3) << 17) |
                           ((uint32_t)(128 >> 4) << 24);
    uint32_t phase = 0;
    int par = 0;
    bool ok = true;                                     // no wait of this thread has run out
    EVWarp acc;
    const float* pct = reinterpret_cast<const float*>(B.pct4);
    const PairCache* pcd = reinterpret_cast<const PairCache*>(B.pcd4);

    // tiles: a contiguous block per CTA, then the last eighth a few at a time
    const long long per = ntiles * 7 / 8 / gridDim.x;
    const long long shared0 = per * gridDim.x;
    bool first = per > 0;
    const DevParamSet* P = nullptr;
    const TupleRec* Rt = nullptr;
    long long bend = 0;                                 // end of the bucket whose tuple and image are loaded
    long long lo = 0, hi = 0;
    for (;;) {
        // a run of tiles of one bucket, the groups in turn
        __syncthreads();                                // (the groups have left the last run)
        if (lo >= hi) {
            if (tid == 0) {
                s_lo = first ? (long long)blockIdx.x * per
                             : shared0 + NG * (long long)atomicAdd(&B.queue[1], 1ull);
                s_hi = min(first ? s_lo + per : s_lo + NG, ntiles);
                if (*(volatile int*)&s_fail) s_hi = s_lo;
            }
            __syncthreads();
            first = false;
            lo = s_lo;
            hi = s_hi;
            if (lo >= hi) break;
        }
        if (lo * C >= bend) {
            const int c0 = max(perm[lo * C], 0);        // (a tile never starts in a bucket's padding)
            int id0[4], s0, u0;
            Rt = cluster_tuple<4>(B, clusters, c0, id0, s0, P, u0);
            bend = max(B.bk_start[B.nbk3 + 1 + B.bk_key4[c0] + 1], (lo + 1) * C);
            const long long img = Rt->tc_off;
            const bool img_ok = ck_bound(B, img >= 0 && img + (long long)kTc3Parts * BFL <= P->n_tc4);
            const float4* src = reinterpret_cast<const float4*>(P->tc4 + (img_ok ? img : 0));
            float4* dst = reinterpret_cast<float4*>(Bs);
            for (int q = tid; q < kTc3Parts * BFL / 4; q += 128 * NG) dst[q] = src[q];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
        const long long end = min(hi, bend / C);
        int cl = lo + grp < end ? perm[(lo + grp) * C + c] : -1;
        for (long long tile = lo + grp; tile < end; tile += NG, par ^= 1) {
            auto& ep = sm.epi[par];
            const int cln = tile + NG < end ? perm[(tile + NG) * C + c] : -1;
            // this cluster's row tables: T, or in variant 1-3 dT/dr of one pair
            float f0[R], f1[R], f2[R];
            int e[3] = {0, 0, 0};
            // sets up pair p (its vector d) for the contraction and the forces
            auto set_pair = [&](int p, const double* d, double r, bool on) {
                float T[R], D[R], fc = 0.0f, fcd = 0.0f;
#pragma unroll
                for (int q = 0; q < R; q++) T[q] = D[q] = 0.0f;
                const bool far = !on || !less_pos(r, Rt->rout[p]);   // compute_4B's early-outs
                if (!far) pair_regs<R>(*P, *Rt, p, r, T, D, fc, fcd, nullptr);
                const int R4 = P->R4;   // the set's own powers; entries above it multiply zero coefficients
#pragma unroll
                for (int q = 0; q < R; q++) {
                    sm.tab[p - P0][q][c] = q < R4 ? T[q] : 0.0f;
                    sm.tab[p - P0][R + q][c] = q < R4 ? D[q] : 0.0f;
                }
                ep.fl[p - P0][c] = (far ? kPairFar : 0) | (!far && less_pos(r, Rt->rin[p]) ? kPairOor : 0);
                ep.fc[p - P0][c] = fc;
                ep.fcd[p - P0][c] = fcd;
                ep.rinv[p - P0][c] = far ? 0.0f : 1.0f / narrow(r);
                for (int k = 0; k < 3; k++) ep.dr[p - P0][k][c] = narrow(d[k]);
            };
            if constexpr (PC) {
#pragma unroll
                for (int q = 0; q < R; q++) f0[q] = f1[q] = f2[q] = 0.0f;
                if (cl >= 0) {
                    for (int k = 0; k < 3; k++) e[k] = B.c4e[3LL * cl + k];
                    load_tab<R, 0>(pct + (long long)e[0] * 2 * R + (warp == 1 ? R : 0), f0);
                    load_tab<R, 0>(pct + (long long)e[1] * 2 * R + (warp == 2 ? R : 0), f1);
                    load_tab<R, 0>(pct + (long long)e[2] * 2 * R + (warp == 3 ? R : 0), f2);
                }
            } else {
                int id[4] = {0, 0, 0, 0}, sy = 0;
                if (cl >= 0) {
                    for (int k = 0; k < 4; k++) id[k] = clusters[4LL * cl + k];
                    sy = B.atom_sys[B.ghost_parent[id[0]]];
                }
                for (int p = warp; p < 6; p += 4) {   // the four warps cover the six pairs
                    double d[3] = {0, 0, 0}, r = 1e300;
                    if (cl >= 0) pair_geom(B, B.sys[sy].h, id[Topo<4>::a(p)], id[Topo<4>::b(p)], d, r);
                    set_pair(p, d, r, cl >= 0);
                }
                group_sync(grp);
#pragma unroll
                for (int q = 0; q < R; q++) {
                    f0[q] = sm.tab[0][(warp == 1 ? R : 0) + q][c];
                    f1[q] = sm.tab[1][(warp == 2 ? R : 0) + q][c];
                    f2[q] = sm.tab[2][(warp == 3 ? R : 0) + q][c];
                }
            }
            // row 32 warp + c of the A operand, KH columns at a time
            int at[4] = {0, 0, 0, 0}, s = 0;
            float* r0 = As + (gt >> 3) * (KH * 8) + (gt & 7) * 4;
#pragma unroll
            for (int hf = 0; hf < NH; hf++) {
                if (hf > 0) {   // the previous part's MMAs have read the buffer
                    ok = ok && mma_wait(bar, phase);
                    phase ^= 1u;
                }
#pragma unroll
                for (int j = 0; j < KH / 4; j++) {
                    float h[4], md[4], l[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int k = hf * KH + 4 * j + u;
                        const int kk = k < N3 ? k : 0;
                        const float x = k < N3 ? f0[kk / (R * R)] * f1[(kk / R) % R] * f2[kk % R] : 0.0f;
                        h[u] = tf32_hi(x);
                        const float rest = x - h[u];
                        md[u] = tf32_hi(rest);
                        l[u] = rest - md[u];
                    }
                    *reinterpret_cast<float4*>(r0 + j * 32) = make_float4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<float4*>(r0 + AFL + j * 32) = make_float4(md[0], md[1], md[2], md[3]);
                    *reinterpret_cast<float4*>(r0 + 2 * AFL + j * 32) = make_float4(l[0], l[1], l[2], l[3]);
                }
                // generic-proxy writes of the operands -> visible to the tensor core
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                group_sync(grp);
                if (gt == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t as = smem_u32(As), bs = smem_u32(Bs);
                    constexpr uint32_t AB = AFL * 4, BB = BFL * 4;   // bytes per part image
                    // small part products smallest first (m.m, h.l, l.h, h.m, m.h) into
                    // the first accumulator, h.h into the second
                    constexpr int pa[6] = {1, 0, 2, 0, 1, 0}, pb[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
                    for (int t = 0; t < 6; t++) {
#pragma unroll
                        for (int ks = 0; ks < KH / 8; ks++) {
                            const uint32_t oa = ks * 256;                       // two core matrices along K per step
                            const uint32_t ob = (hf * (KH / 8) + ks) * 256;
                            const uint32_t dd = t < 5 ? tmem : tmem + DCOL;
                            mma_tf32(dd, umma_desc(as + pa[t] * AB + oa, LBO, SBOA),
                                     umma_desc(bs + pb[t] * BB + ob, LBO, SBOB), idesc,
                                     hf > 0 || ks > 0 || (t > 0 && t < 5));
                        }
                    }
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                                 : "memory");
                }
                if (hf == 0) {
                    if (PC && cl >= 0) {   // warp 0: the atoms; warps 1-3: pair jk, jl or kl
                        int id[4];
                        for (int k = 0; k < 4; k++) {
                            id[k] = clusters[4LL * cl + k];
                            if (!ck_bound(B, id[k] >= 0 && id[k] < B.n_ghost_total)) id[k] = 0;
                        }
                        s = B.atom_sys[B.ghost_parent[id[0]]];
                        if (warp == 0) {
                            for (int k = 0; k < 4; k++) at[k] = B.atom_orig[B.ghost_parent[id[k]]];
                        } else {
                            double d[3], r;
                            pair_geom(B, B.sys[s].h, id[warp < 3 ? 1 : 2], id[warp == 1 ? 2 : 3], d, r);
                            set_pair(2 + warp, d, r, true);
                        }
                    }
                    if (!PC && warp == 0 && cl >= 0)
                        for (int k = 0; k < 4; k++) {
                            const int a = B.ghost_parent[clusters[4LL * cl + k]];
                            if (k == 0) s = B.atom_sys[a];
                            at[k] = B.atom_orig[a];
                        }
                    if (NH == 1) group_sync(grp);
                }
            }
            ok = ok && mma_wait(bar, phase);
            phase ^= 1u;
            if (!ok) s_fail = 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // this thread's TMEM row (small + large products), contracted with the
            // cluster's column tables (jk: d, jl: e, kl: f; J = (d R + e) R + f)
            {
                float T3[R], D3[R], T4[R], D4[R], T5[R], D5[R];
#pragma unroll
                for (int q = 0; q < R; q++) {
                    T3[q] = sm.tab[3 - P0][q][c]; D3[q] = sm.tab[3 - P0][R + q][c];
                    T4[q] = sm.tab[4 - P0][q][c]; D4[q] = sm.tab[4 - P0][R + q][c];
                    T5[q] = sm.tab[5 - P0][q][c]; D5[q] = sm.tab[5 - P0][R + q][c];
                }
                const uint32_t row = tmem + ((uint32_t)(warp * 32) << 16);
                float S = 0.0f, G3 = 0.0f, G4 = 0.0f, G5 = 0.0f;
                float w = 0.0f, w1 = 0.0f, w2 = 0.0f, u = 0.0f, u1 = 0.0f;
#pragma unroll
                for (int q = 0; q < NP / 16; q++) {
                    float W[16], big[16];
                    tmem_ld16(row + 16 * q, W);
                    tmem_ld16(row + DCOL + 16 * q, big);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int v = 0; v < 16; v++) {
                        const int j = 16 * q + v;
                        if (j < N3) {
                            const int d = j / (R * R), ee = (j / R) % R, f = j % R;
                            const float x = W[v] + big[v];
                            u += x * T5[f];
                            u1 += x * D5[f];
                            if (f == R - 1) {
                                w += u * T4[ee];
                                w1 += u * D4[ee];
                                w2 += u1 * T4[ee];
                                u = u1 = 0.0f;
                                if (ee == R - 1) {
                                    S += w * T3[d];
                                    G3 += w * D3[d];
                                    G4 += w1 * T3[d];
                                    G5 += w2 * T3[d];
                                    w = w1 = w2 = 0.0f;
                                }
                            }
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                if (warp == 0) {
                    ep.res[0][c] = S;
                    ep.res[4][c] = G3;
                    ep.res[5][c] = G4;
                    ep.res[6][c] = G5;
                } else {
                    ep.res[warp][c] = S;   // G_ij, G_ik, G_il from the derivative rows
                }
            }
            group_sync(grp);
            if (warp == 0) {
                double e_c = 0.0, vir_c[6] = {0, 0, 0, 0, 0, 0};
                bool active = cl >= 0;
                if (active) {
                    float dr[6][3], rinv[6], fc[6], fcd[6], G[6];
                    int far = 0, oor = 0;
#pragma unroll
                    for (int p = 0; p < 6; p++) {
                        int fl;
                        if (p < P0) {
                            const float4* g = reinterpret_cast<const float4*>(pcd + e[p < 3 ? p : 0]);
                            const float4 u = g[2], v = g[3];
                            dr[p][0] = u.x; dr[p][1] = u.y; dr[p][2] = u.z;
                            rinv[p] = u.w;
                            fc[p] = v.x;
                            fcd[p] = v.y;
                            fl = __float_as_int(v.z);
                        } else {
                            const int t = p < P0 ? 0 : p - P0;
                            dr[p][0] = ep.dr[t][0][c]; dr[p][1] = ep.dr[t][1][c]; dr[p][2] = ep.dr[t][2][c];
                            rinv[p] = ep.rinv[t][c];
                            fc[p] = ep.fc[t][c];
                            fcd[p] = ep.fcd[t][c];
                            fl = ep.fl[t][c];
                        }
                        far |= fl & kPairFar;
                        oor += fl & kPairOor ? 1 : 0;
                        G[p] = ep.res[1 + p][c];
                    }
                    active = !far;
                    if (active) {
                        if (oor) atomicAdd(&B.flags[4], oor);
                        cluster_epilogue_f32<4>(B, at, dr, rinv, fc, fcd, ep.res[0][c], G, e_c, vir_c);
                    }
                }
                acc.add(B, s, e_c, vir_c, active);
            }
            cl = cln;
        }
        lo = end;
    }
    if (warp == 0) acc.flush(B);
    if (!ok) atomicOr(&B.flags[7], 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ALLOC));
}

template <int R, bool PC>
void launch_tc4_rp(const BatchView& B, cudaStream_t st) {
    using Sh = Tc4Shape<R>;
    constexpr int NG = tc4_groups(PC);
    size_t smem = sizeof(float) * kTc3Parts * ((size_t)Sh::BFL + NG * (size_t)Sh::AFL) +
                  NG * sizeof(Tc4Group<R, PC ? 3 : 6>);
    if (smem < kTc4MinSmem) smem = kTc4MinSmem;
    auto kern = k_forcetc4<R, PC>;
    cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const long long need = (B.perm4_cap / kTc4Tile + NG - 1) / NG;
    const long long want = sm_count();
    const unsigned grid = (unsigned)(want < need ? want : (need > 0 ? need : 1));
    const long long* pn = B.bk_start + B.nbk3 + 1 + B.nbk4;
    count_launch(), kern<<<grid, 128 * NG, smem, st>>>(B, B.c4, B.perm4, pn, B.perm4_cap);
}
template <int R>
void launch_tc4_r(const BatchView& B, cudaStream_t st) {
    if (B.use_pc4) launch_tc4_rp<R, true>(B, st);
    else launch_tc4_rp<R, false>(B, st);
}

}  // namespace

bool tc3_supported(int rf3) { return rf3 >= 2 && rf3 <= kTc3MaxR; }
bool tc4_supported(int rf4) { return rf4 >= 2 && rf4 <= kTc4MaxR; }

void launch_force4tc(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm4_cap <= 0 || B.nbk4 <= 0) return;
    switch (L.rf4) {
        case 2: launch_tc4_r<2>(B, st); break;
        case 3: launch_tc4_r<3>(B, st); break;
        case 4: launch_tc4_r<4>(B, st); break;
        default: break;
    }
}

void launch_force3tc(const BatchView& B, const ForceLaunch& L, cudaStream_t st) {
    if (B.perm3_cap <= 0 || B.nbk3 <= 0) return;
    switch (L.rf3) {
        case 2: launch_tc_r<2>(B, st); break;
        case 3: launch_tc_r<3>(B, st); break;
        case 4: launch_tc_r<4>(B, st); break;
        case 5: launch_tc_r<5>(B, st); break;
        case 6: launch_tc_r<6>(B, st); break;
        case 7: launch_tc_r<7>(B, st); break;
        case 8: launch_tc_r<8>(B, st); break;
        case 9: launch_tc_r<9>(B, st); break;
        case 10: launch_tc_r<10>(B, st); break;
        case 11: launch_tc_r<11>(B, st); break;
        default: break;
    }
}

}  // namespace ck
