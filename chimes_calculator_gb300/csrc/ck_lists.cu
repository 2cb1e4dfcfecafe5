// Cluster-list build on the GPU: periodic ghost images, the bin grid, the 2B
// neighbour lists and the 3B/4B cluster enumeration.
//
// The lists must be the reference's lists exactly (same members, same order),
// because cluster membership is decided by floating-point distance tests.
// Every floating-point step whose result decides membership therefore uses
// explicit round-to-nearest intrinsics (__dmul_rn/__dadd_rn/__dsub_rn/
// __ddiv_rn/__dsqrt_rn), which the compiler never fuses, in the reference's
// evaluation order:
//   set-up, wrap, reorient, ghosts ... serial_interface/src/serial_chimes_interface.cpp:150-587
//   bins and lists ................... serial_chimes_interface.cpp:588-864
//   get_dist ......................... serial_interface/src/serial_chimes_interface.h:141-215
//
// Two shortcuts keep the result exact while doing less work than the
// reference:
//  * only the ghost images that can lie within the search radius of the
//    primary cell are generated (host bound in ck_geom.cpp); the bin grid still
//    spans the bounding box of ALL images, which is exact from the corner
//    images alone: a ghost coordinate is a composition of IEEE-rounded sums and
//    products, each monotone in the image shift, so over the shift box its
//    extremes sit at the corners;
//  * distances are first tested in FP32 with a margin (SysDesc::eps) far above
//    the FP32 error; only a distance within the margin of a cutoff, and every
//    distance that is stored, is evaluated exactly in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "ck_common.h"
#include "ck_kernels.h"
#include "ck_launch.cuh"

namespace ck {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// o = m * (x,y,z) with the reference's association ((m0 x + m1 y) + m2 z)
__device__ __forceinline__ void mv(const double* m, double x, double y, double z, double* o) {
    o[0] = add(add(mul(m[0], x), mul(m[1], y)), mul(m[2], z));
    o[1] = add(add(mul(m[3], x), mul(m[4], y)), mul(m[5], z));
    o[2] = add(add(mul(m[6], x), mul(m[7], y)), mul(m[8], z));
}

// get_dist on stored fractional coordinates: |H (f_j - f_i)|; r = H (f_j - f_i)
__device__ __forceinline__ double dist_frac(const double* H, const double* fi, const double* fj, double* r = nullptr) {
    double dx = sub(fj[0], fi[0]), dy = sub(fj[1], fi[1]), dz = sub(fj[2], fi[2]);
    double r0 = add(add(mul(H[0], dx), mul(H[1], dy)), mul(H[2], dz));
    double r1 = add(add(mul(H[3], dx), mul(H[4], dy)), mul(H[5], dz));
    double r2 = add(add(mul(H[6], dx), mul(H[7], dy)), mul(H[8], dz));
    if (r) { r[0] = r0; r[1] = r1; r[2] = r2; }
    return __dsqrt_rn(add(add(mul(r0, r0), mul(r1, r1)), mul(r2, r2)));
}

__device__ __forceinline__ int find_sys_atom(const SysDesc* sys, int n, long long a) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (sys[mid].atom_off <= a) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int find_sys_ghost(const SysDesc* sys, int n, long long g) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (sys[mid].ghost_off <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// order-preserving unsigned key of a double (for atomicMin/atomicMax)
__device__ __forceinline__ unsigned long long okey(double v) {
    unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_inv(unsigned long long k) {
    unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)u);
}

// reference ghost image number of shift (i,j,k): 1.. for the images of
// build_layered_system's (i,j,k) loop, skipping (0,0,0)
__device__ __forceinline__ int image_index(int i, int j, int k, int n, int side) {
    const int full = ((i + n) * side + (j + n)) * side + (k + n);
    const int center = (n * side + n) * side + n;
    return full < center ? full + 1 : full;
}

// kept image shifts of an atom with reoriented fractional coordinates fn:
// s_k in [lo_k, lo_k + cnt_k), shift 0 (the atom itself) always included
struct ShiftBox {
    int lo[3], cnt[3], count;
};
__device__ __forceinline__ void shift_box(const SysDesc& d, const double* fn, ShiftBox& b) {
    const int n = d.n_layers;
    b.count = 1;
    for (int k = 0; k < 3; k++) {
        int lo = (int)ceil(d.ulo[k] - fn[k]), hi = (int)floor(d.uhi[k] - fn[k]);
        lo = lo < -n ? -n : lo;
        hi = hi > n ? n : hi;
        lo = lo > 0 ? 0 : lo;
        hi = hi < 0 ? 0 : hi;
        b.lo[k] = lo;
        b.cnt[k] = hi - lo + 1;
        b.count *= b.cnt[k];
    }
}

// bin grid of a system from its bounding box (build_neigh_lists :622-642)
__device__ __forceinline__ void bin_setup(const BatchView& B, int s, SysDesc& d) {
    long long total = 1;
    for (int c = 0; c < 3; c++) {
        const double mn = okey_inv(__ldcg(&B.minmax[6 * s + c])), mx = okey_inv(__ldcg(&B.minmax[6 * s + 3 + c]));
        d.minpos[c] = mn;
        int nb = (int)ceil(__ddiv_rn(sub(mx, mn), d.search));
        if (nb < 1) nb = 1;
        d.nb[c] = nb;
        total *= nb;
    }
    if (total > d.bin_cap) {
        d.err = kErrCapacity;
        atomicOr(&B.flags[0], 1);
    }
}

// --- 1. atoms: replicate (small=true), wrap, reorient, bounding box --------
// simulation_system::init (:196-322) and reorient (:352-405).  The bounding box
// of all ghost images (build_neigh_lists :590-610) comes from each atom, its
// two corner images per axis, reduced per system.
__global__ void k_atoms(BatchView B) {
    chain_begin();
    const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = r < B.n_atoms_total;
    int s = -1;
    double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    if (valid) {
        s = find_sys_atom(B.sys, B.n_sys, r);
        const SysDesc& d = B.sys[s];
        const int rl = (int)(r - d.atom_off);
        const int a = rl % d.n_in, blk = rl / d.n_in;
        const double* xin = B.in_pos + 3 * (d.in_off + a);
        double x[3] = {xin[0], xin[1], xin[2]};
        if (blk > 0) {
            const int nr1 = d.n_rep + 1;
            const int i = blk / (nr1 * nr1), j = (blk / nr1) % nr1, k = blk % nr1;
            double t[3];
            mv(d.h0i, x[0], x[1], x[2], t);
            t[0] = add(t[0], (double)i); t[1] = add(t[1], (double)j); t[2] = add(t[2], (double)k);
            mv(d.h0, t[0], t[1], t[2], x);
        }
        double f[3], xw[3], fa[3], xn[3], fn[3];
        mv(d.hi, x[0], x[1], x[2], f);
        f[0] = sub(f[0], floor(f[0])); f[1] = sub(f[1], floor(f[1])); f[2] = sub(f[2], floor(f[2]));
        mv(d.h, f[0], f[1], f[2], xw);
        mv(d.hi, xw[0], xw[1], xw[2], fa);
        mv(d.hn, fa[0], fa[1], fa[2], xn);
        mv(d.hni, xn[0], xn[1], xn[2], fn);
        ShiftBox sb;
        shift_box(d, fn, sb);
        if (sb.count > d.gstride) atomicOr(&B.flags[0], 16);   // slot bound violated (cannot happen)
        const int j0 = ((0 - sb.lo[0]) * sb.cnt[1] + (0 - sb.lo[1])) * sb.cnt[2] + (0 - sb.lo[2]);
        const long long q = d.ghost_off + (long long)rl * d.gstride + (j0 < d.gstride ? j0 : 0);
        for (int c = 0; c < 3; c++) {
            B.ghost_fs[3 * q + c] = fa[c];
            B.ghost_fn[3 * q + c] = fn[c];
            B.ghost_xf[3 * q + c] = (float)xn[c];
        }
        B.ghost_parent[q] = (int)r;
        B.ghost_id[q] = rl;
        if (B.ghost_sh) B.ghost_sh[q] = kShiftBias;
        B.atom_self[r] = (int)q;
        B.atom_sys[r] = s;
        B.atom_type[r] = B.in_type[d.in_off + a];
        B.atom_orig[r] = (int)(d.in_off + a);
        const int n = d.n_layers;
        for (int c = 0; c < 3; c++) {
            double tl[3], th[3];
            for (int k = 0; k < 3; k++) {
                const bool up = d.hn[3 * c + k] >= 0.0;
                tl[k] = add(fn[k], (double)(up ? -n : n));
                th[k] = add(fn[k], (double)(up ? n : -n));
            }
            const double vl = add(add(mul(d.hn[3 * c], tl[0]), mul(d.hn[3 * c + 1], tl[1])), mul(d.hn[3 * c + 2], tl[2]));
            const double vh = add(add(mul(d.hn[3 * c], th[0]), mul(d.hn[3 * c + 1], th[1])), mul(d.hn[3 * c + 2], th[2]));
            lo[c] = vl < xn[c] ? vl : xn[c];
            hi[c] = vh > xn[c] ? vh : xn[c];
        }
    }
    const int lane = threadIdx.x & 31;
    const int s0 = __shfl_sync(kFull, s, 0);
    if (s0 < 0) return;   // whole warp out of range (valid lanes form a prefix)
    const bool uniform = __all_sync(kFull, !valid || s == s0);
    unsigned long long kmin[3], kmax[3];
    for (int c = 0; c < 3; c++) {
        kmin[c] = valid ? okey(lo[c]) : ~0ull;
        kmax[c] = valid ? okey(hi[c]) : 0ull;
    }
    int mine = valid ? 1 : 0;   // atoms this lane reports
    if (uniform) {
        for (int off = 16; off; off >>= 1)
            for (int c = 0; c < 3; c++) {
                unsigned long long a = __shfl_xor_sync(kFull, kmin[c], off);
                unsigned long long b = __shfl_xor_sync(kFull, kmax[c], off);
                kmin[c] = a < kmin[c] ? a : kmin[c];
                kmax[c] = b > kmax[c] ? b : kmax[c];
            }
        mine = __popc(__ballot_sync(kFull, valid));
        if (lane != 0) mine = 0;
        s = s0;
    }
    if (mine == 0) return;
    for (int c = 0; c < 3; c++) {
        atomicMin(&B.minmax[6 * s + c], kmin[c]);
        atomicMax(&B.minmax[6 * s + 3 + c], kmax[c]);
    }
    // the lane that completes its system sets the system's bin grid
    __threadfence();
    SysDesc& d = B.sys[s];
    if (atomicAdd(&d.done, mine) + mine != d.n_atoms) return;
    __threadfence();
    bin_setup(B, s, d);
}

// --- 2. kept ghost images, one thread per slot -----------------------------
// build_layered_system (:546-585) for both the input-cell system (fractional
// coordinates for the force evaluation) and the reoriented system (Cartesian
// and fractional coordinates for the lists).
// floor((x - min) / search) as the reference computes it, with the correctly
// rounded FP64 quotient: the FP32 quotient decides unless it lies within its
// error (several times the rounding of the coordinates) of an integer.
__device__ __forceinline__ int bin_axis(double x, double mn, double search, float inv) {
    const float xf = (float)x, mf = (float)mn;
    const float q = (xf - mf) * inv, f = floorf(q);
    const float m = 1e-6f + 1e-6f * (fabsf(xf) + fabsf(mf)) * inv;
    if (q - f > m && q - f < 1.0f - m) return (int)f;
    return (int)floor(__ddiv_rn(sub(x, mn), search));
}
__global__ void k_ghosts(BatchView B) {
    chain_begin();
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= B.n_ghost_total) return;
    const int s = find_sys_ghost(B.sys, B.n_sys, q);
    const SysDesc& d = B.sys[s];
    const long long ql = q - d.ghost_off;
    const int rl = (int)(ql / d.gstride), j = (int)(ql % d.gstride);
    const long long r = d.atom_off + rl;
    const long long qs = B.atom_self[r];
    const double fn[3] = {B.ghost_fn[3 * qs], B.ghost_fn[3 * qs + 1], B.ghost_fn[3 * qs + 2]};
    double t[3], xn[3];
    if (q == qs) {   // the atom itself: the rest was written by k_atoms, from the wrapped coordinates
        const double fa[3] = {B.ghost_fs[3 * qs], B.ghost_fs[3 * qs + 1], B.ghost_fs[3 * qs + 2]};
        mv(d.hn, fa[0], fa[1], fa[2], xn);
    } else {
        ShiftBox sb;
        shift_box(d, fn, sb);
        if (j >= sb.count) {
            B.ghost_id[q] = -1;
            B.ghost_bin[q] = -1;
            return;
        }
        const int i0 = sb.lo[0] + j / (sb.cnt[1] * sb.cnt[2]);
        const int i1 = sb.lo[1] + (j / sb.cnt[2]) % sb.cnt[1];
        const int i2 = sb.lo[2] + j % sb.cnt[2];
        // input cell: only the forces' distances use these, so the image's
        // fractional coordinates are the shifted ones themselves (the reference
        // takes them through Cartesian ones and back, which rounds them)
        B.ghost_fs[3 * q] = add(B.ghost_fs[3 * qs], (double)i0);
        B.ghost_fs[3 * q + 1] = add(B.ghost_fs[3 * qs + 1], (double)i1);
        B.ghost_fs[3 * q + 2] = add(B.ghost_fs[3 * qs + 2], (double)i2);
        // reoriented cell: these decide list membership
        double o[3];
        t[0] = add(fn[0], (double)i0); t[1] = add(fn[1], (double)i1); t[2] = add(fn[2], (double)i2);
        mv(d.hn, t[0], t[1], t[2], xn);
        mv(d.hni, xn[0], xn[1], xn[2], o);
        for (int c = 0; c < 3; c++) {
            B.ghost_fn[3 * q + c] = o[c];
            B.ghost_xf[3 * q + c] = (float)xn[c];
        }
        B.ghost_parent[q] = (int)r;
        if (B.ghost_sh) B.ghost_sh[q] = pack_shift(i0, i1, i2);
        B.ghost_id[q] = image_index(i0, i1, i2, d.n_layers, d.side) * d.n_atoms + rl;
    }
    // bin population (:644-678)
    int ib = -1;
    if (!d.err) {
        const float inv = (float)d.inv_search;
        const int bx = bin_axis(xn[0], d.minpos[0], d.search, inv);
        const int by = bin_axis(xn[1], d.minpos[1], d.search, inv);
        const int bz = bin_axis(xn[2], d.minpos[2], d.search, inv);
        const long long total = (long long)d.nb[0] * d.nb[1] * d.nb[2];
        const long long b = bx + (long long)by * d.nb[0] + (long long)bz * d.nb[0] * d.nb[1];
        if (bx < 0 || by < 0 || bz < 0) atomicExch(&B.flags[1], 1);
        else if (b >= total) atomicExch(&B.flags[1], 2);
        else ib = (int)b;
    }
    B.ghost_bin[q] = ib;
    if (ib >= 0) atomicAdd(&B.bin_count[d.bin_off + ib], 1);
}

// Room for every bin's members in bin_items: which bin comes first does not
// matter, so a block scans its bins and reserves their sum.
__global__ void __launch_bounds__(1024) k_bin_alloc(BatchView B) {
    chain_begin();
    __shared__ int wsum[32];
    __shared__ long long base;
    const long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = b < B.n_bins_total ? B.bin_count[b] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, t, o);
            if (lane >= o) t += y;
        }
        wsum[lane] = t;
        if (lane == 31) base = t > 0 ? (long long)atomicAdd((unsigned long long*)&B.totals[3], (unsigned long long)t) : 0;
    }
    __syncthreads();
    if (b < B.n_bins_total) B.bin_start[b] = base + x - v + (w ? wsum[w - 1] : 0);
}

__global__ void k_bin_scatter(BatchView B, const long long* bin_start) {
    chain_begin();
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= B.n_ghost_total) return;
    const int ib = B.ghost_bin[q];
    if (ib < 0) return;
    const int s = find_sys_ghost(B.sys, B.n_sys, q);
    const long long b = B.sys[s].bin_off + ib;
    const long long pos = bin_start[b] + atomicAdd(&B.bin_fill[b], 1);
    B.bin_items[pos] = (int)q;
}

// FP32 coordinates and parent atom of ghost q at bin position pos (read by
// the pair-list kernel in bin order instead of gathered by ghost id)
__device__ __forceinline__ void put_xp(const BatchView& B, long long pos, int q) {
    const float* x = &B.ghost_xf[3 * (long long)q];
    reinterpret_cast<float4*>(B.bin_xp)[pos] = make_float4(x[0], x[1], x[2], __int_as_float(B.ghost_parent[q]));
}

// each bin's members in ascending ghost id (the reference pushes ghosts into
// bins in index order): a warp takes one bin, or 32 in a large batch (most of
// the reserved bins are empty); a bin of one member needs no sort, larger
// ones are ranked by the whole warp in turn: a member's place is the number of members with a
// smaller id (ids are unique), counted over the warp's registers up to 64
// members, over a shared-memory copy of the ids up to kRankSmem; larger
// bins (none in practice) fall back to an insertion sort by one lane
constexpr int kRankSmem = 256;
__device__ __forceinline__ void rank_bin(const BatchView& B, long long s0, int n, int lane, int* key, int* val) {
    int* v = B.bin_items + s0;
    if (n > 64 && n <= kRankSmem) {
        for (int i = lane; i < n; i += 32) {
            val[i] = v[i];
            key[i] = B.ghost_id[val[i]];
        }
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            const int k = key[i];
            int r = 0;
            for (int j = 0; j < n; j++) r += key[j] < k;
            v[r] = val[i];
            if (B.bin_xp) put_xp(B, s0 + r, val[i]);
        }
        __syncwarp();
        return;
    }
    if (n > 64) {
        if (lane == 0)
            for (int i = 1; i < n; i++) {
                const int k2 = v[i], kid = B.ghost_id[k2];
                int j = i - 1;
                while (j >= 0 && B.ghost_id[v[j]] > kid) { v[j + 1] = v[j]; j--; }
                v[j + 1] = k2;
            }
        __syncwarp();
        if (B.bin_xp)
            for (int i = lane; i < n; i += 32) put_xp(B, s0 + i, v[i]);
        __syncwarp();
        return;
    }
    const int big = 0x7fffffff;
    const int q0 = lane < n ? v[lane] : -1, q1 = lane + 32 < n ? v[lane + 32] : -1;
    const int k0 = q0 >= 0 ? B.ghost_id[q0] : big, k1 = q1 >= 0 ? B.ghost_id[q1] : big;
    int r0 = 0, r1 = 0;
    for (int src = 0; src < 32; src++) {
        const int o0 = __shfl_sync(kFull, k0, src), o1 = __shfl_sync(kFull, k1, src);
        r0 += (o0 < k0) + (o1 < k0);
        r1 += (o0 < k1) + (o1 < k1);
    }
    __syncwarp();
    if (q0 >= 0) {
        v[r0] = q0;
        if (B.bin_xp) put_xp(B, s0 + r0, q0);
    }
    if (q1 >= 0) {
        v[r1] = q1;
        if (B.bin_xp) put_xp(B, s0 + r1, q1);
    }
    __syncwarp();
}

__global__ void __launch_bounds__(256) k_bin_rank(BatchView B, const long long* bin_start, int per) {
    chain_begin();
    __shared__ int s_key[8][kRankSmem], s_val[8][kRankSmem];
    const long long b0 = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (b0 >= B.n_bins_total) return;   // whole warp
    const long long b = b0 + lane;
    int n = 0;
    long long st = 0;
    if (lane < per && b < B.n_bins_total) {
        n = B.bin_count[b];
        if (n > 0) st = bin_start[b];
    }
    if (n == 1 && B.bin_xp) put_xp(B, st, B.bin_items[st]);
    unsigned many = __ballot_sync(kFull, n > 1);
    while (many) {
        const int src = __ffs(many) - 1;
        many &= many - 1;
        rank_bin(B, __shfl_sync(kFull, st, src), __shfl_sync(kFull, n, src), lane, s_key[wib], s_val[wib]);
    }
}

// --- 5. 2B neighbour lists (:680-731): one warp per atom --------------------
// Lane b < 27 owns neighbour bin b in the reference's loop order (x bins
// outermost, z innermost); the candidates of all 27 bins are numbered bin by
// bin and the warp walks them 32 at a time, so the emitted order is the
// reference's and short bins leave no lanes idle.  The FP32 distance decides
// membership and the 3-/4-body range bits of nearly every candidate; the exact
// FP64 distance is taken only within the margin of one of the cutoffs (FP64
// distances of all members bound this kernel before: its pipe at 62%).
// One pass: a warp keeps its members in shared memory (up to kL2Hold; an atom
// with more walks its candidates again), the block reserves room for its
// warps' members with one atomic, and the members are written there.
// Measured, 2000 configurations of 8-512 atoms: 402 + 863 us for a counting and
// a filling pass, and 10 us of scans between; 906 in one pass; 465 us without
// the members' FP64 distances.
constexpr int kL2Block = 256;
constexpr int kL2Hold = 96;
struct L2Hold {
    float x[3][kL2Hold];
    int ghost[kL2Hold];
    unsigned w[kL2Hold];
};
// Open-addressing table of the list entries within the 3- or 4-body range, by
// atom and neighbour key; a slot holds an entry's index (B.l2_slots a power of two,
// at least twice those entries).  (Scanning the atom's list instead, by a lane or
// by a warp, made the enumeration of 384 configurations 440-510 us; with the
// table it takes 258, and the insertions 16 us of the list kernel.)  The mixer takes its
// multipliers from SplitMix64 (the golden ratio's 64 bits, and its first finalising
// constant) and, for the atom, the second prime of xxHash64.
__device__ __forceinline__ unsigned entry_hash(const BatchView& B, int r, long long key) {
    unsigned long long x = (unsigned long long)key * 0x9e3779b97f4a7c15ull + (unsigned)r * 0xc2b2ae3d27d4eb4full;
    x ^= x >> 29;
    x *= 0xbf58476d1ce4e5b9ull;
    return (unsigned)(x >> 32) & (unsigned)(B.l2_slots - 1);
}
__device__ __forceinline__ void put_hash(const BatchView& B, int r, long long key, long long e) {
    unsigned h = entry_hash(B, r, key);
    // (never full: bounded all the same)
    for (long long n = 0; n < B.l2_slots; n++, h = (h + 1) & (unsigned)(B.l2_slots - 1))
        if (atomicCAS(&B.l2_hash[h], -1, (int)e) == -1) return;
}

// An entry: x, y, z the FP32 displacement for the enumeration's prefilter; w the
// neighbour's parent atom (int bits; saves the enumeration a dependent load per
// candidate) with the exact tests dist < c3 and dist < c4 in bits 30 and 31, so
// the enumeration compares no FP64 distances.
__device__ __forceinline__ void put_l2(const BatchView& B, int* l2_owner, long long pos, int r, int ghost, float x,
                                       float y, float z, unsigned w) {
    if (pos >= B.n2_cap) return;
    B.l2_ghost[pos] = ghost;
    l2_owner[pos] = r;
    if (B.l2_key) {
        const long long key = (long long)(w & kL2Parent) << 32 | B.ghost_sh[ghost];
        B.l2_key[pos] = key;
        if (w & (kL2In3 | kL2In4)) put_hash(B, r, key, pos);
    }
    reinterpret_cast<float4*>(B.l2_vec)[pos] = make_float4(x, y, z, __uint_as_float(w));
}

__global__ void __launch_bounds__(kL2Block) k_l2(BatchView B, int* l2_owner) {
    chain_begin();
    constexpr int NWARP = kL2Block / 32;
    __shared__ L2Hold hold[NWARP];
    __shared__ int s_cnt[NWARP];
    __shared__ long long s_base;
    const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const bool have = r < B.n_atoms_total;
    const int s = have ? B.atom_sys[r] : 0;
    const SysDesc& d = B.sys[s];
    const long long gi = have ? B.atom_self[r] : 0;
    int count = 0;
    long long base = -1;   // where entries go: < 0 into shared memory
    L2Hold& H = hold[wib];
    auto walk = [&]() {
        const float xi[3] = {B.ghost_xf[3 * gi], B.ghost_xf[3 * gi + 1], B.ghost_xf[3 * gi + 2]};
        const double sd = d.search, c3 = d.c3, c4 = d.c4;
        const float far2 = d.far2, near2 = B.enum_serial ? -1.0f : d.near2;   // (the sequential form reads l2_dist)
        const float c3lo2 = d.c3lo2, c3hi2 = d.c3hi2, c4lo2 = d.c4lo2, c4hi2 = d.c4hi2;
        const bool has3 = d.has3, has4 = d.has4;
        count = 0;
        // the atom's bin, as k_ghosts placed it
        const int ib0 = B.ghost_bin[gi];
        int bx = -1, by = -1, bz = -1;
        if (ib0 >= 0) {
            bx = ib0 % d.nb[0];
            by = (ib0 / d.nb[0]) % d.nb[1];
            bz = ib0 / (d.nb[0] * d.nb[1]);
        }
        if (bx < 1 || by < 1 || bz < 1) {
            if (lane == 0) atomicExch(&B.flags[1], 3);
            return;
        }
        const long long total = (long long)d.nb[0] * d.nb[1] * d.nb[2];
        long long bst = 0;
        int nbin = 0;
        if (lane < 27) {
            const int i = bx - 1 + lane / 9, j = by - 1 + (lane / 3) % 3, k = bz - 1 + lane % 3;
            const long long ib = i + (long long)j * d.nb[0] + (long long)k * d.nb[0] * d.nb[1];
            if (ib >= total) {
                atomicExch(&B.flags[1], 4);
            } else {
                const long long b = d.bin_off + ib;
                bst = B.bin_start[b];
                nbin = B.bin_count[b];
            }
        }
        int incl = nbin;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        const int excl = incl - nbin;
        const int ncand = __shfl_sync(kFull, incl, 31);
        for (int t0 = 0; t0 < ncand; t0 += 32) {
            const int t = t0 + lane;
            // bin of candidate t: the last bin whose first candidate is <= t
            int lo = 0;
            for (int step = 16; step >= 1; step >>= 1) {
                const int cand = lo + step;
                const int ex = __shfl_sync(kFull, excl, cand & 31);
                if (cand < 27 && ex <= t) lo = cand;
            }
            const long long st = __shfl_sync(kFull, bst, lo);
            const int first = __shfl_sync(kFull, excl, lo);
            bool in = false;
            int ajj = -1, par = -1;
            float ex = 0.f, ey = 0.f, ez = 0.f;
            unsigned w = 0;
            double dd = 0.0;
            if (t < ncand) {
                const long long it = st + (t - first);
                ajj = B.bin_items[it];
                float xj[3];
                if (B.bin_xp) {   // the candidate's coordinates and parent stored in bin order
                    const float4 p = reinterpret_cast<const float4*>(B.bin_xp)[it];
                    xj[0] = p.x; xj[1] = p.y; xj[2] = p.z;
                    par = __float_as_int(p.w);
                } else {
                    par = B.ghost_parent[ajj];
                    xj[0] = B.ghost_xf[3 * (long long)ajj];
                    xj[1] = B.ghost_xf[3 * (long long)ajj + 1];
                    xj[2] = B.ghost_xf[3 * (long long)ajj + 2];
                }
                ex = xj[0] - xi[0]; ey = xj[1] - xi[1]; ez = xj[2] - xi[2];
                const float e2 = ex * ex + ey * ey + ez * ez;
                in = ajj != gi && r <= par && e2 < far2;   // else certainly >= sd
                if (in) {
                    bool in3 = has3 && e2 < c3lo2, in4 = has4 && e2 < c4lo2;
                    if (!(e2 < near2) || (has3 && !in3 && !(e2 >= c3hi2)) || (has4 && !in4 && !(e2 >= c4hi2))) {
                        dd = dist_frac(d.hn, &B.ghost_fn[3 * gi], &B.ghost_fn[3 * (long long)ajj]);
                        in = dd < sd;
                        in3 = dd < c3;   // (c3, c4 are 0 for an absent order)
                        in4 = dd < c4;
                    }
                    w = (unsigned)par | (in3 ? kL2In3 : 0u) | (in4 ? kL2In4 : 0u);
                }
            }
            const unsigned m = __ballot_sync(kFull, in);
            if (in) {
                const int k = count + __popc(m & lt);
                if (base >= 0) {
                    put_l2(B, l2_owner, base + k, (int)r, ajj, ex, ey, ez, w);
                    if (B.enum_serial && base + k < B.n2_cap) B.l2_dist[base + k] = dd;
                } else if (k < kL2Hold) {
                    H.x[0][k] = ex;
                    H.x[1][k] = ey;
                    H.x[2][k] = ez;
                    H.ghost[k] = ajj;
                    H.w[k] = w;
                }
            }
            count += __popc(m);
        }
    };
    if (have && !d.err) walk();
    if (lane == 0) s_cnt[wib] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
        for (int k = 0; k < NWARP; k++) sum += s_cnt[k];
        s_base = sum > 0 ? (long long)atomicAdd((unsigned long long*)&B.totals[0], (unsigned long long)sum) : 0;
    }
    __syncthreads();
    if (!have) return;
    long long at = s_base;
    for (int k = 0; k < wib; k++) at += s_cnt[k];
    if (lane == 0) {
        B.l2_off[r] = at;
        B.l2_count[r] = count;
    }
    if (count > kL2Hold || B.enum_serial) {
        base = at;
        walk();
        return;
    }
    __syncwarp();
    for (int k = lane; k < count; k += 32)
        put_l2(B, l2_owner, at + k, (int)r, H.ghost[k], H.x[0][k], H.x[1][k], H.x[2][k], H.w[k]);
}

// Exact test "distance >= c" for a ghost pair of one atom's list, deciding
// from the FP32 displacement difference when it is farther than eps from c.
struct PairDist {
    const double* hn;
    const double* fa;
    const double* fb;
    float df;
    double exact;
    bool have;
    __device__ bool ge(double c, double eps) {
        if ((double)df < c - eps) return false;
        if ((double)df >= c + eps) return true;
        if (!have) { exact = dist_frac(hn, fa, fb); have = true; }
        return exact >= c;
    }
};

// The same test with the margins as FP32 thresholds (lo <= c - eps, hi >=
// c + eps, rounded outward), so the decided cases take no FP64 instruction.
struct PairDistF {
    const double* hn;
    const double* fa;
    const double* fb;
    float df;
    __device__ bool ge(double c, float lo, float hi) const {
        if (df < lo) return false;
        if (df >= hi) return true;
        return dist_frac(hn, fa, fb) >= c;
    }
};

__device__ __forceinline__ float vdist(const float4& a, const float4& b) {
    const float x = b.x - a.x, y = b.y - a.y, z = b.z - a.z;
    return sqrtf(x * x + y * y + z * z);
}

// --- 6. 3B/4B enumeration (:735-855): one thread per (i, j) list entry -----
// The valid_3mer / valid_4mer flags carry over between k iterations exactly as
// in the reference, so the emitted sets and their order match it.
template <bool FILL>
__device__ void enum_entry(const BatchView& B, const int* l2_owner, long long e) {
    const int r = l2_owner[e];
    const SysDesc& d = B.sys[B.atom_sys[r]];
    int n3 = 0, n4 = 0;
    long long o3 = 0, o4 = 0;
    if (FILL) { o3 = B.e_off3[e]; o4 = B.e_off4[e]; }
    const double c3 = d.c3, c4 = d.c4, eps = d.eps;
    if (d.has3 || d.has4) {
        double hn[9];
        for (int c = 0; c < 9; c++) hn[c] = d.hn[c];
        const int gi = B.atom_self[r];
        long long b0, b1;
        list_range(B, r, b0, b1);
        const float4* vec = reinterpret_cast<const float4*>(B.l2_vec);
        const int jj = B.l2_ghost[e];
        const double dij = B.l2_dist[e];
        bool v3 = true, v4 = true;
        if (dij >= c3) v3 = false;
        if (dij >= c4) v4 = false;
        if (v3 || v4) {
            const double* fj = &B.ghost_fn[3 * (long long)jj];
            const float4 vj = vec[e];
            const int pj = B.ghost_parent[jj];
            for (long long k = b0; k < b1; k++) {
                const int kk = B.l2_ghost[k];
                if (jj == kk) continue;
                const int pk = B.ghost_parent[kk];
                if (pj > pk) continue;
                const double dik = B.l2_dist[k];
                if (dik >= c3) v3 = false;
                if (dik >= c4) v4 = false;
                const float4 vk = vec[k];
                const double* fk = &B.ghost_fn[3 * (long long)kk];
                PairDist jk{hn, fj, fk, vdist(vj, vk), 0.0, false};
                if (jk.ge(c3, eps)) v3 = false;
                if (jk.ge(c4, eps)) v4 = false;
                if (!v3 && !v4) {
                    if (dij < c3) v3 = true;
                    if (dij < c4) v4 = true;
                    continue;
                }
                if (v3) {
                    if (FILL && o3 + n3 < B.n3_cap) {
                        int* out = B.c3 + 3 * (o3 + n3);
                        out[0] = gi; out[1] = jj; out[2] = kk;
                    }
                    n3++;
                }
                if (!d.has4) continue;
                if (!v4) {
                    if (dij < c4) v4 = true;
                    continue;
                }
                for (long long l = b0; l < b1; l++) {
                    const int ll = B.l2_ghost[l];
                    if (jj == ll || kk == ll) continue;
                    const int pl = B.ghost_parent[ll];
                    if (pj > pl) continue;
                    if (pk > pl) continue;
                    if (B.l2_dist[l] >= c4) continue;
                    const float4 vl = vec[l];
                    const double* fl = &B.ghost_fn[3 * (long long)ll];
                    PairDist jl{hn, fj, fl, vdist(vj, vl), 0.0, false};
                    if (jl.ge(c4, eps)) continue;
                    PairDist kl{hn, fk, fl, vdist(vk, vl), 0.0, false};
                    if (kl.ge(c4, eps)) continue;
                    if (v4) {
                        if (FILL && o4 + n4 < B.n4_cap) {
                            int* out = B.c4 + 4 * (o4 + n4);
                            out[0] = gi; out[1] = jj; out[2] = kk; out[3] = ll;
                        }
                        n4++;
                    }
                }
            }
        }
    }
    if (!FILL) { B.e_cnt3[e] = n3; B.e_cnt4[e] = n4; }
}

template <bool FILL>
__global__ void k_enum(BatchView B, const int* l2_owner) {
    const long long n2 = list_total(B);
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < B.n2_cap;
         e += (long long)gridDim.x * blockDim.x) {
        if (e >= n2) {
            if (!FILL) { B.e_cnt3[e] = 0; B.e_cnt4[e] = 0; }
            continue;
        }
        enum_entry<FILL>(B, l2_owner, e);
    }
}

// List entry of the pair (j, k) of two images in one atom's list: the entry of
// j's parent whose neighbour is k's parent at the shift of k relative to j
// (w_j, w_k: their l2_vec.w; sh: packed shifts).  The list of the parent holds
// every pair below the search radius whose parents are in this order, so only a
// pair within rounding of a cutoff can be missing: -1.
__device__ __forceinline__ int find_entry(const BatchView& B, const int* l2_owner, unsigned w_j, int sh_j, unsigned w_k,
                                          int sh_k) {
    const int pj = (int)(w_j & kL2Parent);
    const long long want = (long long)(w_k & kL2Parent) << 32 | (unsigned)(sh_k - sh_j + kShiftBias);
    unsigned h = entry_hash(B, pj, want);
    for (long long n = 0; n < B.l2_slots; n++, h = (h + 1) & (unsigned)(B.l2_slots - 1)) {
        const int e = B.l2_hash[h];
        if (e < 0) return -1;
        if (B.l2_key[e] == want && l2_owner[e] == pj) return e;
    }
    return -1;
}

// The list entries of a cluster's pairs (entries e[0..n) of the first atom):
// those of the first atom alone, or all of them (all_pairs).
template <int N>
__device__ __forceinline__ void put_entries(const BatchView& B, const int* l2_owner, long long q, const int* e,
                                            const unsigned* w, const int* sh) {
    int* out = N == 2 ? B.c3e : B.c4e;
    if (!out) return;
    constexpr int ALL = N * (N + 1) / 2;
    out += (B.all_pairs ? ALL : N) * q;
#pragma unroll
    for (int k = 0; k < N; k++) out[k] = e[k];
    if (!B.all_pairs) return;
    int n = N;
#pragma unroll
    for (int a = 0; a < N; a++)
#pragma unroll
        for (int b = a + 1; b < N; b++) out[n++] = find_entry(B, l2_owner, w[a], sh[a], w[b], sh[b]);
}
__device__ __forceinline__ void put_entries_of(const BatchView& B, const int* l2_owner, long long q, int n, long long a,
                                               long long b, long long c) {
    const long long at[3] = {a, b, c};
    int e[3], sh[3] = {0, 0, 0};
    unsigned w[3];
    for (int k = 0; k < n; k++) {
        e[k] = (int)at[k];
        w[k] = reinterpret_cast<const unsigned*>(B.l2_vec)[4 * at[k] + 3];
        if (B.all_pairs) sh[k] = (int)B.l2_key[at[k]];
    }
    if (n == 2) put_entries<2>(B, l2_owner, q, e, w, sh);
    else put_entries<3>(B, l2_owner, q, e, w, sh);
}

// Per-entry warp form of the same enumeration.  When the 4-body outer cutoff
// does not exceed the 3-body one (or a system lacks one of the two), the
// valid_3mer / valid_4mer flags are restored before every k (the reference's
// reset branch), so each k -- and each l -- is decided on its own: lanes take
// consecutive k (then l) of the atom's list and a ballot plus prefix count
// emits the clusters in the reference's (k, l) order.  Systems with 3- and
// 4-body terms and rc4 > rc3 keep the sequential carry-over (k_enum).  Used
// by k_enuma for atoms whose list is longer than its bit matrices hold.
template <bool FILL>
__device__ void enumw_entry(const BatchView& B, const int* l2_owner, long long e, int r, const SysDesc& d, int lane, unsigned lt,
                            long long at3 = 0, long long at4 = 0) {
    const float4* vec = reinterpret_cast<const float4*>(B.l2_vec);
    const double c3 = d.c3, c4 = d.c4;
    const float4 vj = vec[e];
    const unsigned wj = __float_as_uint(vj.w);
    const bool want3 = d.has3 && (wj & kL2In3), want4 = d.has4 && (wj & kL2In4);
    long long n3 = 0, n4 = 0;
    long long o3 = 0, o4 = 0;
    if (FILL) { o3 = at3 + B.e_off3[e]; o4 = at4 + B.e_off4[e]; }
    if (want3 || want4) {
        const double* hn = d.hn;   // read in place: the exact distances are rare
        const float c3lo = d.c3lo, c3hi = d.c3hi, c4lo = d.c4lo, c4hi = d.c4hi;
        const int gi = B.atom_self[r];
        long long b0, b1;
        list_range(B, r, b0, b1);
        const int jj = B.l2_ghost[e];
        const double* fj = &B.ghost_fn[3 * (long long)jj];
        const int pj = (int)(wj & kL2Parent);
        for (long long kb = b0; kb < b1; kb += 32) {
            const long long k = kb + lane;
            bool ok3 = false, ok4 = false;
            int kk = -1, pk = 0;
            float4 vk = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < b1) {
                kk = B.l2_ghost[k];
                vk = vec[k];
                const unsigned wk = __float_as_uint(vk.w);
                pk = (int)(wk & kL2Parent);
                if (kk != jj && pj <= pk) {
                    const PairDistF jk{hn, fj, &B.ghost_fn[3 * (long long)kk], vdist(vj, vk)};
                    ok3 = want3 && (wk & kL2In3) && !jk.ge(c3, c3lo, c3hi);
                    ok4 = want4 && (wk & kL2In4) && !jk.ge(c4, c4lo, c4hi);
                }
            }
            const unsigned m3 = __ballot_sync(kFull, ok3);
            if (FILL && ok3) {
                const long long q = o3 + n3 + __popc(m3 & lt);
                if (q < B.n3_cap) {
                    int* out = B.c3 + 3 * q;
                    out[0] = gi; out[1] = jj; out[2] = kk;
                    put_entries_of(B, l2_owner, q, 2, e, k, 0);
                }
            }
            n3 += __popc(m3);
            unsigned m4 = __ballot_sync(kFull, ok4);
            while (m4) {
                const int src = __ffs(m4) - 1;
                m4 &= m4 - 1;
                const int ks = __shfl_sync(kFull, kk, src);
                const int pks = __shfl_sync(kFull, pk, src);
                float4 vks;
                vks.x = __shfl_sync(kFull, vk.x, src);
                vks.y = __shfl_sync(kFull, vk.y, src);
                vks.z = __shfl_sync(kFull, vk.z, src);
                vks.w = 0.f;
                const double* fk = &B.ghost_fn[3 * (long long)ks];
                for (long long lb = b0; lb < b1; lb += 32) {
                    const long long l = lb + lane;
                    bool okl = false;
                    int ll = -1;
                    if (l < b1) {
                        ll = B.l2_ghost[l];
                        const float4 vl = vec[l];
                        if (ll != jj && ll != ks) {
                            const unsigned wl = __float_as_uint(vl.w);
                            const int pl = (int)(wl & kL2Parent);
                            if (pj <= pl && pks <= pl && (wl & kL2In4)) {
                                const double* fl = &B.ghost_fn[3 * (long long)ll];
                                const PairDistF jl{hn, fj, fl, vdist(vj, vl)};
                                if (!jl.ge(c4, c4lo, c4hi)) {
                                    const PairDistF kl{hn, fk, fl, vdist(vks, vl)};
                                    okl = !kl.ge(c4, c4lo, c4hi);
                                }
                            }
                        }
                    }
                    const unsigned ml = __ballot_sync(kFull, okl);
                    if (FILL && okl) {
                        const long long q = o4 + n4 + __popc(ml & lt);
                        if (q < B.n4_cap) {
                            int* out = B.c4 + 4 * q;
                            out[0] = gi; out[1] = jj; out[2] = ks; out[3] = ll;
                            put_entries_of(B, l2_owner, q, 3, e, kb + src, l);
                        }
                    }
                    n4 += __popc(ml);
                }
            }
        }
    }
    if (!FILL && lane == 0) { B.e_cnt3[e] = (int)n3; B.e_cnt4[e] = (int)n4; }
}

// Bit-matrix form (G warps per atom i, atoms with at most kEnumRows list
// entries within the 3- or 4-body range; the others of the list start and join
// no cluster).  With the reset semantics above, membership depends only on pair
// tests among the entries of i's list:
//   T[j][k] = want3(j) && in3(k) && j != k && parent(j) <= parent(k) && |r_jk| < rc3
//   Q[j][k] = want4(j) && in4(k) && j != k && parent(j) <= parent(k) && |r_jk| < rc4
// (i, j, k) is a triplet iff T[j][k]; (i, j, k, l) a quadruplet iff Q[j][k]
// && Q[j][l] && Q[k][l] (Q[j][k] implies want4(k), which Q[k][l] carries).
// The warps test every ordered pair of entries once -- the FP32 distance with
// the same thresholds and, inside the margin, the same exact FP64 distance as
// the per-entry form -- and keep the rows T[j], Q[j] as bit masks in shared
// memory.  The masks give the counts, n3(j) = popc T[j] and n4(j) = sum over k in
// Q[j] of popc(Q[j] & Q[k]), room for the atom's clusters is reserved with one
// atomic per body order, and the clusters are emitted from the masks in the
// same order (k ascending, then l ascending), each entry's after the counts of
// the entries before it.  One pass over the atoms: two passes with a scan over
// the entries between them tested every pair twice (2000 configurations: 625 +
// 860 us and about 180 us of scans; 875 us in one pass, 930 with the bucket
// keys, 633 since each atom's list is compacted to its entries in range).
// G = 1 for batches with many atoms; small ones spread an atom over
// up to a whole block so that the launch still fills the GPU.
constexpr int kEnumRows = 96;
constexpr int kEnumWords = kEnumRows / 32;   // odd: column reads of the masks hit distinct banks
constexpr int kEnumWarps = 8;

template <int G>
__device__ __forceinline__ void group_sync(int grp) {
    if (G == 1) __syncwarp();
    else if (G == kEnumWarps) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(32 * G) : "memory");
}

// position of the k-th (from 0) set bit of m
__device__ __forceinline__ int select_bit(unsigned m, int k) {
    int pos = 0;
    for (int sh = 16; sh; sh >>= 1) {
        const int c = __popc(m & ((1u << sh) - 1u));
        if (k >= c) { k -= c; m >>= sh; pos += sh; }
    }
    return pos;
}

// n3 and n4 of entry a from the masks
__device__ __forceinline__ void mask_counts(const unsigned* rt, const unsigned* rq, int a, int nw, int& n3, int& n4) {
    n3 = 0;
    n4 = 0;
    for (int c = 0; c < nw; c++) n3 += __popc(rt[a * kEnumWords + c]);
    for (int c = 0; c < nw; c++) {
        unsigned m = rq[a * kEnumWords + c];
        while (m) {
            const int b = 32 * c + __ffs(m) - 1;
            m &= m - 1;
            for (int c2 = 0; c2 < nw; c2++) n4 += __popc(rq[a * kEnumWords + c2] & rq[b * kEnumWords + c2]);
        }
    }
}

// Bucket key of a cluster from its atoms' types, counted in the block's
// histogram (kBkSmem buckets) or, with more buckets, in B.bk_count.  Called by
// whole warps; on: the lane has a cluster.
__device__ __forceinline__ void count_key(const BatchView& B, int* hist, int at, int key) {
    const unsigned peers = __match_any_sync(kFull, key);
    if (key >= 0 && (threadIdx.x & 31) == __ffs(peers) - 1) {
        if (hist) atomicAdd(&hist[at + key], __popc(peers));
        else atomicAdd(&B.bk_count[at + key], __popc(peers));
    }
}

template <int G>
__global__ void __launch_bounds__(32 * kEnumWarps, 4) k_enuma(BatchView B, const int* l2_owner) {
    chain_begin();
    constexpr int NG = kEnumWarps / G;   // atoms a block works on at a time
    __shared__ float4 s_v[NG][kEnumRows];
    __shared__ int s_g[NG][kEnumRows];
    __shared__ unsigned s_t[NG][kEnumRows * kEnumWords];
    __shared__ unsigned s_q[NG][kEnumRows * kEnumWords];
    __shared__ int s_o[NG][2 * kEnumRows + 2];   // per-entry offsets, then the totals
    __shared__ long long s_at[NG][2];            // where the atom's clusters go
    __shared__ unsigned char s_ty[NG][kEnumRows];   // the entries' types
    __shared__ int s_e[NG][kEnumRows];              // their numbers in the atom's list
    __shared__ int s_sh[NG][kEnumRows];             // their image shifts
    extern __shared__ int s_hist[];              // bucket counts of this block (when B.keyed and few buckets)
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int grp = wib / G, w = wib % G;
    const int nbk = B.keyed ? B.nbk3 + B.nbk4 : 0;
    int* hist = nbk > 0 && nbk <= kBkSmem ? s_hist : nullptr;
    if (hist) {
        for (int k = threadIdx.x; k < nbk; k += blockDim.x) hist[k] = 0;
        __syncthreads();
    }
    const unsigned lt = (1u << lane) - 1u;
    const float4* vec = reinterpret_cast<const float4*>(B.l2_vec);
    float4* sv = s_v[grp];
    int* sg = s_g[grp];
    unsigned* rt = s_t[grp];
    unsigned* rq = s_q[grp];
    int* so = s_o[grp];
    int* se = s_e[grp];
    // room for an atom's t3 triplets and t4 quadruplets (one lane of the group)
    auto reserve = [&](long long r, long long t3, long long t4) {
        const long long a3 = t3 > 0 ? (long long)atomicAdd((unsigned long long*)&B.totals[1], (unsigned long long)t3) : 0;
        const long long a4 = t4 > 0 ? (long long)atomicAdd((unsigned long long*)&B.totals[2], (unsigned long long)t4) : 0;
        B.a_off[2 * r] = s_at[grp][0] = a3;
        B.a_off[2 * r + 1] = s_at[grp][1] = a4;
        B.a_cnt[2 * r] = (int)t3;
        B.a_cnt[2 * r + 1] = (int)t4;
    };
    const long long ngroups = (long long)gridDim.x * NG;
    for (long long r = (long long)blockIdx.x * NG + grp; r < B.n_atoms_total; r += ngroups) {
        long long b0, b1;
        list_range(B, r, b0, b1);
        const SysDesc& d = B.sys[B.atom_sys[r]];
        // the entries within the 3- or 4-body range, in order (about half of the list)
        int L = 0;
        if (d.has3 || d.has4) {
            group_sync<G>(grp);   // the previous atom's masks and offsets are no longer read
            for (long long e0 = b0; e0 < b1; e0 += 32) {   // (every warp of the group counts; the first one keeps)
                const long long e = e0 + lane;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (e < b1) v = vec[e];
                const bool in = e < b1 && (__float_as_uint(v.w) & (kL2In3 | kL2In4));
                const unsigned m = __ballot_sync(kFull, in);
                const int k = L + __popc(m & lt);
                if (in && w == 0 && k < kEnumRows) {
                    sv[k] = v;
                    se[k] = (int)(e - b0);
                    sg[k] = B.l2_ghost[e];
                    s_ty[grp][k] = (unsigned char)B.atom_type[__float_as_uint(v.w) & kL2Parent];
                    if (B.all_pairs) s_sh[grp][k] = (int)B.l2_key[e];
                }
                L += __popc(m);
            }
        }
        if (L <= 0) {
            if (w == 0 && lane == 0) {
                B.a_off[2 * r] = B.a_off[2 * r + 1] = 0;
                B.a_cnt[2 * r] = B.a_cnt[2 * r + 1] = 0;
            }
            continue;
        }
        if (L > kEnumRows) {
            // counts per entry, their offsets, then the clusters
            for (long long e = b0 + w; e < b1; e += G) enumw_entry<false>(B, l2_owner, e, (int)r, d, lane, lt);
            __threadfence_block();
            group_sync<G>(grp);
            if (w == 0) {
                long long c3 = 0, c4 = 0;
                for (long long e0 = b0; e0 < b1; e0 += 32) {
                    const long long e = e0 + lane;
                    const int n3 = e < b1 ? B.e_cnt3[e] : 0, n4 = e < b1 ? B.e_cnt4[e] : 0;
                    int i3 = n3, i4 = n4;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y3 = __shfl_up_sync(kFull, i3, o), y4 = __shfl_up_sync(kFull, i4, o);
                        if (lane >= o) { i3 += y3; i4 += y4; }
                    }
                    if (e < b1) { B.e_off3[e] = c3 + i3 - n3; B.e_off4[e] = c4 + i4 - n4; }
                    c3 += __shfl_sync(kFull, i3, 31);
                    c4 += __shfl_sync(kFull, i4, 31);
                }
                if (lane == 0) reserve(r, c3, c4);
            }
            __threadfence_block();
            group_sync<G>(grp);
            for (long long e = b0 + w; e < b1; e += G)
                enumw_entry<true>(B, l2_owner, e, (int)r, d, lane, lt, s_at[grp][0], s_at[grp][1]);
            if (nbk > 0) {
                // their keys, from the clusters as written
                __threadfence_block();
                group_sync<G>(grp);
                const DevParamSet& P = B.psets[d.pset];
                auto type = [&](int g) { return B.atom_type[B.ghost_parent[g]]; };
                for (int nb = 3; nb <= 4; nb++) {
                    const long long at = s_at[grp][nb - 3], n = B.a_cnt[2 * r + nb - 3], cap = nb == 3 ? B.n3_cap : B.n4_cap;
                    const int* cl = nb == 3 ? B.c3 : B.c4;
                    for (long long t0 = 32 * w; t0 < n; t0 += 32 * G) {
                        const long long q = at + t0 + lane;
                        int key = -1;
                        if (t0 + lane < n && q < cap) {
                            int u = 0;
                            for (int k = 0; k < nb; k++) u = u * P.ntypes + type(cl[nb * q + k]);
                            key = (nb == 3 ? P.key3 : P.key4)[u];
                            if (key >= 0) key += nb == 3 ? P.bk3 : P.bk4;
                            (nb == 3 ? B.bk_key3 : B.bk_key4)[q] = key;
                        }
                        count_key(B, hist, nb == 3 ? 0 : B.nbk3, key);
                    }
                }
            }
            continue;
        }
        group_sync<G>(grp);
        const int nw = (L + 31) >> 5;
        {
            const double* hn = d.hn;   // read in place: the exact distances are rare
            const double c3 = d.c3, c4 = d.c4;
            // squared FP32 thresholds: the prefilter needs no square root
            const float c3lo2 = d.c3lo2, c3hi2 = d.c3hi2, c4lo2 = d.c4lo2, c4hi2 = d.c4hi2;
            const bool has3 = d.has3, has4 = d.has4;
            for (int c = 0; c < nw; c++) {
                // this lane's candidate k (column b of every row) stays in registers
                const int b = 32 * c + lane;
                float4 vb = make_float4(0.f, 0.f, 0.f, 0.f);
                int gb = -1;
                if (b < L) { vb = sv[b]; gb = sg[b]; }
                const unsigned wb = __float_as_uint(vb.w);
                const int pb = (int)(wb & kL2Parent);
                const bool in3 = has3 && (wb & kL2In3), in4 = has4 && (wb & kL2In4);
                for (int a = w; a < L; a += G) {
                    const float4 va = sv[a];
                    const unsigned wa = __float_as_uint(va.w);
                    const int ga = sg[a];
                    const bool t0 = in3 && (wa & kL2In3) && b < L && gb != ga && (int)(wa & kL2Parent) <= pb;
                    const bool q0 = in4 && (wa & kL2In4) && b < L && gb != ga && (int)(wa & kL2Parent) <= pb;
                    bool t = false, q = false;
                    if (t0 || q0) {
                        const float ex = vb.x - va.x, ey = vb.y - va.y, ez = vb.z - va.z;
                        const float e2 = ex * ex + ey * ey + ez * ez;
                        // inside the margin of a cutoff: decided by the exact distance
                        // (FP64 only on that rare branch: GB300 issues FP64 at a small
                        // fraction of the FP32 rate)
                        const bool x3 = t0 && !(e2 < c3lo2) && !(e2 >= c3hi2);
                        const bool x4 = q0 && !(e2 < c4lo2) && !(e2 >= c4hi2);
                        t = t0 && e2 < c3lo2;
                        q = q0 && e2 < c4lo2;
                        if (x3 || x4) {
                            const double dx = dist_frac(hn, &B.ghost_fn[3 * (long long)ga], &B.ghost_fn[3 * (long long)gb]);
                            if (x3) t = dx < c3;
                            if (x4) q = dx < c4;
                        }
                    }
                    const unsigned bt = __ballot_sync(kFull, t), bq = __ballot_sync(kFull, q);
                    if (lane == 0) { rt[a * kEnumWords + c] = bt; rq[a * kEnumWords + c] = bq; }
                }
            }
        }
        group_sync<G>(grp);
        // offsets of the entries within the atom (triplets, quadruplets) and
        // room for the atom's totals
        if (w == 0) {
            int c3 = 0, c4 = 0;
            for (int a0 = 0; a0 < L; a0 += 32) {
                const int a = a0 + lane;
                int n3 = 0, n4 = 0;
                if (a < L) mask_counts(rt, rq, a, nw, n3, n4);
                int i3 = n3, i4 = n4;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y3 = __shfl_up_sync(kFull, i3, o), y4 = __shfl_up_sync(kFull, i4, o);
                    if (lane >= o) { i3 += y3; i4 += y4; }
                }
                if (a < L) { so[2 * a] = c3 + i3 - n3; so[2 * a + 1] = c4 + i4 - n4; }
                c3 += __shfl_sync(kFull, i3, 31);
                c4 += __shfl_sync(kFull, i4, 31);
            }
            if (lane == 0) {
                so[2 * L] = c3;
                so[2 * L + 1] = c4;
                reserve(r, c3, c4);
            }
        }
        group_sync<G>(grp);
        // the atom's clusters in the reference's order, one per lane: the t-th
        // triplet belongs to the last entry whose offset is <= t and is that
        // entry's (t - offset)-th set bit of T; the t-th quadruplet likewise,
        // walking the entry's k in Q and the set bits of Q[j] & Q[k]
        const int gi = B.atom_self[r];
        const long long base3 = s_at[grp][0], base4 = s_at[grp][1];
        const int t3 = so[2 * L], t4 = so[2 * L + 1];
        const DevParamSet& P = B.psets[d.pset];
        const int nt = P.ntypes, ti = B.atom_type[r];
        for (int t0 = 32 * w; t0 < t3; t0 += 32 * G) {
            const int t = t0 + lane;
            int key = -1;
            if (t < t3) {
                int lo = 0, hi = L - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (so[2 * mid] <= t) lo = mid; else hi = mid - 1;
                }
                const int a = lo;
                int rk = t - so[2 * a], bk = 0;
                for (int c = 0; c < nw; c++) {
                    const unsigned m = rt[a * kEnumWords + c];
                    const int pc = __popc(m);
                    if (rk < pc) { bk = 32 * c + select_bit(m, rk); break; }
                    rk -= pc;
                }
                const long long q = base3 + t;
                if (q < B.n3_cap) {
                    int* out = B.c3 + 3 * q;
                    out[0] = gi; out[1] = sg[a]; out[2] = sg[bk];
                    if (B.c3e) {
                        const int e[2] = {(int)b0 + se[a], (int)b0 + se[bk]};
                        const unsigned wv[2] = {__float_as_uint(sv[a].w), __float_as_uint(sv[bk].w)};
                        const int sh[2] = {s_sh[grp][a], s_sh[grp][bk]};
                        put_entries<2>(B, l2_owner, q, e, wv, sh);
                    }
                    if (nbk > 0) {
                        key = P.key3[(ti * nt + s_ty[grp][a]) * nt + s_ty[grp][bk]];
                        if (key >= 0) key += P.bk3;
                        B.bk_key3[q] = key;
                    }
                }
            }
            if (nbk > 0) count_key(B, hist, 0, key);
        }
        for (int t0 = 32 * w; t0 < t4; t0 += 32 * G) {
            const int t = t0 + lane;
            int key = -1;
            if (t < t4) {
                int lo = 0, hi = L - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (so[2 * mid + 1] <= t) lo = mid; else hi = mid - 1;
                }
                const int a = lo;
                int rk = t - so[2 * a + 1], bk = 0, lk = 0;
                bool found = false;
                for (int c = 0; c < nw && !found; c++) {
                    unsigned mb = rq[a * kEnumWords + c];
                    while (mb && !found) {
                        const int bb = 32 * c + __ffs(mb) - 1;
                        mb &= mb - 1;
                        for (int c2 = 0; c2 < nw; c2++) {
                            const unsigned x = rq[a * kEnumWords + c2] & rq[bb * kEnumWords + c2];
                            const int pc = __popc(x);
                            if (rk < pc) { bk = bb; lk = 32 * c2 + select_bit(x, rk); found = true; break; }
                            rk -= pc;
                        }
                    }
                }
                const long long q = base4 + t;
                if (q < B.n4_cap) {
                    int* out = B.c4 + 4 * q;
                    out[0] = gi; out[1] = sg[a]; out[2] = sg[bk]; out[3] = sg[lk];
                    if (B.c4e) {
                        const int e[3] = {(int)b0 + se[a], (int)b0 + se[bk], (int)b0 + se[lk]};
                        const unsigned wv[3] = {__float_as_uint(sv[a].w), __float_as_uint(sv[bk].w),
                                                __float_as_uint(sv[lk].w)};
                        const int sh[3] = {s_sh[grp][a], s_sh[grp][bk], s_sh[grp][lk]};
                        put_entries<3>(B, l2_owner, q, e, wv, sh);
                    }
                    if (nbk > 0) {
                        key = P.key4[((ti * nt + s_ty[grp][a]) * nt + s_ty[grp][bk]) * nt + s_ty[grp][lk]];
                        if (key >= 0) key += P.bk4;
                        B.bk_key4[q] = key;
                    }
                }
            }
            if (nbk > 0) count_key(B, hist, B.nbk3, key);
        }
    }
    if (hist) {
        __syncthreads();
        for (int k = threadIdx.x; k < nbk; k += blockDim.x)
            if (hist[k]) atomicAdd(&B.bk_count[k], hist[k]);
    }
}

template <int G>
void launch_enuma(const BatchView& B, const int* l2_owner, cudaStream_t st) {
    constexpr int NG = kEnumWarps / G;
    const long long want = (long long)sm_count() * 4;   // 4 blocks of 8 warps per SM
    const long long need = (B.n_atoms_total + NG - 1) / NG;
    const unsigned grid = (unsigned)(want < need ? want : need);
    const int nbk = B.keyed ? B.nbk3 + B.nbk4 : 0;
    const size_t smem = nbk <= kBkSmem ? sizeof(int) * (size_t)nbk : 0;
    // (with one warp per atom the static arrays take 45.9 KB: more than 528 buckets pass
    // the 48 KB that a block gets without asking)
    if (smem > 0)
        cudaFuncSetAttribute((const void*)k_enuma<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(int) * kBkSmem);
    count_launch(), launch_chained(k_enuma<G>, grid, 32 * kEnumWarps, smem, st, B, l2_owner);
}

// --- reset of accumulators, counters and bins -------------------------------
__global__ void k_reset(BatchView B) {
    chain_begin();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < B.n_bins_total; i += stride) {
        B.bin_count[i] = 0;
        B.bin_fill[i] = 0;
    }
    for (long long i = t; i < 3 * B.n_in_total; i += stride) B.force[i] = 0.0;
    for (long long i = t; i < 8LL * B.n_sys; i += stride) {
        B.ev[i] = 0.0;
        if (i < 6LL * B.n_sys) B.minmax[i] = (i % 6) < 3 ? ~0ull : 0ull;
        if (i < B.n_sys) {
            B.sys[i].err = 0;
            B.sys[i].done = 0;
        }
    }
    if (B.bk_count)
        for (long long i = t; i < B.nbk3 + B.nbk4; i += stride) {
            B.bk_count[i] = 0;
            B.bk_fill[i] = 0;
        }
    if (B.l2_hash)
        for (long long i = t; i < B.l2_slots / 4; i += stride) reinterpret_cast<int4*>(B.l2_hash)[i] = make_int4(-1, -1, -1, -1);
    if (t < 8) B.flags[t] = 0;
    if (t < 2) B.queue[t] = 0ull;
    if (t < 4 && B.totals) B.totals[t] = 0;
}

// --- exclusive scan (three phases, recursive on block sums) -----------------
constexpr int kScanBlock = 1024;

__global__ void k_scan_block(const int* in, const long long* in64, long long* out, long long n, long long* sums) {
    __shared__ long long wsum[32];
    const long long i = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    long long v = 0;
    if (i < n) v = in ? (long long)in[i] : in64[i];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long x = v;
    for (int off = 1; off < 32; off <<= 1) {
        long long y = __shfl_up_sync(kFull, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        long long t = wsum[lane];
        for (int off = 1; off < 32; off <<= 1) {
            long long y = __shfl_up_sync(kFull, t, off);
            if (lane >= off) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    const long long incl = x + (w ? wsum[w - 1] : 0);
    if (i < n) out[i] = incl - v;
    if (threadIdx.x == kScanBlock - 1) sums[blockIdx.x] = incl;
}

__global__ void k_scan_add(long long* out, long long n, const long long* offs) {
    const long long i = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    if (i < n) out[i] += offs[blockIdx.x];
}

__global__ void k_scan_total(long long* out, long long n, const int* in, const long long* in64) {
    // out[n] = out[n-1] + in[n-1]
    if (n == 0) { out[0] = 0; return; }
    out[n] = out[n - 1] + (in ? (long long)in[n - 1] : in64[n - 1]);
}

void scan_rec(const int* in, const long long* in64, long long* out, long long n, long long* tmp, cudaStream_t st) {
    if (n == 0) return;
    const long long nb = (n + kScanBlock - 1) / kScanBlock;
    long long* sums = tmp;
    long long* sums_scan = tmp + nb;
    count_launch(), k_scan_block<<<(unsigned)nb, kScanBlock, 0, st>>>(in, in64, out, n, sums);
    if (nb > 1) {
        scan_rec(nullptr, sums, sums_scan, nb, tmp + 2 * nb, st);
        count_launch(), k_scan_add<<<(unsigned)nb, kScanBlock, 0, st>>>(out, n, sums_scan);
    }
}

unsigned grid_for(long long n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace

// Kernel launches enqueued by this library (all threads; a per-engine count
// is the difference across one enqueue sequence on that engine's thread).
static std::atomic<long long> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long launch_counter() { return g_launches.load(std::memory_order_relaxed); }

size_t scan_tmp_bytes(long long n) {
    size_t total = 0;
    long long m = n;
    while (m > 1) {
        long long nb = (m + kScanBlock - 1) / kScanBlock;
        total += 2 * nb;
        m = nb;
    }
    return (total + 16) * sizeof(long long);
}

namespace {

// Up to two scans side by side (blockIdx.y): tiles of kScanBlock scanned in
// place with the tile sums recorded; a single tile also writes the total.
struct ScanPair {
    const int* in[2];
    long long* out[2];
    long long* sums[2];
};

__global__ void __launch_bounds__(kScanBlock) k_scan_tiles(ScanPair a, long long n) {
    const int y = blockIdx.y;
    __shared__ long long wsum[32];
    const long long i = (long long)blockIdx.x * kScanBlock + threadIdx.x;
    const long long v = i < n ? (long long)a.in[y][i] : 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long x = v;
    for (int off = 1; off < 32; off <<= 1) {
        const long long t = __shfl_up_sync(kFull, x, off);
        if (lane >= off) x += t;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        long long t = wsum[lane];
        for (int off = 1; off < 32; off <<= 1) {
            const long long u = __shfl_up_sync(kFull, t, off);
            if (lane >= off) t += u;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    const long long incl = x + (w ? wsum[w - 1] : 0);
    if (i < n) a.out[y][i] = incl - v;
    if (threadIdx.x == kScanBlock - 1) {
        a.sums[y][blockIdx.x] = incl;
        if (gridDim.x == 1) a.out[y][n] = incl;
    }
}

// tile b adds the sum of tiles 0..b-1 (reduced by the block itself, at most
// kScanBlock tiles); the last tile writes the total at out[n]
__global__ void __launch_bounds__(kScanBlock) k_scan_offsets(ScanPair a, long long n) {
    const int y = blockIdx.y;
    const int b = blockIdx.x;
    __shared__ long long wsum[32];
    long long v = threadIdx.x < b ? a.sums[y][threadIdx.x] : 0;
    for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
    __syncthreads();
    long long offs = 0;
    for (int k = 0; k < kScanBlock / 32; k++) offs += wsum[k];
    const long long i = (long long)b * kScanBlock + threadIdx.x;
    if (i < n) a.out[y][i] += offs;
    if (b == (int)gridDim.x - 1 && threadIdx.x == 0) a.out[y][n] = offs + a.sums[y][b];
}

// nb <= kScanBlock tiles: two launches for one or two arrays
void scan_small(int m, const int* ia, long long* oa, const int* ib, long long* ob, long long n, long long* tmp,
                cudaStream_t st) {
    const long long nb = (n + kScanBlock - 1) / kScanBlock;
    ScanPair a;
    a.in[0] = ia; a.out[0] = oa; a.sums[0] = tmp;
    a.in[1] = ib; a.out[1] = ob; a.sums[1] = tmp + nb;
    const dim3 grid((unsigned)nb, (unsigned)m);
    count_launch(), k_scan_tiles<<<grid, kScanBlock, 0, st>>>(a, n);
    if (nb > 1) count_launch(), k_scan_offsets<<<grid, kScanBlock, 0, st>>>(a, n);
}

}  // namespace

void exclusive_scan(const int* in, long long* out, long long n, void* tmp, cudaStream_t st) {
    if (n > 0 && n <= (long long)kScanBlock * kScanBlock) {
        scan_small(1, in, out, in, out, n, (long long*)tmp, st);
        return;
    }
    scan_rec(in, nullptr, out, n, (long long*)tmp, st);
    count_launch(), k_scan_total<<<1, 1, 0, st>>>(out, n, in, nullptr);
}

void exclusive_scan2(const int* in_a, long long* out_a, const int* in_b, long long* out_b, long long n, void* tmp,
                     cudaStream_t st) {
    if (n > 0 && n <= (long long)kScanBlock * kScanBlock) {
        scan_small(2, in_a, out_a, in_b, out_b, n, (long long*)tmp, st);
        return;
    }
    exclusive_scan(in_a, out_a, n, tmp, st);
    exclusive_scan(in_b, out_b, n, tmp, st);
}

void launch_atoms(const BatchView& B, cudaStream_t st) {
    // small blocks: the per-atom cell algebra is FP64 work, spread over as many SMs as possible
    if (B.n_atoms_total) count_launch(), launch_chained(k_atoms, grid_for(B.n_atoms_total, 32), 32, 0, st, B);
}
void launch_ghosts(const BatchView& B, cudaStream_t st) {
    if (B.n_ghost_total) count_launch(), launch_chained(k_ghosts, grid_for(B.n_ghost_total, 64), 64, 0, st, B);
}
void launch_bin_alloc(const BatchView& B, cudaStream_t st) {
    if (B.n_bins_total) count_launch(), launch_chained(k_bin_alloc, grid_for(B.n_bins_total, 1024), 1024, 0, st, B);
}
void launch_bin_scatter(const BatchView& B, cudaStream_t st) {
    if (B.n_ghost_total) count_launch(), launch_chained(k_bin_scatter, grid_for(B.n_ghost_total, 256), 256, 0, st, B, B.bin_start);
}
void launch_bin_sort(const BatchView& B, cudaStream_t st) {
    if (!B.n_bins_total) return;
    // bins per warp: one while that still gives a few warps per resident slot
    // (a small batch's bins are few and mostly occupied), else 32 (a large
    // batch reserves many times the bins its ghost clouds occupy)
    const int per = B.n_bins_total > 64LL * 32 * sm_count() ? 32 : 1;
    const long long warps = (B.n_bins_total + per - 1) / per;
    count_launch(), launch_chained(k_bin_rank, grid_for(warps * 32, 256), 256, 0, st, B, B.bin_start, per);
}
void launch_l2(const BatchView& B, int* l2_owner, cudaStream_t st) {
    if (B.n_atoms_total)
        count_launch(), launch_chained(k_l2, grid_for(B.n_atoms_total * 32, kL2Block), kL2Block, 0, st, B, l2_owner);
}
void launch_enum(const BatchView& B, const int* l2_owner, void* scan_tmp, cudaStream_t st) {
    if (!B.n2_cap) return;
    if (B.enum_serial) {
        long long want = (long long)sm_count() * 16;
        long long need = (B.n2_cap + 127) / 128;
        const unsigned grid = (unsigned)(want < need ? want : need);
        count_launch(), k_enum<false><<<grid, 128, 0, st>>>(B, l2_owner);
        exclusive_scan2(B.e_cnt3, B.e_off3, B.e_cnt4, B.e_off4, B.n2_cap, scan_tmp, st);
        count_launch(), k_enum<true><<<grid, 128, 0, st>>>(B, l2_owner);
        return;
    }
    // warps per atom: the fewest that still give about two warps per
    // resident warp slot (32 per SM)
    const long long target = 64LL * sm_count();
    const long long n = B.n_atoms_total;
    const int G = n >= target ? 1 : 2 * n >= target ? 2 : 4 * n >= target ? 4 : 8;
    switch (G) {
    case 1: launch_enuma<1>(B, l2_owner, st); break;
    case 2: launch_enuma<2>(B, l2_owner, st); break;
    case 4: launch_enuma<4>(B, l2_owner, st); break;
    default: launch_enuma<8>(B, l2_owner, st); break;
    }
}
void launch_reset(const BatchView& B, cudaStream_t st) {
    long long n = std::max(std::max(8LL * B.n_sys, 3 * B.n_in_total), std::max(B.n_bins_total, 8LL));
    if (B.l2_hash) n = std::max(n, B.l2_slots / 4);
    n = std::min((n + 255) / 256, 16LL * sm_count());
    count_launch(), k_reset<<<(unsigned)n, 256, 0, st>>>(B);
}

}  // namespace ck
