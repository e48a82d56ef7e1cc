// Differentiable LP layer: K unrolled PDHG iterations with fixed steps and
// their exact reverse mode (igaos_pdhg_unrolled_*).
//
// One thread-block cluster of C CTAs per instance (C = 1 for small ones). The
// rows and columns are sorted by length and dealt to the CTAs in slices of 32,
// one lane per row; a CTA keeps its slices' entries in shared memory, values
// and 16-bit indices, jagged: the k-th entries of a slice's rows that have one
// lie next to each other (the longest rows have the lowest lanes, so these are
// a prefix), and a warp reads a run of consecutive words without padding.
// Vectors that rows or columns read and write themselves are held by their
// CTA in that order, and the gathered ones (x_bar and y; the adjoints of z and
// of the reduced cost) lie in it too, rank after rank, with a copy in every
// CTA: a warp writes its slice of them as one run, to its own shared memory
// and to the others' (distributed shared memory). The staged indices are
// positions in that order. An iteration touches global memory only for
// checkpoints and replay records. Each row's products are
// summed by its lane in the order of the CSR (CSC), whatever the mapping, so
// results depend neither on C nor on the launch.
// An instance whose share does not fit reads its matrix from global memory.
//
// The forward stores (x_k, y_k) every `checkpoint` iterations. The backward
// walks the segments last to first: it replays a segment from its
// checkpoint, keeping each step's extrapolated primal x_bar, the dual y_k
// and the clamp outcome of every coordinate, then runs the segment's adjoint
// steps in reverse. The gradient of A's values is accumulated by the row
// pass alone (row i owns its nonzeros), in the CSR order of the input.
//
// Iteration (reference sign convention, d = c + A^T y; kern_primal /
// kern_dual in src/pdhg/pdhg.cu:33-58; ridge term in the primal prox):
//   g = c + A^T y;  v = (x - tau g) kappa, kappa = 1 / (1 + 2 ridge tau)
//   x+ = clamp(v, cl, cu);  xb = 2 x+ - x
//   t = y + sigma A xb;  y+ = t - sigma clamp(t / sigma, rmin, rmax)
// Clamps are differentiated almost everywhere: the gradient passes to the
// argument where it lies inside the bounds (ties included), to the bound
// where it lies strictly outside.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "device.cuh"
#include "engine.hpp"

namespace igx {
namespace {

constexpr int kLT = 512;          // most threads per CTA
constexpr int kLW = kLT / 32;
constexpr int kMaxCluster = 8;    // CTAs per instance (portable cluster size)
constexpr int kBins = 1024;       // length classes of the counting sort
constexpr unsigned kFull = 0xffffffffu;

template <typename T>
struct UArgs {
    int K, ck;
    T ridge;
    const int *row_off, *col_off, *nz_off, *ap, *ai, *cp, *ci, *cperm;
    const T *c, *cl, *cu, *rmin, *rmax, *ax, *tau, *sigma;
    T *x, *y, *obj, *ckpt;
    long long nck;
    // backward
    const T *xK, *gx, *gy, *gobj;
    T *gc, *gcl, *gcu, *grmin, *grmax, *gax;
    T* seg;
    unsigned char* segf;
    // steps
    T omega;
    T *tau_o, *sigma_o;
    // launch geometry (plan())
    int max_m, max_n, lc, lr;  // sizes and local slices (columns, rows) of the largest instance
    int ngc, ngr;              // entries of a gathered column and row vector
    int per_cta;               // row entries of a CTA of the largest instance
    int vec_bytes, ent_bytes;  // shared memory of the vectors, and of the staged entries
    bool lean;                 // backward: see bwd_elems
};

struct UInst {
    int m, n, nnz, nz0;
    long long r0, c0;
};

template <typename T>
__device__ __forceinline__ UInst uinst(const UArgs<T>& a, int b) {
    UInst I;
    I.r0 = a.row_off[b];
    I.c0 = a.col_off[b];
    I.m = a.row_off[b + 1] - (int)I.r0;
    I.n = a.col_off[b + 1] - (int)I.c0;
    I.nz0 = a.nz_off[b];
    I.nnz = a.nz_off[b + 1] - I.nz0;
    return I;
}

// CTAs of the launch's cluster that work on instance I: as many as keep a
// CTA's share (entries and slices) at most the largest instance's. The others leave at once, and
// their SMs take the next instance (a cluster barrier counts the threads that
// have not exited).
template <typename T>
__device__ __forceinline__ int u_ctas(const UArgs<T>& a, const UInst& I) {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    const int by_slices = max(((I.n + 31) / 32 + a.lc - 1) / a.lc, ((I.m + 31) / 32 + a.lr - 1) / a.lr);
    return min((int)r, max(max(1, by_slices), (I.nnz + a.per_cta - 1) / a.per_cta));
}

// ------------------------------------------------------------ the cluster
__device__ __forceinline__ int u_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ int u_instance() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return blockIdx.x / r;
}
// every thread of the instance's CTAs; orders shared memory, the copies in
// other CTAs' shared memory and global memory
__device__ __forceinline__ void u_sync(int C) {
    if (C == 1) {
        __syncthreads();
    } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
                     "barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}
// v into the entry `at` (an address in this CTA's copy) of every copy
template <typename V>
__device__ __forceinline__ void bcast(V* at, V v, int C) {
    if (C == 1) {
        *at = v;
        return;
    }
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    for (int r = 0; r < C; ++r) *cl.map_shared_rank(at, r) = v;
}

// ------------------------------------------------------------- numerics
// Comparisons of doubles on the integer pipe (this GPU's FP64 pipe does two
// operations per clock per SM and bounds the FP64 kernels); -0 equals +0 and
// nothing compares with a NaN, as in FP64 instructions.
__device__ __forceinline__ bool u_lt(float a, float b) { return a < b; }
__device__ __forceinline__ bool u_lt(double a, double b) {
    const long long inf = 0x7ff0000000000000LL;
    long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    if ((x & ~(1LL << 63)) > inf || (y & ~(1LL << 63)) > inf) return false;
    x = x < 0 ? (1LL << 63) - x : x;  // -0 -> 0, negatives in their order
    y = y < 0 ? (1LL << 63) - y : y;
    return x < y;
}
// clamp with its outcome: 0 inside (ties included), 1 below lo, 2 above hi
template <typename T>
__device__ __forceinline__ T clampf(T v, T lo, T hi, int& f) {
    if (u_lt(v, lo)) {
        f = 1;
        return lo;
    }
    if (u_lt(hi, v)) {
        f = 2;
        return hi;
    }
    f = 0;
    return v;
}
// t / s for one divisor s many times, is = u_recip(s). FP64: the product with
// the correctly rounded reciprocal and one remainder step, the correctly rounded
// quotient (Markstein 1990) in three operations on the FP64 pipe instead of the
// division's. (Where t / s is so close to the middle of two doubles that the step's
// own error could decide, the product is half an ulp off, and the error s / 2^54 of
// what a quotient's distance from a middle is at least.) Operands far from 1
// by hundreds of binades, where a step could leave the normal range, divide.
__device__ __forceinline__ bool u_tame(double v) {
    const int ex = (__double2hiint(v) >> 20) & 0x7ff;
    return ex > 512 && ex < 1536;
}
__device__ __forceinline__ float u_recip(float) { return 0.f; }
__device__ __forceinline__ double u_recip(double s) { return u_tame(s) ? 1.0 / s : 0.0; }
__device__ __forceinline__ float u_div(float t, float s, float) { return t / s; }
__device__ __forceinline__ double u_div(double t, double s, double is) {
    const double q0 = t * is;
    if (!u_tame(q0) || !u_tame(t)) return t / s;
    return fma(fma(-s, q0, t), is, q0);
}
// Exact widening of a staged float (zero or normal: stage() leaves an
// instance with others in global memory) on the integer pipe; the conversion
// instruction runs at the FP64 pipe's rate.
__device__ __forceinline__ bool u_plain(double) { return true; }
__device__ __forceinline__ bool u_plain(float v) {
    const int ex = (__float_as_int(v) >> 23) & 0xff;
    return (ex != 0 && ex != 0xff) || v == 0.f;
}
__device__ __forceinline__ double u_wide(float v) {
    const int b = __float_as_int(v), mag = b & 0x7fffffff;
    return __hiloint2double((b & 0x80000000) | (mag ? (mag >> 3) + (896 << 20) : 0), b << 29);
}

// ---------------------------------------------------------------- staging
// One orientation's rows as this CTA holds them: local slice l is slice
// l C + rank of the sorted rows (ranks in reverse order in every other l, so
// that no rank keeps getting the longest), its lane i holds row id[32 l + i]
// with len[32 l + i] entries (0 past the last row).
template <typename T>
struct Share {
    int rows, slices, first;  // first: position of local slice 0 in the gathered order
    uint16_t* id;
    int* len;
    int* base;             // first staged entry of each local slice
    T* val;                // staged entries (resident instances)
    uint16_t* idx;
    const int *ptr, *gidx, *gperm;  // the CSR (gperm: CSC entry -> CSR entry)
    const T* gval;
    const uint16_t* gpos;  // position of each index gidx in the gathered order
};
__device__ __forceinline__ int u_slice(int l, int rank, int C) {
    return l * C + ((l & 1) ? C - 1 - rank : rank);
}
// local slices of `rank` among `slices`
__device__ __forceinline__ int u_local(int slices, int rank, int C) {
    const int l = slices / C;
    return l + (u_slice(l, rank, C) < slices ? 1 : 0);
}

// Shared memory of one instance; the same carving on every CTA.
template <typename T>
struct Plan {
    Share<T> col, row;
    bool resident;
    T* gax;                // backward: gradient of the staged row entries
    unsigned char* vec;    // vectors (unused until staging is done)
};

// rows by decreasing length (classes of at least kBins - 1 unsorted): order
// by a counting sort, whose ties are in no fixed order
__device__ void sort_rows(const int* ptr, int rows, uint16_t* order, int* bins) {
    const int nt = blockDim.x;
    for (int k = threadIdx.x; k < kBins; k += nt) bins[k] = 0;
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += nt)
        atomicAdd(&bins[kBins - 1 - min(ptr[r + 1] - ptr[r], kBins - 1)], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
        constexpr int kPer = kBins / 32;
        int s = 0;
        for (int k = 0; k < kPer; ++k) s += bins[threadIdx.x * kPer + k];
        int pre = s;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kFull, pre, o);
            if ((int)threadIdx.x >= o) pre += v;
        }
        int run = pre - s;
        for (int k = 0; k < kPer; ++k) {
            const int v = bins[threadIdx.x * kPer + k];
            bins[threadIdx.x * kPer + k] = run;
            run += v;
        }
    }
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += nt)
        order[atomicAdd(&bins[kBins - 1 - min(ptr[r + 1] - ptr[r], kBins - 1)], 1)] = (uint16_t)r;
    __syncthreads();
}

// length and row of position q of the order, sorted again inside the slice
// (longest first; rows beyond the last: length 0, row 0xffff)
__device__ __forceinline__ void slice_rows(const int* ptr, int rows, const uint16_t* order, int s,
                                           int& row, int& len) {
    const int lane = threadIdx.x & 31, q = s * 32 + lane;
    row = 0xffff;
    long long key = -1;
    if (q < rows) {
        row = order[q];
        key = (long long)(ptr[row + 1] - ptr[row]) << 16 | row;
    }
    for (int k = 2; k <= 32; k <<= 1)
        for (int o = k >> 1; o > 0; o >>= 1) {
            const long long other = __shfl_xor_sync(kFull, key, o);
            const bool larger = ((lane & o) == 0) == ((lane & k) == 0);
            key = larger == (key > other) ? key : other;
        }
    row = key < 0 ? 0xffff : (int)(key & 0xffff);
    len = key < 0 ? 0 : (int)(key >> 16);
}

// shared memory of the meta data of a CTA: lengths, slice bases and ids of
// its rows, the positions of every column and row
__host__ __device__ inline size_t meta_bytes(int m, int n, int lc, int lr) {
    return ((size_t)(lc + lr) * (32 * (4 + 2) + 4) + (size_t)(m + n) * 2 + 15) & ~(size_t)15;
}
// staging's own scratch, inside the vectors' space
__host__ __device__ inline size_t scratch_bytes(int m, int n) {
    return kBins * 4 + (size_t)(m + n) * 2 + ((size_t)(m + n) / 32 + 2) * 4 + 64;
}

// entries of rank r's share (all threads of the calling warp get the sum)
__device__ __forceinline__ int share_total(const int* tot, int slices, int r, int C) {
    int s = 0;
    for (int l = threadIdx.x & 31; l < u_local(slices, r, C); l += 32) s += tot[u_slice(l, r, C)];
    return __reduce_add_sync(kFull, s);
}

// Carves the CTA's shared memory, sorts the instance's rows and columns and
// stages this CTA's entries; ends with every thread past a block barrier.
// GRAD reserves the gradient of the row entries; WIDE: the products are in
// FP64. The values are staged as they are (the CSC ones gathered through each
// entry's CSR position).
template <typename T, bool GRAD, bool WIDE>
__device__ Plan<T> stage(const UArgs<T>& a, const UInst& I, int b, unsigned char* smem, int rank,
                         int C) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int m = I.m, n = I.n;
    __shared__ int s_res, s_ent[2];
    bool odd = false;  // a staged value that u_wide does not take
    Plan<T> P;
    P.vec = smem;
    unsigned char* meta = smem + a.vec_bytes;
    unsigned char* ent = meta + meta_bytes(a.max_m, a.max_n, a.lc, a.lr);
    int* words = reinterpret_cast<int*>(meta);
    uint16_t* ids = reinterpret_cast<uint16_t*>(words + 33 * (a.lc + a.lr));
    uint16_t* pos_c = ids + 32 * (a.lc + a.lr);
    uint16_t* pos_r = pos_c + n;
    P.col = Share<T>{n, 0, 32 * a.lc * rank, ids, words, words + 32 * a.lc, nullptr, nullptr,
                     a.cp + I.c0 + b, a.ci + I.nz0, a.cperm + I.nz0, a.ax + I.nz0, pos_r};
    words += 33 * a.lc;
    P.row = Share<T>{m, 0, 32 * a.lr * rank, ids + 32 * a.lc, words, words + 32 * a.lr, nullptr, nullptr,
                     a.ap + I.r0 + b, a.ai + I.nz0, nullptr, a.ax + I.nz0, pos_c};
    const int sc = (n + 31) / 32, sr = (m + 31) / 32;
    P.col.slices = u_local(sc, rank, C);
    P.row.slices = u_local(sr, rank, C);
    // scratch: length classes, entries per slice, the two orders
    int* bins = reinterpret_cast<int*>(smem);
    int* tot_c = bins + kBins;
    int* tot_r = tot_c + sc;
    uint16_t* ord_c = reinterpret_cast<uint16_t*>(tot_r + sr);
    uint16_t* ord_r = ord_c + n;
    if (rank == 0) {
        sort_rows(P.col.ptr, n, ord_c, bins);
        sort_rows(P.row.ptr, m, ord_r, bins);
    }
    if (C > 1) {  // every CTA works on rank 0's order
        u_sync(C);
        if (rank != 0) {
            cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
            const uint16_t* from = cl.map_shared_rank(ord_c, 0);
            for (int q = threadIdx.x; q < n + m; q += blockDim.x) ord_c[q] = from[q];
        }
        u_sync(C);
    }
    for (int w = wp; w < sc + sr; w += nw) {
        const bool c = w < sc;
        const Share<T>& S = c ? P.col : P.row;
        const int s = c ? w : w - sc, l = s / C, r = (l & 1) ? C - 1 - s % C : s % C;
        int row, len;
        slice_rows(S.ptr, S.rows, c ? ord_c : ord_r, s, row, len);
        if (row != 0xffff)
            (c ? pos_c : pos_r)[row] = (uint16_t)(32 * ((c ? a.lc : a.lr) * r + l) + lane);
        if (r == rank) {
            S.id[32 * l + lane] = (uint16_t)row;
            S.len[32 * l + lane] = len;
        }
        len = __reduce_add_sync(kFull, len);
        if (lane == 0) tot_c[w] = len;
    }
    __syncthreads();
    if (wp == 0) {  // does every rank's share fit?
        bool fits = true;
        for (int r = 0; r < C; ++r) {
            const int ec = share_total(tot_c, sc, r, C), er = share_total(tot_r, sr, r, C);
            const long long need = (long long)(ec + er) * (sizeof(T) + 2) +
                                   (GRAD ? (long long)er * sizeof(T) : 0) + 16;
            fits = fits && need <= a.ent_bytes;
            if (r == rank && lane == 0) {
                s_ent[0] = ec;
                s_ent[1] = er;
            }
        }
        if (lane == 0) s_res = fits;
        for (int o = 0; o < 2; ++o) {  // first entry of each local slice
            const int* tot = o ? tot_r : tot_c;
            int* base = o ? P.row.base : P.col.base;
            const int cnt = o ? P.row.slices : P.col.slices;
            int run = 0;
            for (int l0 = 0; l0 < cnt; l0 += 32) {
                const int l = l0 + lane, v = l < cnt ? tot[u_slice(l, rank, C)] : 0;
                int pre = v;
                for (int d = 1; d < 32; d <<= 1) {
                    const int w = __shfl_up_sync(kFull, pre, d);
                    if (lane >= d) pre += w;
                }
                if (l < cnt) base[l] = run + pre - v;
                run += __shfl_sync(kFull, pre, 31);
            }
        }
    }
    __syncthreads();
    P.resident = s_res != 0;
    const int ec = s_ent[0], er = s_ent[1];
    P.col.val = reinterpret_cast<T*>(ent);
    P.row.val = P.col.val + ec;
    P.gax = P.row.val + er;
    P.col.idx = reinterpret_cast<uint16_t*>(P.gax + (GRAD ? er : 0));
    P.row.idx = P.col.idx + ec;
    for (int w = wp; P.resident && w < P.col.slices + P.row.slices; w += nw) {
        const bool c = w < P.col.slices;
        const Share<T>& S = c ? P.col : P.row;
        const int l = c ? w : w - P.col.slices;
        const int row = S.id[32 * l + lane], len = S.len[32 * l + lane];
        const int p0 = row == 0xffff ? 0 : S.ptr[row];
        const int longest = __shfl_sync(kFull, len, 0);
        int off = S.base[l];
        for (int k = 0; k < longest; ++k) {
            const bool on = k < len;
            if (on) {
                const int p = p0 + k;
                const T v = S.gval[c ? S.gperm[p] : p];
                S.idx[off + lane] = S.gpos[S.gidx[p]];
                S.val[off + lane] = v;
                if (WIDE) odd = odd || !u_plain(v);
                if (GRAD && !c) P.gax[off + lane] = T(0);
            }
            off += __popc(__ballot_sync(kFull, on));
        }
    }
    if (WIDE && __syncthreads_or(odd)) P.resident = false;
    u_sync(C);  // the scratch is free for the vectors from here, in every CTA
    return P;
}

// acc + the products of the lane's row with v, in the row's order; U is the
// accumulator's type (FP64 products of FP32 values: two chains, even and odd
// entries). Up to the shortest row of the slice every lane has an entry, at
// fixed offsets: batches without predicates or offsets to find. The rest goes
// four at a time with a ballot each (rows of a slice are of like length).
template <bool RES, typename T, typename U>
__device__ __forceinline__ U row_dot(const Share<T>& S, int l, int q, const U* __restrict__ v,
                                     U acc) {
    constexpr bool kTwo = !std::is_same<T, U>::value;
    constexpr int B = sizeof(U) == 4 ? 8 : 4;
    const int lane = threadIdx.x & 31, len = S.len[q];
    int k = 0;
    if constexpr (RES) {
        const int longest = __shfl_sync(kFull, len, 0);
        const int shortest = __shfl_sync(kFull, len, 31);
        const int first = S.base[l];
        const T* val = S.val + first + lane;
        const uint16_t* idx = S.idx + first + lane;
        U odd = U(0);
        for (; k + B <= shortest; k += B) {
            T a[B];
            int j[B];
            U x[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                a[u] = val[32 * u];
                j[u] = idx[32 * u];
            }
#pragma unroll
            for (int u = 0; u < B; ++u) x[u] = v[j[u]];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                if constexpr (std::is_same<T, U>::value) acc = fma(a[u], x[u], acc);
                else if (u & 1) odd = fma(u_wide(a[u]), x[u], odd);
                else acc = fma(u_wide(a[u]), x[u], acc);
            }
            val += 32 * B;
            idx += 32 * B;
        }
        for (; k < longest; k += 4) {
            T a[4];
            int j[4];
            U x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool on = k + u < len;
                a[u] = T(0);
                j[u] = 0;
                if (on) {
                    a[u] = *val;
                    j[u] = *idx;
                }
                const int cnt = __popc(__ballot_sync(kFull, on));
                val += cnt;
                idx += cnt;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = v[j[u]];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                // (uniform: an FP64 instruction takes its slot with no lane on)
                if (sizeof(U) == 8 && k + u >= longest) break;
                if (k + u < len) {
                    if constexpr (std::is_same<T, U>::value) acc = fma(a[u], x[u], acc);
                    else if (u & 1) odd = fma(u_wide(a[u]), x[u], odd);
                    else acc = fma(u_wide(a[u]), x[u], acc);
                }
            }
        }
        if constexpr (kTwo) acc += odd;
    } else {
        const int p0 = len > 0 ? S.ptr[S.id[q]] : 0;
        U odd = U(0);
        for (; k < len; k += 4) {
            U a[4], x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int p = p0 + min(k + u, len - 1);
                a[u] = (U)S.gval[S.gperm ? S.gperm[p] : p];
                x[u] = v[S.gpos[S.gidx[p]]];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k + u < len) {
                    if (kTwo && (u & 1)) odd = fma(a[u], x[u], odd);
                    else acc = fma(a[u], x[u], acc);
                }
        }
        if constexpr (kTwo) acc += odd;
        __syncwarp();
    }
    return acc;
}

// ---------------------------------------------------------------- forward
// Vectors of the forward pass by local position (32 slices + lane), and the
// gathered copies.
template <typename T>
struct FwdVec {
    T *x, *c, *lo, *hi;  // columns
    T *rl, *rh;          // rows
    T *xb, *y;           // copies (ngc, ngr)
};
template <typename T>
__host__ __device__ inline size_t fwd_elems(int lc, int lr, int C) {
    return (size_t)32 * ((4 + C) * (size_t)lc + (2 + C) * (size_t)lr);
}
template <typename T>
__device__ __forceinline__ FwdVec<T> fwd_vec(const UArgs<T>& a, unsigned char* base) {
    const int qc = 32 * a.lc, qr = 32 * a.lr;
    T* p = reinterpret_cast<T*>(base);
    FwdVec<T> V;
    V.x = p;
    V.c = V.x + qc;
    V.lo = V.c + qc;
    V.hi = V.lo + qc;
    V.rl = V.hi + qc;
    V.rh = V.rl + qr;
    V.xb = V.rh + qr;
    V.y = V.xb + a.ngc;
    return V;
}

// one column's primal step, q its local position; returns the clamp outcome
template <bool RES, typename T>
__device__ __forceinline__ int fwd_col(const Plan<T>& P, int l, int q, T* x, T c, T l0, T h0, T* xb,
                                       const T* y, T tau, T kappa, int C, T& xbv) {
    const T xv = x[q];
    const T g = row_dot<RES, T, T>(P.col, l, q, y, c);
    const T v = (xv - tau * g) * kappa;
    int f;
    const T xn = clampf(v, l0, h0, f);
    xbv = T(2) * xn - xv;
    x[q] = xn;
    bcast(xb + P.col.first + q, xbv, C);
    return f;
}

// one row's dual step from its dual yv; returns the clamp outcome
template <bool RES, typename T>
__device__ __forceinline__ int fwd_row(const Plan<T>& P, int l, int q, T l0, T h0, const T* xb, T* y,
                                       T yv, T sigma, T isigma, int C) {
    const T z = row_dot<RES, T, T>(P.row, l, q, xb, T(0));
    const T t = fma(sigma, z, yv);
    int f;
    const T pr = clampf(u_div(t, sigma, isigma), l0, h0, f);
    bcast(y + P.row.first + q, fma(-sigma, pr, t), C);
    return f;
}

template <bool RES, typename T>
__device__ void fwd_body(const UArgs<T>& a, const UInst& I, int b, const Plan<T>& P, int C) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int m = I.m, n = I.n;
    const FwdVec<T> V = fwd_vec(a, P.vec);
    const T tau = a.tau[b], sigma = a.sigma[b];
    const T kappa = T(1) / (T(1) + T(2) * a.ridge * tau);
    const T isigma = u_recip(sigma);
    for (int l = wp; l < P.col.slices; l += nw) {
        const int q = 32 * l + lane, j = P.col.id[q];
        if (j == 0xffff) {
            V.c[q] = V.lo[q] = V.hi[q] = V.x[q] = T(0);
            continue;
        }
        int f;
        V.c[q] = a.c[I.c0 + j];
        V.lo[q] = a.cl[I.c0 + j];
        V.hi[q] = a.cu[I.c0 + j];
        V.x[q] = clampf(T(0), V.lo[q], V.hi[q], f);
    }
    for (int l = wp; l < P.row.slices; l += nw) {
        const int q = 32 * l + lane, i = P.row.id[q];
        V.rl[q] = i == 0xffff ? T(0) : a.rmin[I.r0 + i];
        V.rh[q] = i == 0xffff ? T(0) : a.rmax[I.r0 + i];
    }
    for (int i = threadIdx.x; i < a.ngr; i += blockDim.x) V.y[i] = T(0);
    T* ck = a.ckpt + a.nck * (I.c0 + I.r0);
    int next = 0;
    u_sync(C);
    for (int k = 0; k < a.K; ++k) {
        if (k == next) {
            next += a.ck;
            for (int l = wp; l < P.col.slices; l += nw) {
                const int q = 32 * l + lane, j = P.col.id[q];
                if (j != 0xffff) ck[j] = V.x[q];
            }
            for (int l = wp; l < P.row.slices; l += nw) {
                const int q = 32 * l + lane, i = P.row.id[q];
                if (i != 0xffff) ck[n + i] = V.y[P.row.first + q];
            }
            ck += n + m;
        }
        for (int l = wp; l < P.col.slices; l += nw) {
            const int q = 32 * l + lane;
            T xb;
            fwd_col<RES>(P, l, q, V.x, V.c[q], V.lo[q], V.hi[q], V.xb, V.y, tau, kappa, C, xb);
        }
        u_sync(C);
        for (int l = wp; l < P.row.slices; l += nw) {
            const int q = 32 * l + lane;
            const T yv = V.y[P.row.first + q];
            fwd_row<RES>(P, l, q, V.rl[q], V.rh[q], V.xb, V.y, yv, sigma, isigma, C);
        }
        u_sync(C);
    }
    for (int l = wp; l < P.col.slices; l += nw) {
        const int q = 32 * l + lane, j = P.col.id[q];
        if (j != 0xffff) a.x[I.c0 + j] = V.x[q];
    }
    for (int l = wp; l < P.row.slices; l += nw) {
        const int q = 32 * l + lane, i = P.row.id[q];
        if (i != 0xffff) a.y[I.r0 + i] = V.y[P.row.first + q];
    }
    u_sync(C);
}

// Bound by the shared-memory pipe in FP32 (72 % busy: a warp's 32 gathers fall
// on random banks, about 3.5 wavefronts, beside one each for values and
// indices) and by the FP64 pipe in FP64 (65 %). 152 LPs of 500 x 1,000, 200
// iterations, FP32: 0.66 ms; 1.0 ms with one lane per row walking a CSR.
template <typename T>
__global__ void __launch_bounds__(kLT) k_unroll_fwd(UArgs<T> a) {
    extern __shared__ __align__(16) unsigned char u_smem[];
    __shared__ double red[kLW];
    const int rank = u_rank(), b = u_instance(), t = threadIdx.x;
    const UInst I = uinst(a, b);
    const int C = u_ctas(a, I);
    if (rank >= C) return;
    const Plan<T> P = stage<T, false, false>(a, I, b, u_smem, rank, C);
    if (P.resident) fwd_body<true>(a, I, b, P, C);
    else fwd_body<false>(a, I, b, P, C);
    if (rank != 0) return;
    // the objective, in index order in the shape of kLW warps, whatever the
    // launch
    for (int w = t >> 5; w < kLW; w += blockDim.x >> 5) {
        double o = 0.0;
        for (int j = 32 * w + (t & 31); j < I.n; j += kLT) {
            const T xv = __ldcg(a.x + I.c0 + j);
            o += (double)a.c[I.c0 + j] * (double)xv + (double)a.ridge * (double)xv * (double)xv;
        }
        o = warp_sum(o);
        if ((t & 31) == 0) red[w] = o;
    }
    __syncthreads();
    if (t == 0) {
        double s = 0.0;
        for (int w = 0; w < kLW; ++w) s += red[w];
        a.obj[b] = (T)s;
    }
}

// --------------------------------------------------------------- backward
// Vectors of the backward pass by local position, and the gathered copies.
// Replay and reverse steps share the copies' space: the duals' with
// the adjoint of z, x_bar's and x with the pairs (adjoint of the reduced cost,
// x_bar).
template <typename T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

template <typename T>
struct BwdVec {
    T *c, *lo, *hi, *xh, *gc, *gl, *gu;  // columns
    T *rl, *rh, *yh, *th, *grl, *grh;    // rows
    typename Pair<T>::type* gp;          // copy (ngc): reverse steps
    T *xb, *x, *y;                       // replay: copy and x (gp's space); copy (ngr)
    T* zh;                               // copy (ngr): reverse steps (y's space)
};
// Lean: costs and bounds (c, lo, hi, rl, rh) are read where the caller has them
// instead, in global memory.
template <typename T>
__host__ __device__ inline size_t bwd_elems(int lc, int lr, int C, bool lean) {
    return (size_t)32 * (((lean ? 4 : 7) + 2 * C) * (size_t)lc + ((lean ? 4 : 6) + C) * (size_t)lr);
}
template <bool LEAN, typename T>
__device__ __forceinline__ BwdVec<T> bwd_vec(const UArgs<T>& a, unsigned char* base) {
    const int qc = 32 * a.lc, qr = 32 * a.lr;
    T* p = reinterpret_cast<T*>(base);
    BwdVec<T> V;
    V.gp = reinterpret_cast<typename Pair<T>::type*>(p);
    V.xb = p;
    V.x = p + a.ngc;
    V.xh = p + 2 * (size_t)a.ngc;
    V.gc = V.xh + qc;
    V.gl = V.gc + qc;
    V.gu = V.gl + qc;
    V.c = V.gu + qc;
    V.lo = V.c + (LEAN ? 0 : qc);
    V.hi = V.lo + (LEAN ? 0 : qc);
    V.rl = V.hi + (LEAN ? 0 : qc);
    V.rh = V.rl + (LEAN ? 0 : qr);
    V.yh = V.rh + (LEAN ? 0 : qr);
    V.th = V.yh + qr;
    V.grl = V.th + qr;
    V.grh = V.grl + qr;
    V.y = V.zh = V.grh + qr;
    return V;
}

template <bool RES, bool LEAN, typename T>
__device__ void bwd_body(const UArgs<T>& a, const UInst& I, int b, const Plan<T>& P, int rank,
                         int C) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int m = I.m, n = I.n;
    const BwdVec<T> V = bwd_vec<LEAN>(a, P.vec);
    const T tau = a.tau[b], sigma = a.sigma[b];
    const T kappa = T(1) / (T(1) + T(2) * a.ridge * tau);
    const T isigma = u_recip(sigma);
    const T go = a.gobj ? a.gobj[b] : T(0);
    T* gax = RES ? P.gax : a.gax + I.nz0;
    // adjoints of the outputs; the objective adds c + 2 ridge x_K to x's
    // adjoint and x_K to c's gradient
    for (int l = wp; l < P.col.slices; l += nw) {
        const int q = 32 * l + lane, j = P.col.id[q];
        V.gl[q] = V.gu[q] = T(0);
        if (j == 0xffff) {
            if constexpr (!LEAN) V.c[q] = V.lo[q] = V.hi[q] = T(0);
            V.xh[q] = V.gc[q] = T(0);
            continue;
        }
        const long long gj = I.c0 + j;
        const T xk = a.xK[gj];
        if constexpr (!LEAN) {
            V.c[q] = a.c[gj];
            V.lo[q] = a.cl[gj];
            V.hi[q] = a.cu[gj];
        }
        V.xh[q] = (a.gx ? a.gx[gj] : T(0)) + go * (a.c[gj] + T(2) * a.ridge * xk);
        V.gc[q] = go * xk;
    }
    for (int l = wp; l < P.row.slices; l += nw) {
        const int q = 32 * l + lane, i = P.row.id[q];
        if constexpr (!LEAN) {
            V.rl[q] = i == 0xffff ? T(0) : a.rmin[I.r0 + i];
            V.rh[q] = i == 0xffff ? T(0) : a.rmax[I.r0 + i];
        }
        V.yh[q] = i != 0xffff && a.gy ? a.gy[I.r0 + i] : T(0);
        V.grl[q] = V.grh[q] = T(0);
        if constexpr (!RES) {
            const int len = P.row.len[q], p0 = len > 0 ? P.row.ptr[i] : 0;
            for (int k = 0; k < len; ++k) gax[p0 + k] = T(0);
        }
    }
    const T* ck = a.ckpt + a.nck * (I.c0 + I.r0);
    // a step's records: x_bar and y_k, and the clamp outcomes, in the order
    // of the global slices (this CTA's own only)
    T* seg = a.seg + (long long)a.ck * (I.c0 + I.r0);
    unsigned char* segf = a.segf + (long long)a.ck * (I.c0 + I.r0);
    const int nseg = (a.K + a.ck - 1) / a.ck;
    auto costs = [&](int q, int j, T& c, T& l0, T& h0) {  // of column j at q
        if constexpr (!LEAN) {
            c = V.c[q];
            l0 = V.lo[q];
            h0 = V.hi[q];
        } else {
            c = l0 = h0 = T(0);
            if (j == 0xffff) return;
            c = a.c[I.c0 + j];
            l0 = a.cl[I.c0 + j];
            h0 = a.cu[I.c0 + j];
        }
    };
    auto bounds = [&](int q, int i, T& l0, T& h0) {  // of row i at q
        if constexpr (!LEAN) {
            l0 = V.rl[q];
            h0 = V.rh[q];
        } else {
            l0 = h0 = T(0);
            if (i == 0xffff) return;
            l0 = a.rmin[I.r0 + i];
            h0 = a.rmax[I.r0 + i];
        }
    };
    auto pos = [&](int l) { return 32 * u_slice(l, rank, C) + lane; };
    for (int s = nseg - 1; s >= 0; --s) {
        const int k0 = s * a.ck, k1 = min(a.K, k0 + a.ck);
        const T* slot = ck + (long long)s * (n + m);
        u_sync(C);  // the last segment's reverse steps are done with the copies
        for (int l = wp; l < P.col.slices; l += nw) {
            const int q = 32 * l + lane, j = P.col.id[q];
            V.x[q] = j == 0xffff ? T(0) : slot[j];
        }
        for (int l = wp; l < P.row.slices; l += nw) {
            const int q = 32 * l + lane, i = P.row.id[q];
            bcast(V.y + P.row.first + q, i == 0xffff ? T(0) : slot[n + i], C);
        }
        u_sync(C);
        // replay: keep x_bar_k, y_k and the clamp outcomes of every step
        for (int k = k0; k < k1; ++k) {
            T* sk = seg + (long long)(k - k0) * (n + m);
            unsigned char* fk = segf + (long long)(k - k0) * (n + m);
            // a warp's last slice is recorded past the barrier: a cluster
            // barrier waits for the global stores made before it
            T xb = T(0), yv = T(0);
            int at = -1, f = 0;
            for (int l = wp; l < P.col.slices; l += nw) {
                if (at >= 0) {
                    sk[at] = xb;
                    fk[at] = (unsigned char)f;
                }
                const int q = 32 * l + lane, j = P.col.id[q];
                T c, l0, h0;
                costs(q, j, c, l0, h0);
                f = fwd_col<RES>(P, l, q, V.x, c, l0, h0, V.xb, V.y, tau, kappa, C, xb);
                at = j != 0xffff ? pos(l) : -1;
            }
            u_sync(C);
            if (at >= 0) {
                sk[at] = xb;
                fk[at] = (unsigned char)f;
            }
            at = -1;
            for (int l = wp; l < P.row.slices; l += nw) {
                if (at >= 0) {
                    sk[at] = yv;
                    fk[at] = (unsigned char)f;
                }
                const int q = 32 * l + lane, i = P.row.id[q];
                yv = V.y[P.row.first + q];
                T l0, h0;
                bounds(q, i, l0, h0);
                f = fwd_row<RES>(P, l, q, l0, h0, V.xb, V.y, yv, sigma, isigma, C);
                at = i != 0xffff ? n + pos(l) : -1;
            }
            u_sync(C);
            if (at >= 0) {
                sk[at] = yv;
                fk[at] = (unsigned char)f;
            }
        }
        // dual prox y+ = t - sigma clamp(t / sigma): dy+/dt = 1 where the
        // clamp is active, 0 inside; -sigma to the active bound
        auto dual = [&](int q, int f, T yv) {
            const T tv = f ? yv : T(0);
            if (f == 1) V.grl[q] -= sigma * yv;
            if (f == 2) V.grh[q] -= sigma * yv;
            V.th[q] = tv;
            bcast(V.zh + P.row.first + q, sigma * tv, C);
        };
        {
            const unsigned char* fk = segf + (long long)(k1 - 1 - k0) * (n + m);
            for (int l = wp; l < P.row.slices; l += nw) {
                const int q = 32 * l + lane, i = P.row.id[q];
                dual(q, i == 0xffff ? 0 : fk[n + pos(l)], V.yh[q]);
            }
        }
        // reverse steps k1-1 .. k0; a row pass ends a step and begins the next
        for (int k = k1 - 1; k >= k0; --k) {
            const T* sk = seg + (long long)(k - k0) * (n + m);
            const unsigned char* fk = segf + (long long)(k - k0) * (n + m);
            const unsigned char* fp = fk - (n + m);
            // the records of the warp's first slices, loaded ahead
            T yk0 = T(0), xb0 = T(0);
            int f0 = 0, fc0 = 0;
            if (wp < P.col.slices && P.col.id[32 * wp + lane] != 0xffff) {
                xb0 = sk[pos(wp)];
                fc0 = fk[pos(wp)];
            }
            if (wp < P.row.slices && P.row.id[32 * wp + lane] != 0xffff) {
                yk0 = sk[n + pos(wp)];
                if (k > k0) f0 = fp[n + pos(wp)];
            }
            u_sync(C);
            // A^T of the dual adjoint; primal prox and the extrapolation
            for (int l = wp; l < P.col.slices; l += nw) {
                const int q = 32 * l + lane, j = P.col.id[q];
                T xb = xb0;
                int f = fc0;
                if (l != wp && j != 0xffff) {
                    xb = sk[pos(l)];
                    f = fk[pos(l)];
                }
                const T xhv = V.xh[q];
                const T d = row_dot<RES, T, T>(P.col, l, q, V.zh, T(0));
                const T xt = fma(T(2), d, xhv);
                const T vh = f ? T(0) : xt;
                if (f == 1) V.gl[q] += xt;
                if (f == 2) V.gu[q] += xt;
                const T g = -kappa * tau * vh;
                V.xh[q] = fma(kappa, vh, -d);
                V.gc[q] += g;
                typename Pair<T>::type pr;
                pr.x = g;
                pr.y = xb;
                bcast(V.gp + P.col.first + q, pr, C);
            }
            u_sync(C);
            // A of the cost adjoint -> adjoint of y_k; A's value gradient
            // (from A x_bar and from A^T y) by the row that owns the entry
            for (int l = wp; l < P.row.slices; l += nw) {
                const int q = 32 * l + lane, i = P.row.id[q], len = P.row.len[q];
                T yk = yk0;
                int f = f0;
                if (l != wp && i != 0xffff) {
                    yk = sk[n + pos(l)];
                    if (k > k0) f = fp[n + pos(l)];
                }
                const T zi = sigma * V.th[q];
                T s2 = T(0);
                auto entry = [&](T v, T ga, const typename Pair<T>::type& g) {
                    s2 = fma(v, g.x, s2);
                    return fma(yk, g.x, fma(zi, g.y, ga));
                };
                if constexpr (RES) {
                    const int longest = __shfl_sync(kFull, len, 0);
                    const int shortest = __shfl_sync(kFull, len, 31);
                    int off = P.row.base[l] + lane, e = 0;
                    for (; e + 4 <= shortest; e += 4, off += 128) {
                        T v[4], ga[4];
                        typename Pair<T>::type g[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            v[u] = P.row.val[off + 32 * u];
                            ga[u] = gax[off + 32 * u];
                            g[u] = V.gp[P.row.idx[off + 32 * u]];
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) gax[off + 32 * u] = entry(v[u], ga[u], g[u]);
                    }
                    for (; e < longest; e += 2) {
                        T v[2], ga[2];
                        int at[2];
                        typename Pair<T>::type g[2];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const bool on = e + u < len;
                            at[u] = off;
                            off += __popc(__ballot_sync(kFull, on));
                            if (on) {
                                v[u] = P.row.val[at[u]];
                                ga[u] = gax[at[u]];
                                g[u] = V.gp[P.row.idx[at[u]]];
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if (sizeof(T) == 8 && e + u >= longest) break;
                            if (e + u < len) gax[at[u]] = entry(v[u], ga[u], g[u]);
                        }
                    }
                } else {
                    const int p0 = len > 0 ? P.row.ptr[i] : 0;
                    for (int e = p0; e < p0 + len; ++e)
                        gax[e] = entry(P.row.gval[e], gax[e], V.gp[P.row.gpos[P.row.gidx[e]]]);
                    __syncwarp();
                }
                const T yv = V.th[q] + s2;
                V.yh[q] = yv;
                if (k > k0) dual(q, f, yv);
            }
        }
    }
    // x0 = clamp(0, cl, cu)
    for (int l = wp; l < P.col.slices; l += nw) {
        const int q = 32 * l + lane, j = P.col.id[q];
        if (j == 0xffff) continue;
        const long long gj = I.c0 + j;
        T l0 = V.gl[q], u0 = V.gu[q], c, lo, hi;
        costs(q, j, c, lo, hi);
        if (T(0) < lo) l0 += V.xh[q];
        else if (T(0) > hi) u0 += V.xh[q];
        a.gc[gj] = V.gc[q];
        a.gcl[gj] = l0;
        a.gcu[gj] = u0;
    }
    for (int l = wp; l < P.row.slices; l += nw) {
        const int q = 32 * l + lane, i = P.row.id[q], len = P.row.len[q];
        if (i != 0xffff) {
            a.grmin[I.r0 + i] = V.grl[q];
            a.grmax[I.r0 + i] = V.grh[q];
        }
        if constexpr (RES) {
            T* out = a.gax + I.nz0 + (len > 0 ? P.row.ptr[i] : 0);
            const int longest = __shfl_sync(kFull, len, 0);
            int off = P.row.base[l];
            for (int k = 0; k < longest; ++k) {
                const bool on = k < len;
                if (on) out[k] = gax[off + lane];
                off += __popc(__ballot_sync(kFull, on));
            }
        }
    }
    u_sync(C);  // no CTA leaves while another may still write its copies
}

// The same bounds; the gradient of A's values, read and written once per
// entry and step, and the pairs' gathers (64 bits each) are the largest share.
// As above: 1.69 ms against 2.6.
// OCC: CTAs of kLT threads per SM that it is compiled for, 1: 128 registers, 2:
// 64 (in FP64 412 bytes spilled). 200 iterations of 1,024 LPs of 150 x 300
// (2,250 entries): FP32 5.8 ms with the first, 3.7 with the second, FP64 16.6
// and 13.2; 304 of 500 x 1,000 (one CTA per SM either way) 3.6 and 3.9, 15.3 and
// 16.5. plan() takes the second where it lets more CTAs reside.
template <typename T, int OCC>
__global__ void __launch_bounds__(kLT, OCC) k_unroll_bwd(UArgs<T> a) {
    extern __shared__ __align__(16) unsigned char u_smem[];
    const int rank = u_rank(), b = u_instance();
    const UInst I = uinst(a, b);
    const int C = u_ctas(a, I);
    if (rank >= C) return;
    const Plan<T> P = stage<T, true, false>(a, I, b, u_smem, rank, C);
    if (P.resident && !a.lean) bwd_body<true, false>(a, I, b, P, rank, C);
    else if (P.resident) bwd_body<true, true>(a, I, b, P, rank, C);
    else if (!a.lean) bwd_body<false, false>(a, I, b, P, rank, C);
    else bwd_body<false, true>(a, I, b, P, rank, C);
}

// ------------------------------------------------------------------ steps
// eta = 0.9 / ||A||_2 by 100 products of A^T A from the uniform vector, in
// FP64. A product scales its input by the power of two that brings the last
// one's largest entry near 1 (exact, from an integer maximum of the entries'
// high words) instead of dividing by its norm, so that an iteration has two
// barriers and no FP64 work but the products; lambda is the quotient of the
// last two norms.
template <bool RES, typename T>
__device__ void steps_body(const UArgs<T>& a, const UInst& I, int b, const Plan<T>& P, int rank,
                           int C, unsigned* s_max, double* red) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n = I.n;
    double* v = reinterpret_cast<double*>(P.vec);
    double* w = v + a.ngc;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const double v0 = 1.0 / sqrt((double)n);
    for (int j = threadIdx.x; j < a.ngc; j += blockDim.x) v[j] = v0;
    for (int i = threadIdx.x; i < a.ngr; i += blockDim.x) w[i] = 0.0;
    constexpr int kProducts = 100;
    double nrm[2] = {1.0, 1.0};  // ||v|| before and after the last product
    double scale = 1.0;
    u_sync(C);
    for (int it = 0; it < kProducts; ++it) {
        for (int l = wp; l < P.row.slices; l += nw) {
            const int q = 32 * l + lane;
            const double s = row_dot<RES, T, double>(P.row, l, q, v, 0.0);
            bcast(w + P.row.first + q, s * scale, C);
        }
        // the slot two products ahead is free: its readers are behind a barrier
        if (threadIdx.x == 0) s_max[(it + 1) % 3] = 0u;
        u_sync(C);
        unsigned mx = 0;
        for (int l = wp; l < P.col.slices; l += nw) {
            const int q = 32 * l + lane;
            const double s = row_dot<RES, T, double>(P.col, l, q, w, 0.0);
            bcast(v + P.col.first + q, s, C);
            mx = max(mx, (unsigned)__double2hiint(s) & 0x7fffffffu);
        }
        mx = __reduce_max_sync(kFull, mx);
        if (lane == 0)
            for (int r = 0; r < C; ++r) atomicMax(cl.map_shared_rank(&s_max[it % 3], r), mx);
        u_sync(C);
        const unsigned top = *(volatile unsigned*)&s_max[it % 3];
        if (it >= kProducts - 2) {
            // the norm of this CTA's copy, summed in index order in the
            // shape of kLW warps, whatever the launch
            for (int k = wp; k < kLW; k += nw) {
                double s = 0.0;
                for (int j = 32 * k + lane; j < n; j += kLT) {
                    const double u = v[P.row.gpos[j]];
                    s = fma(u, u, s);
                }
                s = warp_sum(s);
                if (lane == 0) red[k] = s;
            }
            __syncthreads();
            double s = 0.0;
            for (int k = 0; k < kLW; ++k) s += red[k];
            // this product's input was `scale` times the last one's output
            nrm[0] = nrm[1] * scale;
            nrm[1] = sqrt(s);
            __syncthreads();
        }
        if (top == 0u || top >= 0x7ff00000u) {  // nothing left, or not finite
            nrm[0] = 1.0;
            nrm[1] = top == 0u ? 0.0 : CUDART_INF;
            break;
        }
        const int ex = (int)(top >> 20) - 1023;  // 2^-ex, kept in the normal range
        scale = __hiloint2double((1023 - min(max(ex, -1000), 1000)) << 20, 0);
    }
    if (threadIdx.x == 0 && rank == 0) {
        const double lam = nrm[1] / nrm[0];
        const double eta = (lam > 0.0 && isfinite(lam)) ? 0.9 / sqrt(lam) : 1.0;
        a.tau_o[b] = (T)(eta / (double)a.omega);
        a.sigma_o[b] = (T)(eta * (double)a.omega);
    }
    u_sync(C);
}

// Bound by the FP64 pipe (74 % busy): 152 LPs of 500 x 1,000 0.90 ms, 2.6 ms
// from global memory with norms and divisions in every product.
template <typename T>
__global__ void __launch_bounds__(kLT) k_unroll_steps(UArgs<T> a) {
    extern __shared__ __align__(16) unsigned char u_smem[];
    __shared__ unsigned s_max[3];
    __shared__ double red[kLW];
    const int rank = u_rank(), b = u_instance();
    const UInst I = uinst(a, b);
    const int C = u_ctas(a, I);
    if (rank >= C) return;
    if (threadIdx.x < 3) s_max[threadIdx.x] = 0u;
    const Plan<T> P = stage<T, false, true>(a, I, b, u_smem, rank, C);
    if (P.resident) steps_body<true>(a, I, b, P, rank, C, s_max, red);
    else steps_body<false>(a, I, b, P, rank, C, s_max, red);
}

int fail_cuda(cudaError_t e) {
    char buf[256];
    std::snprintf(buf, sizeof(buf), "CUDA error in PDHG unrolled layer: %s", cudaGetErrorString(e));
    return igx_set_error(IGAOS_PDHG_ERR_CUDA, buf);
}

int check_layout(const igaos_pdhg_unrolled_layout* L) {
    if (!L) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL layout");
    if (L->count <= 0) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "count must be positive");
    if (L->precision != IGAOS_PDHG_FP32 && L->precision != IGAOS_PDHG_FP64)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "precision must be IGAOS_PDHG_FP32 or IGAOS_PDHG_FP64");
    if (L->iterations < 1 || L->checkpoint < 1)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "iterations and checkpoint must be >= 1");
    if (!(L->ridge >= 0.0) || !std::isfinite(L->ridge))
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "ridge must be finite and >= 0");
    if (L->max_m < 1 || L->max_n < 1 || L->total_m < L->max_m || L->total_n < L->max_n ||
        L->max_nnz < 0 || L->total_nnz < L->max_nnz)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "inconsistent layout sizes");
    if (!L->row_off || !L->col_off || !L->nz_off || !L->ap || !L->ai || !L->cp || !L->ci ||
        !L->cperm)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL layout array");
    return IGAOS_PDHG_OK;
}

size_t elem_size(const igaos_pdhg_unrolled_layout* L) {
    return L->precision == IGAOS_PDHG_FP64 ? sizeof(double) : sizeof(float);
}

// The vectors' shared memory that bounds the instances the layer takes.
size_t vec_bwd(const igaos_pdhg_unrolled_layout* L) {
    return (size_t)(7 * (size_t)L->max_n + 6 * (size_t)L->max_m) * elem_size(L);
}

constexpr int kMaxDevices = 16;
constexpr int kClusterPerSm = 2;  // CTAs of a cluster launch per SM at most

struct Device {
    int index, optin, sms;
};
int device_info(Device* d) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    d->index = dev;
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&d->optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&d->sms, cudaDevAttrMultiProcessorCount, dev);
    return e == cudaSuccess ? IGAOS_PDHG_OK : fail_cuda(e);
}

template <typename T>
UArgs<T> base_args(const igaos_pdhg_unrolled_layout* L) {
    UArgs<T> a{};
    a.K = L->iterations;
    a.ck = L->checkpoint;
    a.ridge = (T)L->ridge;
    a.row_off = L->row_off;
    a.col_off = L->col_off;
    a.nz_off = L->nz_off;
    a.ap = L->ap;
    a.ai = L->ai;
    a.cp = L->cp;
    a.ci = L->ci;
    a.cperm = L->cperm;
    a.nck = (L->iterations + L->checkpoint - 1) / L->checkpoint;
    return a;
}

// static shared memory of the layer kernels stays below this
constexpr size_t kStaticSmem = 1024;

// Lets a kernel's launches take any size up to the device's limit. The
// attribute belongs to the kernel, not to a launch: set to one launch's size, it
// made another host thread's larger launch fail.
template <typename K>
cudaError_t allow_smem(K kernel, const Device& dev) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                dev.optin - (int)kStaticSmem);
}

int too_large(size_t need, int optin) {
    char buf[192];
    std::snprintf(buf, sizeof(buf),
                  "instance too large for the unrolled layer: needs %zu bytes of shared memory "
                  "per CTA, device allows %d", need, optin);
    return igx_set_error(IGAOS_PDHG_ERR_INVALID, buf);
}

enum Pass { kSteps, kForward, kBackward };
constexpr int kVariants = 2;  // of a pass's kernel, by registers

template <typename T>
struct Kernels {
    Pass pass;
    void (*fn[kVariants])(UArgs<T>);  // the second one may be missing
};

struct Launch {
    int C, threads, variant;
    int per_sm;  // CTAs that one SM holds
    size_t smem;
};

cudaLaunchConfig_t cluster_config(cudaLaunchAttribute* at, unsigned grid, int C, int threads,
                                  size_t smem, cudaStream_t st) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = C;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// CTAs of so many warps that a kernel's registers let one SM hold; asked once
// for each kernel and number of warps.
template <typename T>
int by_registers(const Kernels<T>& k, int variant, const Device& dev, int warps) {
    static std::atomic<int> known[kMaxDevices][3][kVariants][kLW + 1];
    std::atomic<int>* slot =
        dev.index < kMaxDevices ? &known[dev.index][k.pass][variant][warps] : nullptr;
    if (slot && slot->load() > 0) return slot->load();
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void*)k.fn[variant], 32 * warps, 0) !=
        cudaSuccess)
        cudaGetLastError();
    n = std::max(1, n);
    if (slot) slot->store(n);
    return n;
}

// Dynamic shared memory that leaves room for per_sm CTAs on an SM.
size_t smem_at(const Device& dev, int per_sm) {
    const size_t room = (size_t)dev.optin - kStaticSmem, sm = (size_t)dev.optin + 1024;
    return std::min(room, sm / per_sm - 1024 - kStaticSmem) & ~(size_t)15;
}

// Clusters of C CTAs that are resident at once at `per_sm` CTAs per SM (the
// GPU's processing clusters hold no whole number of them); asked once for each
// kernel, C, per_sm and number of warps, at the shared memory of smem_at.
template <typename T>
int resident_clusters(const Kernels<T>& k, int variant, const Device& dev, int C, int per_sm,
                      int warps) {
    if (C == 1) return dev.sms * per_sm;
    static std::atomic<int> known[kMaxDevices][3][kVariants][kMaxCluster + 1][kClusterPerSm + 1][kLW + 1];
    std::atomic<int>* slot =
        dev.index < kMaxDevices ? &known[dev.index][k.pass][variant][C][per_sm][warps] : nullptr;
    if (slot && slot->load() > 0) return slot->load();
    int n = 0;
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = cluster_config(at, C, C, 32 * warps, smem_at(dev, per_sm), nullptr);
    if (allow_smem(k.fn[variant], dev) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, (const void*)k.fn[variant], &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    if (slot && n > 0) slot->store(n);
    return n;
}

// Cluster size, threads and shared memory of a pass. One CTA holds a small
// instance; a larger one is spread over up to kMaxCluster CTAs when it does
// not fit one, or when that leaves fewer SMs idle. The time of an iteration is
// modelled as the products on the busiest SM plus a fixed cost per barrier
// (the latency of a phase), times the rounds the batch takes; the figures were
// fitted to measured passes (500 x 1,000 LPs of 10,000 entries): FP32 256 of
// them on one CTA each 23.6 ms, on two 34.6; FP64 96 of them 11.3 ms on two or
// three, 10.4 on five; 96 of up to 1,300 rows (67,000 entries) 8 ms on seven,
// 32 ms where the largest are read from global memory.
// One-CTA instances stand on an SM as often as registers, threads and the
// shared memory they need allow: with at most two, each asking for half of the
// SM's memory, 200 iterations of 1,024 LPs of 60 x 120 took 1.1 ms forward and
// 3.1 backward in FP32, now 0.50 and 1.5; 3.4 and 8.0 in FP64, now 1.7 and 5.7.
// A backward that does not quite fit one CTA leaves costs and bounds in global
// memory (lean): 1,024 FP64 LPs of 150 x 300 with 7,000 entries 58 ms on two
// CTAs each, 30 on one.
template <typename T>
Launch plan(const Kernels<T>& k, const igaos_pdhg_unrolled_layout* L, const Device& dev,
            UArgs<T>& a) {
    const Pass pass = k.pass;
    const size_t es = sizeof(T), room = (size_t)dev.optin - kStaticSmem;
    const int sc = (L->max_n + 31) / 32, sr = (L->max_m + 31) / 32;
    const double nnz = (double)L->max_nnz;
    const bool wide = es == 8 || pass == kSteps;
    // instances of the largest one's size that make up the batch's work
    const double count = std::min((double)L->count,
                                  1.0 + (double)L->total_nnz / std::max(1.0, nnz));
    const double products = (pass == kBackward ? 6.0 : 2.0) * nnz * (wide ? 0.38e-3 : 0.1e-3);
    const double barriers = pass == kBackward ? 4.0 : 2.0;
    Launch best{};
    double best_us = 0.0;
    for (int C = 1; C <= kMaxCluster; ++C) {
        if (best.C == 1 && nnz < 4096) break;  // latency-bound on one CTA
        bool lean = false;
        const int lc = (sc + C - 1) / C, lr = (sr + C - 1) / C;
        auto vectors = [&]() {
            const size_t v = pass == kSteps     ? (size_t)32 * C * (lc + lr) * sizeof(double)
                             : pass == kForward ? fwd_elems<T>(lc, lr, C) * es
                                                : bwd_elems<T>(lc, lr, C, lean) * es;
            return (std::max(v, scratch_bytes(L->max_m, L->max_n)) + 15) & ~(size_t)15;
        };
        size_t vec = vectors();
        size_t fixed = vec + meta_bytes(L->max_m, L->max_n, lc, lr);
        if (fixed + 64 > room) continue;
        // entries of the largest share: slices are dealt evenly, by length
        const double pc = sc ? (double)lc / sc : 0.0, pr = sr ? (double)lr / sr : 0.0;
        double need = nnz * (pc * (es + 2) + pr * (es + 2 + (pass == kBackward ? es : 0)));
        if (C > 1) need = 1.02 * need + 1024;
        if (pass == kBackward && C == 1 && fixed + (size_t)need + 64 > room) {
            lean = true;
            const size_t less = vectors();
            lean = fixed - (vec - less) + (size_t)need + 64 <= room;
            if (lean) {
                fixed -= vec - less;
                vec = less;
            }
        }
        const size_t want = fixed + (size_t)need + 64;
        const bool fits = want <= room;
        const int warps = std::min(kLW, std::max(4, std::max(lc, lr)));
        const size_t sm_bytes = (size_t)dev.optin + 1024;
        const int by_smem = fits ? (int)(sm_bytes / (want + kStaticSmem + 1024)) : 1;
        const int most = std::min(by_smem, C == 1 ? 64 / warps : kClusterPerSm);
        int variant = 0, per_sm = std::max(1, std::min(most, by_registers(k, 0, dev, warps)));
        if (k.fn[1] && count * C > (double)per_sm * dev.sms) {
            const int more = std::min(most, by_registers(k, 1, dev, warps));
            if (more > per_sm) {
                variant = 1;
                per_sm = more;
            }
        }
        // a cluster asks for all that this residency leaves: shares of uneven
        // rows fit better
        const size_t smem = C == 1 && fits ? (want + 15) & ~(size_t)15 : smem_at(dev, per_sm);
        const int slots = resident_clusters(k, variant, dev, C, per_sm, warps);
        if (slots < 1) continue;
        const double rounds = std::ceil(count / slots);
        const double used = std::max(1.0, std::min((double)per_sm, std::ceil(count * C / dev.sms)));
        // (too few warps on an SM leave the FP64 units' latency in the open)
        const double open = wide ? std::max(1.0, 8.0 / (used * warps)) : 1.0;
        const double us = rounds * (used * open * products * 0.5 * (pc + pr) * (fits ? 1.0 : 8.0) +
                                    barriers * (wide ? 2.0 : C == 1 ? 0.6 : 1.25));
        if (best.C == 0 || us < 0.95 * best_us) {
            best = Launch{C, 32 * warps, variant, per_sm, smem};
            best_us = us;
            a.lc = lc;
            a.lr = lr;
            a.ngc = 32 * lc * C;
            a.ngr = 32 * lr * C;
            a.per_cta = std::max(1, (int)((L->max_nnz + C - 1) / C));
            a.lean = lean;
            a.vec_bytes = (int)vec;
            a.ent_bytes = (int)(smem - fixed);
        }
    }
    a.max_m = L->max_m;
    a.max_n = L->max_n;
    return best;
}

template <typename T>
Kernels<T> kernels(Pass pass) {
    return pass == kSteps     ? Kernels<T>{pass, {k_unroll_steps<T>, nullptr}}
           : pass == kForward ? Kernels<T>{pass, {k_unroll_fwd<T>, nullptr}}
                              : Kernels<T>{pass, {k_unroll_bwd<T, 1>, k_unroll_bwd<T, 2>}};
}

// One cluster of C CTAs per instance.
template <typename T>
cudaError_t launch(const Kernels<T>& k, const Launch& l, int count, const UArgs<T>& a,
                   const Device& dev, cudaStream_t st) {
    if (l.C == 0) return cudaErrorInvalidConfiguration;
    void (*kernel)(UArgs<T>) = k.fn[l.variant];
    const cudaError_t e = allow_smem(kernel, dev);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg =
        cluster_config(at, (unsigned)count * l.C, l.C, l.threads, l.smem, st);
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <typename T>
int run_steps(const igaos_pdhg_unrolled_layout* L, const void* ax, double omega, void* tau,
              void* sigma, cudaStream_t st, const Device& dev) {
    UArgs<T> a = base_args<T>(L);
    a.ax = static_cast<const T*>(ax);
    a.tau_o = static_cast<T*>(tau);
    a.sigma_o = static_cast<T*>(sigma);
    a.omega = (T)omega;
    const Kernels<T> k = kernels<T>(kSteps);
    const Launch l = plan<T>(k, L, dev, a);
    const cudaError_t e = launch<T>(k, l, L->count, a, dev, st);
    return e == cudaSuccess ? igx_set_error(IGAOS_PDHG_OK, "") : fail_cuda(e);
}

template <typename T>
int run_forward(const igaos_pdhg_unrolled_layout* L, const void* c, const void* cl,
                const void* cu, const void* rmin, const void* rmax, const void* ax,
                const void* tau, const void* sigma, void* x, void* y, void* obj, void* ckpt,
                cudaStream_t st, const Device& dev) {
    UArgs<T> a = base_args<T>(L);
    a.c = static_cast<const T*>(c);
    a.cl = static_cast<const T*>(cl);
    a.cu = static_cast<const T*>(cu);
    a.rmin = static_cast<const T*>(rmin);
    a.rmax = static_cast<const T*>(rmax);
    a.ax = static_cast<const T*>(ax);
    a.tau = static_cast<const T*>(tau);
    a.sigma = static_cast<const T*>(sigma);
    a.x = static_cast<T*>(x);
    a.y = static_cast<T*>(y);
    a.obj = static_cast<T*>(obj);
    a.ckpt = static_cast<T*>(ckpt);
    const Kernels<T> k = kernels<T>(kForward);
    const Launch l = plan<T>(k, L, dev, a);
    const cudaError_t e = launch<T>(k, l, L->count, a, dev, st);
    return e == cudaSuccess ? igx_set_error(IGAOS_PDHG_OK, "") : fail_cuda(e);
}

template <typename T>
int run_backward(const igaos_pdhg_unrolled_layout* L, const void* c, const void* cl,
                 const void* cu, const void* rmin, const void* rmax, const void* ax,
                 const void* tau, const void* sigma, const void* ckpt, const void* x,
                 const void* gx, const void* gy, const void* gobj, void* gc, void* gcl,
                 void* gcu, void* grmin, void* grmax, void* gax, void* work, cudaStream_t st,
                 const Device& dev) {
    UArgs<T> a = base_args<T>(L);
    a.c = static_cast<const T*>(c);
    a.cl = static_cast<const T*>(cl);
    a.cu = static_cast<const T*>(cu);
    a.rmin = static_cast<const T*>(rmin);
    a.rmax = static_cast<const T*>(rmax);
    a.ax = static_cast<const T*>(ax);
    a.tau = static_cast<const T*>(tau);
    a.sigma = static_cast<const T*>(sigma);
    a.ckpt = const_cast<T*>(static_cast<const T*>(ckpt));
    a.xK = static_cast<const T*>(x);
    a.gx = static_cast<const T*>(gx);
    a.gy = static_cast<const T*>(gy);
    a.gobj = static_cast<const T*>(gobj);
    a.gc = static_cast<T*>(gc);
    a.gcl = static_cast<T*>(gcl);
    a.gcu = static_cast<T*>(gcu);
    a.grmin = static_cast<T*>(grmin);
    a.grmax = static_cast<T*>(grmax);
    a.gax = static_cast<T*>(gax);
    const long long per = (long long)L->checkpoint * (L->total_n + L->total_m);
    const long long vb = (per * (long long)sizeof(T) + 255) / 256 * 256;
    a.seg = static_cast<T*>(work);
    a.segf = static_cast<unsigned char*>(work) + vb;
    const Kernels<T> k = kernels<T>(kBackward);
    const Launch l = plan<T>(k, L, dev, a);
    const cudaError_t e = launch<T>(k, l, L->count, a, dev, st);
    return e == cudaSuccess ? igx_set_error(IGAOS_PDHG_OK, "") : fail_cuda(e);
}

// common checks of the three entry points; fills the device's figures
int prepare(const igaos_pdhg_unrolled_layout* L, Device* dev) {
    int rc = check_layout(L);
    if (rc != IGAOS_PDHG_OK) return rc;
    if ((rc = device_info(dev)) != IGAOS_PDHG_OK) return rc;
    const size_t need = std::max(vec_bwd(L), (size_t)(2 * L->max_n + L->max_m) * sizeof(double));
    if (need + kStaticSmem > (size_t)dev->optin) return too_large(need, dev->optin);
    return IGAOS_PDHG_OK;
}

}  // namespace
}  // namespace igx

extern "C" int64_t igaos_pdhg_unrolled_checkpoint_elems(const igaos_pdhg_unrolled_layout* L) {
    if (igx::check_layout(L) != IGAOS_PDHG_OK) return -1;
    const int64_t nck = (L->iterations + L->checkpoint - 1) / L->checkpoint;
    return nck * (L->total_n + L->total_m);
}

extern "C" int64_t igaos_pdhg_unrolled_workspace_bytes(const igaos_pdhg_unrolled_layout* L) {
    if (igx::check_layout(L) != IGAOS_PDHG_OK) return -1;
    const int64_t per = (int64_t)L->checkpoint * (L->total_n + L->total_m);
    // values, then one clamp-outcome byte per value after a 256-byte boundary
    const int64_t vb = ((per * (int64_t)igx::elem_size(L)) + 255) / 256 * 256;
    return vb + per;
}

// The launch of a pass (0 steps, 1 forward, 2 backward) over a layout: CTAs per
// instance, threads, CTAs per SM, dynamic shared memory, the kernel's variant,
// whether the backward is lean. For tests; not in the public header.
extern "C" int igx_unrolled_plan(const igaos_pdhg_unrolled_layout* L, int pass, int* out) {
    using namespace igx;
    Device dev{};
    const int rc = prepare(L, &dev);
    if (rc != IGAOS_PDHG_OK) return rc;
    if (pass < kSteps || pass > kBackward || !out)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "no such pass");
    auto fill = [&](auto a) {
        using T = std::remove_const_t<std::remove_pointer_t<decltype(a.ax)>>;
        const Launch l = plan<T>(kernels<T>((Pass)pass), L, dev, a);
        out[0] = l.C;
        out[1] = l.threads;
        out[2] = l.per_sm;
        out[3] = (int)l.smem;
        out[4] = l.variant;
        out[5] = a.lean;
    };
    if (L->precision == IGAOS_PDHG_FP64) fill(base_args<double>(L));
    else fill(base_args<float>(L));
    return IGAOS_PDHG_OK;
}

extern "C" int igaos_pdhg_unrolled_steps(const igaos_pdhg_unrolled_layout* L, const void* ax,
                                         double omega, void* tau, void* sigma, void* stream) {
    using namespace igx;
    Device dev{};
    int rc = prepare(L, &dev);
    if (rc != IGAOS_PDHG_OK) return rc;
    if (!ax || !tau || !sigma) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL device pointer");
    if (!(omega > 0.0) || !std::isfinite(omega))
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "omega must be positive and finite");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return L->precision == IGAOS_PDHG_FP64 ? run_steps<double>(L, ax, omega, tau, sigma, st, dev)
                                           : run_steps<float>(L, ax, omega, tau, sigma, st, dev);
}

extern "C" int igaos_pdhg_unrolled_forward(const igaos_pdhg_unrolled_layout* L, const void* c,
                                           const void* cl, const void* cu, const void* rmin,
                                           const void* rmax, const void* ax, const void* tau,
                                           const void* sigma, void* x, void* y, void* obj,
                                           void* ckpt, void* stream) {
    using namespace igx;
    Device dev{};
    int rc = prepare(L, &dev);
    if (rc != IGAOS_PDHG_OK) return rc;
    if (!c || !cl || !cu || !rmin || !rmax || !ax || !tau || !sigma || !x || !y || !obj || !ckpt)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL device pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return L->precision == IGAOS_PDHG_FP64
               ? run_forward<double>(L, c, cl, cu, rmin, rmax, ax, tau, sigma, x, y, obj, ckpt,
                                     st, dev)
               : run_forward<float>(L, c, cl, cu, rmin, rmax, ax, tau, sigma, x, y, obj, ckpt,
                                    st, dev);
}

extern "C" int igaos_pdhg_unrolled_backward(const igaos_pdhg_unrolled_layout* L, const void* c,
                                            const void* cl, const void* cu, const void* rmin,
                                            const void* rmax, const void* ax, const void* tau,
                                            const void* sigma, const void* ckpt, const void* x,
                                            const void* gx, const void* gy, const void* gobj,
                                            void* gc, void* gcl, void* gcu, void* grmin,
                                            void* grmax, void* gax, void* work, void* stream) {
    using namespace igx;
    Device dev{};
    int rc = prepare(L, &dev);
    if (rc != IGAOS_PDHG_OK) return rc;
    if (!c || !cl || !cu || !rmin || !rmax || !ax || !tau || !sigma || !ckpt || !x || !gc ||
        !gcl || !gcu || !grmin || !grmax || !gax || !work)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL device pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return L->precision == IGAOS_PDHG_FP64
               ? run_backward<double>(L, c, cl, cu, rmin, rmax, ax, tau, sigma, ckpt, x, gx, gy,
                                      gobj, gc, gcl, gcu, grmin, grmax, gax, work, st, dev)
               : run_backward<float>(L, c, cl, cu, rmin, rmax, ax, tau, sigma, ckpt, x, gx, gy,
                                     gobj, gc, gcl, gcu, grmin, grmax, gax, work, st, dev);
}
