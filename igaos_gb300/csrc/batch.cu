// Batched PDHG: thousands of independent LPs of uneven sizes solved in one
// persistent launch (igaos_pdhg_solve_batch).
//
// Each CTA takes instances from a work queue (largest first, an atomic
// counter; no CTA waits on another) and runs one LP to the end on its own:
// deterministic CSC build, Ruiz equilibration (src/pdhg/pdhg.cu:472-492),
// power iteration (:605-631), and the reference iteration -- adaptive line
// search (:751-794), averaging (:795-799), KKT checks every `check`
// iterations with the termination test (:835-840), restarts and the
// primal-weight update (:1001-1075) -- with per-instance restart and
// termination. Attempts stream FP32 (compensated row sums); the iterates are
// FP32 deltas from an FP64 anchor that every restart re-sets, with the
// residual data (reduced costs, shifted row bounds and box) formed in FP64
// from the original FP64 values, so the termination metrics -- evaluated in
// FP64 on anchor + delta -- reach FP64-level accuracy. Incumbent/rollback and
// dual repair are not part of this path.
//
// FP32 iterates can stall where FP64 ones do not (one instance of a 4,096-LP
// set needs 255,872 FP32 + refinement iterations against 54,336 in FP64),
// and the launch lasts as long as its slowest instance. So the first
// `handoff_max` instances still running at `handoff_at` iterations stop
// there (a device counter bounds how many), and, with those the launch left
// at max_iterations, the host finishes them in FP64 with the single-LP engine,
// several at once on their own streams and threads.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include "device.cuh"
#include "engine.hpp"

namespace igx {
namespace {

// Threads of a CTA, by class (below). The first kBT at most are workers: one
// owns columns (rows) t, t + kBT, ...; with fewer threads than kBT every column
// has its own, so the per-thread sums of the step's dot products, and their
// merge over warps, do not depend on the class. Threads past kBT take part in
// the products alone, and the last warp takes the step decisions.
constexpr int kBT = 512;
constexpr int kBW = kBT / 32;
constexpr unsigned kFull = 0xffffffffu;

struct BatchDesc {
    int m, n, nnz, mode;  // mode: where the instance is held (kHeld...)
    long long pad_c, pad_r;  // staged entries of the sorted slices, columns and rows
    int long_c, long_r;      // slices laid in steps
    int longer_c, longer_r;  // columns and rows of more than kLongRow entries
    long long ap_off, cp_off, nz_off, row_off, col_off;
    long long base_off;  // slice bases (in units of 32 entries): columns'
                         // (slices + 1), then rows'
    long long out_off;   // kHeldOut, kHeldWide: staged entries in global memory
    long long long_c_at, long_r_at;  // the tables of the slices laid in steps
};

// kHeldWide: everything in global memory. kHeldOut: the matrix too (16-bit
// indices), the gathered vectors in shared memory. kHeldMatrix: the matrix and the
// gathered vectors in shared memory. kHeldAll: the iterates and the residual
// data too.
enum { kHeldWide = 0, kHeldOut = 1, kHeldMatrix = 2, kHeldAll = 3 };

__host__ __device__ inline int slices_of(int rows) { return (rows + 31) / 32; }
// A slice laid in steps: 32, 16, .. 1 lanes wide, step s as deep as the row of
// lane step_lane(s) is long, so that half of its lanes or more hold entries all the
// way. Such slices follow the others (which see them as empty), behind a table
// {slice, first unit} of them; each has a unit for the depths of its steps, then its
// entries, step after step.
constexpr int kSteps = 6;
constexpr int kLongRow = 64;  // entries of a row that one thread walks at most (each_row)
__host__ __device__ inline int step_lane(int s) { return 16 >> s; }
// staged values and 16-bit indices, x_bar, both slots of y, A~ x_bar, the
// slices' bases and the rows' numbers
__host__ __device__ inline size_t matrix_bytes(const BatchDesc& d) {
    const size_t pad = (size_t)d.pad_c + d.pad_r;
    return ((4 * pad + 4 * (size_t)d.n + 12 * (size_t)d.m +
             4 * (size_t)(slices_of(d.n) + slices_of(d.m) + 2) + 2 * pad +
             2 * ((size_t)d.n + d.m)) + 15) & ~(size_t)15;
}
__host__ __device__ inline size_t state_bytes(const BatchDesc& d) {
    return 4 * (9 * (size_t)d.n + 7 * (size_t)d.m);
}

struct BatchOut {
    int status, handed;  // handed: stopped at handoff_at for the FP64 finish
    double objective, pinf, dinf, gap, prow;
    long long iterations, attempts, restarts;
    long long ns;  // device time of the instance (global timer)
};

__device__ __forceinline__ long long global_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr int kFacTab = 1 << 16;  // tabulated 1 - k^-0.3, 1 + k^-0.6

struct BatchArgs {
    int count;           // instances of this launch's class
    const int* order;    // their indices, largest first
    unsigned int* queue;
    const BatchDesc* desc;
    const int *ap, *ai;
    const float* ax;     // original values, FP32 (Ruiz, scaled FP32 copies)
    const double* axd;   // original values, FP64 (anchor residuals)
    const double *c, *cl, *cu, *rmin, *rmax;
    int *cp, *ci, *cnt;
    float *cax, *sax, *scax;
    double* cax64;       // original values in CSC order, FP64
    const int *order_c, *order_r;  // columns and rows by decreasing length
    const int* bases;              // first staged entry of each slice of 32 of them
    const int* longs;              // tables of the slices laid in steps
    float* out_val;                // staged entries of kHeldOut and kHeldWide instances
    int* out_idx;
    float *dr, *dc, *sc, *scl, *scu, *srmin, *srmax, *yh32;
    float *x[2], *xa[2], *xbar, *vt, *g[2], *ab;
    float *y[2], *ya[2], *axc[2], *mt;
    double *rdr, *rdc;
    double *xh, *yh, *pesx, *pesy, *axh, *atyh;
    const float* fac;
    double tol;
    long long maxit;
    long long handoff_at;        // iterations after which an instance may be handed off
    unsigned int* handoff_count; // instances that asked (device counter)
    int handoff_max;             // at most this many are handed off
    int check;
    double* x_out;
    double* y_out;
    BatchOut* out;
};

// The step being attempted, written by the decision warp.
struct BatchStep {
    float tau, sigma, w;
    int parity;   // slot of the accepted iterates
    int check, done, restart, use_avg;
};

struct BMetrics {
    double pinf, dinf, gap, op, od, prow, err;
    bool finite;
};

// Controller state used at checks only (the decision warp's first lane).
struct BatchRare {
    double epoch_kkt, prev_cand;
    long long epoch_start, restarts;
    int status, asked, handed, have_pe;
    BMetrics last, now[2];
};

struct BatchShared {
    BatchRare rare;
    Acc<float> acc[kBW * 3];
    double dred[kBW * 8];
    int part[kBT];
    int inst;
    int longs[2];  // slices laid in steps, columns and rows
    BatchStep step;
};

// The CTA's dynamic shared memory: BatchShared, then what the instance holds.
// Functions name it themselves, rather than take pointers into it: loads and
// stores then are shared-memory ones, and nothing of the hot loops' state has
// to be in memory for the calls they make now and then.
constexpr size_t kSharedHead = (sizeof(BatchShared) + 15) & ~(size_t)15;
__device__ __forceinline__ unsigned char* b_mem() {
    extern __shared__ __align__(16) unsigned char b_smem[];
    return b_smem;
}
__device__ __forceinline__ BatchShared& b_shared() {
    return *reinterpret_cast<BatchShared*>(b_mem());
}

// ---- block-level helpers (every thread of the CTA calls them; `workers` is
// the number of worker threads; the others take no part) ------------------
template <int NV>
__device__ void bmerge(Acc<float> (&v)[NV], int workers) {
    BatchShared& sh = b_shared();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NV; ++q)
        for (int o = 16; o > 0; o >>= 1) v[q].shfl_xor(kFull, o, 32);
    __syncthreads();
    if (lane == 0 && (int)threadIdx.x < workers)
#pragma unroll
        for (int q = 0; q < NV; ++q) sh.acc[wp * NV + q] = v[q];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            Acc<float> s = sh.acc[q];
            for (int k = 1; k < workers / 32; ++k) s.merge(sh.acc[k * NV + q]);
            v[q] = s;
        }
    }
    __syncthreads();
}

// exclusive block scan of cnt[0..len) into out[0..len], out[len] = total
__device__ void bscan(const int* cnt, int* out, int len, int workers) {
    BatchShared& sh = b_shared();
    const int t = threadIdx.x;
    const int per = (len + workers - 1) / workers;
    const int b = min(len, t * per), e = min(len, b + per);
    int s = 0;
    for (int j = b; j < e; ++j) s += cnt[j];
    if (t < workers) sh.part[t] = s;
    __syncthreads();
    if (t == 0) {
        int run = 0;
        for (int k = 0; k < workers; ++k) {
            const int v = sh.part[k];
            sh.part[k] = run;
            run += v;
        }
        out[len] = run;
    }
    __syncthreads();
    int run = t < workers ? sh.part[t] : 0;
    for (int j = b; j < e; ++j) {
        out[j] = run;
        run += cnt[j];
    }
    __syncthreads();
}

struct Inst {
    int m, n;
    const int *ap, *ai;
    const float* ax;
    const double* axd;
    const double *c, *cl, *cu, *rmin, *rmax;
    int *cp, *ci, *cnt;
    float *cax, *sax, *scax;
    double* cax64;
    float *dr, *dc, *vt, *mt;
    double *rdr, *rdc;   // 1 / dr, 1 / dc
    double *xh, *yh, *pesx, *pesy, *axh, *atyh;
};

__device__ Inst make_inst(const BatchArgs& a, const BatchDesc& d) {
    Inst I;
    I.m = d.m;
    I.n = d.n;
    I.ap = a.ap + d.ap_off;
    I.ai = a.ai + d.nz_off;
    I.ax = a.ax + d.nz_off;
    I.axd = a.axd + d.nz_off;
    I.c = a.c + d.col_off;
    I.cl = a.cl + d.col_off;
    I.cu = a.cu + d.col_off;
    I.rmin = a.rmin + d.row_off;
    I.rmax = a.rmax + d.row_off;
    I.cp = a.cp + d.cp_off;
    I.ci = a.ci + d.nz_off;
    I.cnt = a.cnt + d.col_off;
    I.cax = a.cax + d.nz_off;
    I.cax64 = a.cax64 + d.nz_off;
    I.sax = a.sax + d.nz_off;
    I.scax = a.scax + d.nz_off;
    I.rdr = a.rdr + d.row_off;
    I.rdc = a.rdc + d.col_off;
    I.dr = a.dr + d.row_off;
    I.dc = a.dc + d.col_off;
    I.vt = a.vt + d.col_off;
    I.mt = a.mt + d.row_off;
    I.xh = a.xh + d.col_off;
    I.pesx = a.pesx + d.col_off;
    I.atyh = a.atyh + d.col_off;
    I.yh = a.yh + d.row_off;
    I.pesy = a.pesy + d.row_off;
    I.axh = a.axh + d.row_off;
    return I;
}

// The iterates and residual data the iteration works on, and the scaled
// matrix by slices of 32 columns (rows) of like length: the k-th entries of a
// slice's rows lie next to each other, padded with (0, entry 0) to its longest
// row, so a warp reads runs of words and no lane tests a length (a pad adds
// 0 x, nothing, to a sum; an infinite x ends the LP at its step's dot
// products). A slice that pads would more than double (a full row among short
// ones: a budget, a normalisation) is laid in steps instead: as wide
// as the rows that reach there, rounded up to a power of two. Every row's sum keeps
// the order of its entries.
template <int MODE>
struct Held {
    using Idx = typename std::conditional<MODE == kHeldWide, int, uint16_t>::type;
    int m, n;
    const int *cbase, *rbase;
    const uint16_t *cid, *rid;     // row numbers by position, or
    const int *cid32, *rid32;      // (up to kHeldOut) these
    const float *cv, *rv;
    const Idx *ci, *ri;
    float *xbar, *ab, *ys;  // ys: both slots of y
    // the vectors below follow each other in shared memory (kHeldAll) and
    // start at cols and rows; else they are the instance's in global memory
    float *cols, *rows;
    const BatchArgs* a;
    long long c0, r0;
    __device__ __forceinline__ float* col(int k, float* out) const {
        if constexpr (MODE == kHeldAll) return cols + k * n;
        else return out + c0;
    }
    __device__ __forceinline__ float* row(int k, float* out) const {
        if constexpr (MODE == kHeldAll) return rows + k * m;
        else return out + r0;
    }
    __device__ __forceinline__ float* sc() const { return col(0, a->sc); }
    __device__ __forceinline__ float* scl() const { return col(1, a->scl); }
    __device__ __forceinline__ float* scu() const { return col(2, a->scu); }
    __device__ __forceinline__ float* x(int p) const { return col(3 + p, p ? a->x[1] : a->x[0]); }
    __device__ __forceinline__ float* xa(int p) const { return col(5 + p, p ? a->xa[1] : a->xa[0]); }
    __device__ __forceinline__ float* g(int p) const { return col(7 + p, p ? a->g[1] : a->g[0]); }
    __device__ __forceinline__ float* srmin() const { return row(0, a->srmin); }
    __device__ __forceinline__ float* srmax() const { return row(1, a->srmax); }
    __device__ __forceinline__ float* yh32() const { return row(2, a->yh32); }
    __device__ __forceinline__ float* ya(int p) const { return row(3 + p, p ? a->ya[1] : a->ya[0]); }
    __device__ __forceinline__ float* axc(int p) const { return row(5 + p, p ? a->axc[1] : a->axc[0]); }
    __device__ __forceinline__ float* y(int p) const {
        if constexpr (MODE == kHeldWide) return (p ? a->y[1] : a->y[0]) + r0;
        else return ys + p * m;
    }
};

template <int MODE>
__device__ __forceinline__ Held<MODE> make_work(const BatchArgs& a, const BatchDesc& d) {
    unsigned char* smem = b_mem() + kSharedHead;
    Held<MODE> W;
    const int m = d.m, n = d.n;
    W.m = m;
    W.n = n;
    W.a = &a;
    W.c0 = d.col_off;
    W.r0 = d.row_off;
    W.cols = W.rows = W.ys = nullptr;
    const int sc = slices_of(n), sr = slices_of(m);
    if constexpr (MODE <= kHeldOut) {
        W.cbase = a.bases + d.base_off;
        W.rbase = W.cbase + sc + 1;
        W.cid = W.rid = nullptr;
        W.cid32 = a.order_c + d.col_off;
        W.rid32 = a.order_r + d.row_off;
        W.cv = a.out_val + d.out_off;
        W.rv = W.cv + d.pad_c;
        W.ci = reinterpret_cast<const typename Held<MODE>::Idx*>(a.out_idx + d.out_off);
        W.ri = W.ci + d.pad_c;
        if constexpr (MODE == kHeldOut) {
            W.xbar = reinterpret_cast<float*>(smem);
            W.ys = W.xbar + n;
        } else {
            W.xbar = a.xbar + d.col_off;
        }
        W.ab = a.ab + d.row_off;
    } else {
        float* v = reinterpret_cast<float*>(smem);
        W.cv = v;
        W.rv = v + d.pad_c;
        W.xbar = v + d.pad_c + d.pad_r;
        W.ys = W.xbar + n;
        W.ab = W.ys + 2 * m;
        int* p = reinterpret_cast<int*>(W.ab + m);
        W.cbase = p;
        W.rbase = p + sc + 1;
        uint16_t* i = reinterpret_cast<uint16_t*>(p + sc + sr + 2);
        W.ci = i;
        W.ri = i + d.pad_c;
        W.cid = i + d.pad_c + d.pad_r;
        W.rid = W.cid + n;
        W.cid32 = W.rid32 = nullptr;
        W.cols = reinterpret_cast<float*>(smem + matrix_bytes(d));
        W.rows = W.cols + 9 * (size_t)n;
    }
    return W;
}

// Fills the staged matrix (by the worker warps, a slice at a time).
template <int MODE, bool LONG>
__device__ __noinline__ void fill_work(const BatchArgs& a, const BatchDesc* dp, int workers) {
    const BatchDesc d = *dp;
    const Inst I = make_inst(a, d);
    const Held<MODE> W = make_work<MODE>(a, d);
    using Idx = typename Held<MODE>::Idx;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, nw = workers >> 5;
    const int sc = slices_of(I.n), sr = slices_of(I.m);
    const int* order[2] = {a.order_c + d.col_off, a.order_r + d.row_off};
    const int* bases = a.bases + d.base_off;
    if constexpr (MODE > kHeldOut) {
        for (int s = t; s < sc + sr + 2; s += blockDim.x) const_cast<int*>(W.cbase)[s] = bases[s];
        for (int j = t; j < I.n; j += blockDim.x)
            const_cast<uint16_t*>(W.cid)[j] = (uint16_t)order[0][j];
        for (int i = t; i < I.m; i += blockDim.x)
            const_cast<uint16_t*>(W.rid)[i] = (uint16_t)order[1][i];
    }
    for (int w = wp; w < sc + sr && wp < nw; w += nw) {
        const bool r = w >= sc;
        const int s = r ? w - sc : w, q = 32 * s + lane;
        const int* ptr = r ? I.ap : I.cp;
        const int* idx = r ? I.ai : I.ci;
        const float* val = r ? I.sax : I.scax;
        const int b0 = bases[r ? sc + 1 + s : s], b1 = bases[r ? sc + 2 + s : s + 1];
        float* v0 = const_cast<float*>(r ? W.rv : W.cv);
        Idx* ix0 = const_cast<Idx*>(r ? W.ri : W.ci);
        float* v = v0 + 32LL * b0 + lane;
        Idx* ix = ix0 + 32LL * b0 + lane;
        int p = 0, e = 0;
        if (q < (r ? I.m : I.n)) {
            const int row = order[r ? 1 : 0][q];
            p = ptr[row];
            e = ptr[row + 1];
        }
        auto put = [&]() {
            *v = p < e ? val[p] : 0.f;
            *ix = (Idx)(p < e ? idx[p] : 0);
        };
        if (!LONG || b1 > b0 || __all_sync(kFull, p == e)) {
            for (int k = b0; k < b1; ++k, ++p, v += 32, ix += 32) put();
            continue;
        }
        // in steps: the entry of the slices' table (written here as well), depths, entries
        const int* table = a.longs + (r ? d.long_r_at : d.long_c_at);
        const int units = bases[r ? sc + 1 + sr : sc];
        int at = 0;
        while (table[2 * at] != s) ++at;
        if (lane < 2) v0[32LL * units + 2 * at + lane] = __int_as_float(table[2 * at + lane]);
        const long long first = 32LL * table[2 * at + 1];
        const int len = e - p;
        v = v0 + first + 32 + lane;
        ix = ix0 + first + 32 + lane;
        for (int st = 0, k = 0; st < kSteps; ++st) {
            const int w = 32 >> st, to = __shfl_sync(kFull, len, step_lane(st));
            if (lane == st) v0[first + st] = __int_as_float(to - k);
            for (; k < to; ++k, ++p, v += w, ix += w)
                if (lane < w) put();
        }
    }
    __syncthreads();
}

// The products of the lane's staged row (slice entries 32 b0 .. 32 b1) with
// v, compensated FP32, in the order of the entries.
template <bool OUT, class Idx>
__device__ __forceinline__ Acc<float> padded_dot(const Idx* idx, const float* val,
                                                 const float* __restrict__ v, int b0, int b1) {
    using At = typename std::conditional<OUT, long long, int>::type;
    constexpr int kAhead = OUT ? 4 : 2;  // loads in flight
    At at = 32 * (At)b0 + (threadIdx.x & 31);
    int left = b1 - b0;
    Acc<float> acc;
#pragma unroll 1
    for (; left >= kAhead; left -= kAhead, at += 32 * kAhead) {
        float w[kAhead], x[kAhead];
        int j[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            w[u] = val[at + 32 * u];
            j[u] = idx[at + 32 * u];
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) x[u] = v[j[u]];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) acc.add(w[u], x[u]);
    }
#pragma unroll 1
    for (; left; --left, at += 32) acc.add(val[at], v[idx[at]]);
    return acc;
}

// Adds `steps` products (with their errors) to each lane's sum, in order: lane's
// from the lanes mine, mine + wide, ...
__device__ __forceinline__ void lane_sums(Acc<float>& acc, float p, float pe, int wide, int mine,
                                          int steps) {
    int u = 0;
#pragma unroll 1
    for (; u + 8 <= steps; u += 8) {
        float ps[8], es[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            ps[k] = __shfl_sync(kFull, p, (u + k) * wide + mine);
            es[k] = __shfl_sync(kFull, pe, (u + k) * wide + mine);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) acc.add_product(ps[k], es[k]);
    }
#pragma unroll 1
    for (; u < steps; ++u)
        acc.add_product(__shfl_sync(kFull, p, u * wide + mine), __shfl_sync(kFull, pe, u * wide + mine));
}

// The same of a slice laid in steps, from its first entry (depths). The lanes
// take 32 entries at once, loads and products, and the sums then run over them in
// order, the row's lane getting each product from the lane that formed it.
template <class Idx>
__device__ __forceinline__ Acc<float> stepped_dot(const Idx* idx, const float* val,
                                                  const float* __restrict__ v, long long first) {
    const int lane = threadIdx.x & 31;
    long long at = first + 32;
    Acc<float> acc;
#pragma unroll 1
    for (int st = 0; st < kSteps; ++st) {
        const int wide = 32 >> st, mine = lane & (wide - 1), per = 1 << st;
        const int depth = __float_as_int(val[first + st]);
        const long long end = at + (long long)wide * depth;
        float w = 0.f, x = 0.f;
        auto load = [&](long long k) {
            w = x = 0.f;
            if (k + lane < end) {
                w = val[k + lane];
                x = v[idx[k + lane]];
            }
        };
        load(at);
        const Acc<float> before = acc;
#pragma unroll 1
        for (int left = depth; left > 0; left -= per) {
            const float p = w * x, pe = fmaf(w, x, -p);
            at += 32;
            load(at);
            lane_sums(acc, p, pe, wide, mine, min(left, per));
        }
        if (lane >= wide) acc = before;  // (the other lanes' rows have ended)
        at = end;
    }
    return acc;
}

// Either of them, by slice.
template <bool OUT, bool LONG, class Idx>
__device__ __forceinline__ Acc<float> any_dot(const int* base, const Idx* idx, const float* val,
                                              const float* v, int s, int rows, int longs) {
    if constexpr (LONG) {
        const float* table = val + 32LL * base[slices_of(rows)];
        for (int i = 0; i < longs; ++i)
            if (__float_as_int(table[2 * i]) == s)
                return stepped_dot(idx, val, v, 32LL * __float_as_int(table[2 * i + 1]));
    }
    return padded_dot<OUT>(idx, val, v, base[s], base[s + 1]);
}

// Rows of the CSR (columns of the CSC): f by one of the `workers` threads each,
// those of more than kLongRow entries g by a warp each (they come first in the
// order by length).
template <bool LONG, class F, class G>
__device__ __forceinline__ void each_row(const int* ptr, const int* order, int longer, int rows, int t,
                                         int workers, F f, G g) {
    if constexpr (!LONG) {
        for (int r = t; r < rows; r += workers) f(r);
        return;
    }
    for (int r = t; r < rows; r += workers)
        if (ptr[r + 1] - ptr[r] <= kLongRow) f(r);
    if (t >= workers) return;
    __syncwarp();
    for (int q = t >> 5; q < longer; q += workers >> 5) g(order[q]);
}
// f(p) for every entry p of a row, by a warp
template <class F>
__device__ __forceinline__ void warp_entries(const int* ptr, int r, F f) {
    for (int p = ptr[r] + (threadIdx.x & 31); p < ptr[r + 1]; p += 32) f(p);
}
// the sum of a(p) * x(p) over a row by a warp, as one thread takes it: the
// factors by 32 lanes at once, the chain over them in order in every lane
template <class A, class X>
__device__ __forceinline__ double warp_chain(const int* ptr, int r, A a, X x) {
    double s = 0.0;
    for (int b = ptr[r], e = ptr[r + 1]; b < e; b += 32) {
        const int p = min(b + (int)(threadIdx.x & 31), e - 1);
        const double av = a(p), xv = x(p);
        for (int u = 0; u < min(32, e - b); ++u)
            s = fma(__shfl_sync(kFull, av, u), __shfl_sync(kFull, xv, u), s);
    }
    return s;
}
// row_dot by a warp, in every lane
__device__ __forceinline__ Acc<float> warp_row_dot(const int* ptr, const int* idx, const float* val,
                                                   const float* v, int r) {
    Acc<float> acc;
    for (int b = ptr[r], e = ptr[r + 1]; b < e; b += 32) {
        const int p = b + (threadIdx.x & 31);
        const float w = p < e ? val[p] : 0.f, x = p < e ? v[idx[p]] : 0.f, pr = w * x;
        lane_sums(acc, pr, fmaf(w, x, -pr), 1, 0, min(32, e - b));
    }
    return acc;
}

// one row of a CSR times v (thread per row, compensated FP32)
__device__ __forceinline__ Acc<float> row_dot(const int* ptr, const int* idx, const float* val,
                                              const float* v, int r) {
    Acc<float> acc;
    for (int p = ptr[r]; p < ptr[r + 1]; ++p) acc.add(val[p], v[idx[p]]);
    return acc;
}

// Full FP64 column value of delta dx (scaled units), with the at-bound rule:
// a delta on its FP32 shifted bound is exactly at the bound.
template <int MODE>
__device__ __forceinline__ double full_x(const Inst& I, const Held<MODE>& W, int j, float dx) {
    if (dx == W.scl()[j]) return I.cl[j] / (double)I.dc[j];
    if (dx == W.scu()[j]) return I.cu[j] / (double)I.dc[j];
    return I.xh[j] + (double)dx;
}

// Residual data of the LP seen from the anchor (xh, yh), FP64 -> FP32:
// sc = c~ + A~^T yh, [scl, scu] = box~ - xh, [srmin, srmax] = rows~ - A~ xh,
// with A~_ij = a_ij dc_j / dr_i formed in FP64 from the FP64 values.
template <int MODE, bool LONG>
__device__ __noinline__ void anchor_data(const BatchArgs& a, const BatchDesc* d, int t,
                                         int workers) {
    const Inst I = make_inst(a, *d);
    const Held<MODE> W = make_work<MODE>(a, *d);
    auto row = [&](int i, double dri, double s) {
        I.axh[i] = s;
        W.srmin()[i] = (float)(I.rmin[i] / dri - s);
        W.srmax()[i] = (float)(I.rmax[i] / dri - s);
        W.yh32()[i] = (float)I.yh[i];
    };
    each_row<LONG>(I.ap, a.order_r + d->row_off, d->longer_r, I.m, t, workers,
             [&](int i) {
                 const double dri = I.dr[i];
                 double s = 0.0;
                 for (int p = I.ap[i]; p < I.ap[i + 1]; ++p) {
                     const int j = I.ai[p];
                     s = fma(I.axd[p] * (double)I.dc[j] / dri, I.xh[j], s);
                 }
                 row(i, dri, s);
             },
             [&](int i) {
                 const double dri = I.dr[i];
                 const double s = warp_chain(
                     I.ap, i, [&](int p) { return I.axd[p] * (double)I.dc[I.ai[p]] / dri; },
                     [&](int p) { return I.xh[I.ai[p]]; });
                 if ((threadIdx.x & 31) == 0) row(i, dri, s);
             });
    auto column = [&](int j, double dcj, double s) {
        I.atyh[j] = s;
        W.sc()[j] = (float)(I.c[j] * dcj + s);
        W.scl()[j] = (float)(I.cl[j] / dcj - I.xh[j]);
        W.scu()[j] = (float)(I.cu[j] / dcj - I.xh[j]);
    };
    each_row<LONG>(I.cp, a.order_c + d->col_off, d->longer_c, I.n, t, workers,
             [&](int j) {
                 const double dcj = I.dc[j];
                 double s = 0.0;
                 for (int p = I.cp[j]; p < I.cp[j + 1]; ++p) {
                     const int i = I.ci[p];
                     s = fma(I.cax64[p] * dcj / (double)I.dr[i], I.yh[i], s);
                 }
                 column(j, dcj, s);
             },
             [&](int j) {
                 const double dcj = I.dc[j];
                 const double s = warp_chain(
                     I.cp, j, [&](int p) { return I.cax64[p] * dcj / (double)I.dr[I.ci[p]]; },
                     [&](int p) { return I.yh[I.ci[p]]; });
                 if ((threadIdx.x & 31) == 0) column(j, dcj, s);
             });
    __syncthreads();
}

// ---- setup: CSC, Ruiz, scaled data, power iteration ----------------------
// (t: this thread among the workers, beyond every size for the decision warp)
template <bool LONG>
__device__ __noinline__ void setup(const BatchArgs& a, const BatchDesc* d, int t, int workers,
                                   float& eta0, float& omega0) {
    const Inst I = make_inst(a, *d);
    const int m = I.m, n = I.n;
    const int *by_row = a.order_r + d->row_off, *by_col = a.order_c + d->col_off;
    const bool first_lane = (threadIdx.x & 31) == 0;
    // CSC by counting sort; each column's entries ordered by row afterwards
    for (int j = t; j < n; j += workers) I.cnt[j] = 0;
    __syncthreads();
    auto count = [&](int p) { atomicAdd(&I.cnt[I.ai[p]], 1); };
    each_row<LONG>(I.ap, by_row, d->longer_r, m, t, workers,
             [&](int i) {
                 for (int p = I.ap[i]; p < I.ap[i + 1]; ++p) count(p);
             },
             [&](int i) { warp_entries(I.ap, i, count); });
    __syncthreads();
    bscan(I.cnt, I.cp, n, workers);
    for (int j = t; j < n; j += workers) I.cnt[j] = I.cp[j];
    __syncthreads();
    auto place = [&](int i, int p) {
        const int q = atomicAdd(&I.cnt[I.ai[p]], 1);
        I.ci[q] = i;
        I.cax64[q] = I.axd[p];
    };
    each_row<LONG>(I.ap, by_row, d->longer_r, m, t, workers,
             [&](int i) {
                 for (int p = I.ap[i]; p < I.ap[i + 1]; ++p) place(i, p);
             },
             [&](int i) {
                 // lanes that meet in a column (entries that the row has twice) in order
                 const int lane = threadIdx.x & 31;
                 for (int p = I.ap[i] + lane, e = I.ap[i + 1]; p - lane < e; p += 32) {
                     const unsigned on = __ballot_sync(kFull, p < e);
                     if (p < e) {
                         const unsigned peers = __match_any_sync(on, I.ai[p]);
                         const int first = __ffs(peers) - 1;
                         int q = 0;
                         if (lane == first) q = atomicAdd(&I.cnt[I.ai[p]], __popc(peers));
                         __syncwarp(on);
                         q = __shfl_sync(on, q, first) + __popc(peers & ((1u << lane) - 1));
                         I.ci[q] = i;
                         I.cax64[q] = I.axd[p];
                     }
                     __syncwarp();
                 }
             });
    __syncthreads();
    for (int j = t; j < n; j += workers) {  // insertion sort by row index
        const int b = I.cp[j], e = I.cp[j + 1];
        for (int q = b + 1; q < e; ++q) {
            const int r = I.ci[q];
            const double v = I.cax64[q];
            int k = q - 1;
            while (k >= b && I.ci[k] > r) {
                I.ci[k + 1] = I.ci[k];
                I.cax64[k + 1] = I.cax64[k];
                --k;
            }
            I.ci[k + 1] = r;
            I.cax64[k + 1] = v;
        }
        for (int q = b; q < e; ++q) I.cax[q] = (float)I.cax64[q];
    }
    // Ruiz, 10 sweeps (FP32 factors)
    for (int i = t; i < m; i += workers) I.dr[i] = 1.f;
    for (int j = t; j < n; j += workers) I.dc[j] = 1.f;
    __syncthreads();
    for (int sweep = 0; sweep < 10; ++sweep) {
        auto top = [&](float mx) {  // of a warp
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
            return mx;
        };
        auto row_max = [&](int i, int p) { return fabsf(I.ax[p]) * I.dc[I.ai[p]] / I.dr[i]; };
        auto scale_row = [&](int i, float mx) {
            if (mx > 0.f && isfinite(mx)) I.dr[i] *= sqrtf(mx);
        };
        each_row<LONG>(I.ap, by_row, d->longer_r, m, t, workers,
                 [&](int i) {
                     float mx = 0.f;
                     for (int p = I.ap[i]; p < I.ap[i + 1]; ++p) mx = fmaxf(mx, row_max(i, p));
                     scale_row(i, mx);
                 },
                 [&](int i) {
                     float mx = 0.f;
                     warp_entries(I.ap, i, [&](int p) { mx = fmaxf(mx, row_max(i, p)); });
                     mx = top(mx);
                     if (first_lane) scale_row(i, mx);
                 });
        __syncthreads();
        auto col_max = [&](int j, int p) { return fabsf(I.cax[p]) / I.dr[I.ci[p]] * I.dc[j]; };
        auto scale_col = [&](int j, float mx) {
            if (mx > 0.f && isfinite(mx)) I.dc[j] /= sqrtf(mx);
        };
        each_row<LONG>(I.cp, by_col, d->longer_c, n, t, workers,
                 [&](int j) {
                     float mx = 0.f;
                     for (int p = I.cp[j]; p < I.cp[j + 1]; ++p) mx = fmaxf(mx, col_max(j, p));
                     scale_col(j, mx);
                 },
                 [&](int j) {
                     float mx = 0.f;
                     warp_entries(I.cp, j, [&](int p) { mx = fmaxf(mx, col_max(j, p)); });
                     mx = top(mx);
                     if (first_lane) scale_col(j, mx);
                 });
        __syncthreads();
    }
    for (int i = t; i < m; i += workers) I.rdr[i] = 1.0 / (double)I.dr[i];
    for (int j = t; j < n; j += workers) I.rdc[j] = 1.0 / (double)I.dc[j];
    // scaled FP32 matrix; initial weight from the scaled cost and row bounds
    Acc<float> nq[2];
    auto scaled = [&](int i, int p) { I.sax[p] = I.ax[p] * I.dc[I.ai[p]] / I.dr[i]; };
    auto scaled_c = [&](int j, int p) { I.scax[p] = I.cax[p] * I.dc[j] / I.dr[I.ci[p]]; };
    each_row<LONG>(I.ap, by_row, d->longer_r, m, t, workers,
             [&](int i) {
                 for (int p = I.ap[i]; p < I.ap[i + 1]; ++p) scaled(i, p);
             },
             [&](int i) { warp_entries(I.ap, i, [&](int p) { scaled(i, p); }); });
    each_row<LONG>(I.cp, by_col, d->longer_c, n, t, workers,
             [&](int j) {
                 for (int p = I.cp[j]; p < I.cp[j + 1]; ++p) scaled_c(j, p);
             },
             [&](int j) { warp_entries(I.cp, j, [&](int p) { scaled_c(j, p); }); });
    for (int i = t; i < m; i += workers) {
        const float lo = (float)I.rmin[i] / I.dr[i], hi = (float)I.rmax[i] / I.dr[i];
        const float q = isfinite(hi) ? hi : (isfinite(lo) ? lo : 0.f);
        nq[1].add(q, q);
    }
    for (int j = t; j < n; j += workers) {
        const float cs = (float)I.c[j] * I.dc[j];
        nq[0].add(cs, cs);
    }
    bmerge<2>(nq, workers);
    if (t == 0) {
        const double cn = nq[0].result_d(), qn = nq[1].result_d();
        omega0 = (cn > 1e-24 && qn > 1e-24) ? fminf(3.f, fmaxf(0.3f, (float)sqrt(cn / qn))) : 1.f;
    }
    // power iteration for ||A~||_2^2
    const float v0 = rsqrtf((float)n);
    for (int j = t; j < n; j += workers) I.vt[j] = v0;
    __syncthreads();
    __shared__ float s_norm;
    for (int it = 0; it < 31; ++it) {
        each_row<LONG>(I.ap, by_row, d->longer_r, m, t, workers,
                 [&](int i) { I.mt[i] = row_dot(I.ap, I.ai, I.sax, I.vt, i).result(); },
                 [&](int i) {
                     const float s = warp_row_dot(I.ap, I.ai, I.sax, I.vt, i).result();
                     if (first_lane) I.mt[i] = s;
                 });
        __syncthreads();
        if (it == 30) break;
        // (normalised below, past the barrier)
        Acc<float> nrm[1];
        if constexpr (!LONG) {
            for (int j = t; j < n; j += workers) {
                const float wv = row_dot(I.cp, I.ci, I.scax, I.mt, j).result();
                I.vt[j] = wv;
                nrm[0].add(wv, wv);
            }
        } else {
            each_row<LONG>(I.cp, by_col, d->longer_c, n, t, workers,
                     [&](int j) { I.vt[j] = row_dot(I.cp, I.ci, I.scax, I.mt, j).result(); },
                     [&](int j) {
                         const float s = warp_row_dot(I.cp, I.ci, I.scax, I.mt, j).result();
                         if (first_lane) I.vt[j] = s;
                     });
            __syncthreads();
            for (int j = t; j < n; j += workers) nrm[0].add(I.vt[j], I.vt[j]);
        }
        bmerge<1>(nrm, workers);
        if (t == 0) s_norm = sqrtf((float)nrm[0].result_d());
        __syncthreads();
        const float nw = s_norm;
        if (!(nw > 1e-30f)) break;
        for (int j = t; j < n; j += workers) I.vt[j] = I.vt[j] / nw;
        __syncthreads();
    }
    Acc<float> na[1];
    for (int i = t; i < m; i += workers) na[0].add(I.mt[i], I.mt[i]);
    bmerge<1>(na, workers);
    if (t == 0) {
        double lam = na[0].result_d();
        if (!(lam > 0) || !isfinite(lam)) lam = 1.0;
        eta0 = (float)(1.2 / sqrt(lam));
    }
    __syncthreads();
}

// ---- FP64 metrics of both candidates (anchor + delta, original units) ----
// FP64 comparisons cost a hundred cycles of latency and a slot of the one
// FP64 unit of an SM; these run on the integer pipe. blt: a < b, false with a
// NaN; bmax: maximum of values >= 0 (a NaN counts as nothing).
__device__ __forceinline__ bool blt(double a, double b) {
    const long long inf = 0x7ff0000000000000LL, sign = (long long)(1ULL << 63);
    long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    if ((x & ~sign) > inf || (y & ~sign) > inf) return false;
    x = x < 0 ? sign - x : x;  // -0 -> 0, negatives in their order
    y = y < 0 ? sign - y : y;
    return x < y;
}
__device__ __forceinline__ double bsel_max(double a, double b) { return blt(a, b) ? b : a; }
__device__ __forceinline__ double bsel_min(double a, double b) { return blt(b, a) ? b : a; }
__device__ __forceinline__ double bmax(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return y > x && y <= 0x7ff0000000000000LL ? b : a;
}
__device__ __forceinline__ double warp_bmax(double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(kFull, hi);
    const unsigned ml = __reduce_max_sync(kFull, hi == mh ? lo : 0u);
    return __hiloint2double((int)mh, (int)ml);
}

// a / b for one divisor b, rb = 1 / b correctly rounded: one remainder step, the
// correctly rounded quotient (Markstein 1990). The divisors are scale factors and
// weights, near 1.
__device__ __forceinline__ double div_by(double a, double b, double rb) {
    const double q0 = a * rb;
    return dfinite(q0) ? fma(fma(-b, q0, a), rb, q0) : q0;
}

// The metrics of the current (0) and averaged (1) iterates; valid in the
// decision warp's first lane. Two barriers; the candidates share them and the
// loads of the LP's data.
template <int MODE, bool LONG>
__device__ __noinline__ void metrics(const BatchArgs& a, const BatchDesc* d, int pc, int t,
                                     int workers, double cmax, BMetrics* out) {
    BatchShared& sh = b_shared();
    const Inst I = make_inst(a, *d);
    const Held<MODE> W = make_work<MODE>(a, *d);
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, nw = workers >> 5;
    const bool works = wp < nw;
    const float* xs[2] = {W.x(pc), W.xa(pc)};
    const float* ys[2] = {W.y(pc), W.ya(pc)};
    double mx[2][4] = {};  // pv, pa, prow, ymax
    for (int s = wp; works && 32 * s < I.m; s += nw) {
        const int q = 32 * s + lane;
        const int i = q < I.m ? (MODE <= kHeldOut ? W.rid32[q] : (int)W.rid[q]) : I.m;
        for (int v = 0; v < 2; ++v) {
            const Acc<float> ad = any_dot<MODE <= kHeldOut, LONG>(W.rbase, W.ri, W.rv, xs[v], s, I.m, sh.longs[1]);
            if (i >= I.m) continue;
            const double Ax = (I.axh[i] + ad.result_d()) * (double)I.dr[i];
            const double lo = I.rmin[i], hi = I.rmax[i];
            const double vi = bsel_max(lo - Ax, Ax - hi);
            mx[v][0] = bmax(mx[v][0], vi);
            mx[v][1] = bmax(mx[v][1], dabs(bsel_min(bsel_max(Ax, lo), hi)));
            if (blt(mx[v][2], vi)) {  // vi / (1 + scale) <= vi
                double scv = dabs(Ax);
                if (dfinite(lo)) scv = bsel_max(scv, dabs(lo));
                if (dfinite(hi)) scv = bsel_max(scv, dabs(hi));
                mx[v][2] = bmax(mx[v][2], vi / (1.0 + scv));
            }
            mx[v][3] = bmax(mx[v][3], dabs(div_by(I.yh[i] + (double)ys[v][i], I.dr[i], I.rdr[i])));
        }
    }
    if (works)
        for (int v = 0; v < 2; ++v)
            for (int q = 0; q < 4; ++q) {
                const double r = warp_bmax(mx[v][q]);
                if (lane == 0) sh.dred[wp * 8 + 4 * v + q] = r;
            }
    __syncthreads();
    double yz[2], top[2][3];
    for (int v = 0; v < 2; ++v) {
        double ymax = 0.0;
        for (int k = 0; k < nw; ++k) ymax = bmax(ymax, sh.dred[k * 8 + 4 * v + 3]);
        yz[v] = 1e-8 * (1.0 + ymax);
        if (!works)
            for (int q = 0; q < 3; ++q) {
                top[v][q] = 0.0;
                for (int k = 0; k < nw; ++k) top[v][q] = bmax(top[v][q], sh.dred[k * 8 + 4 * v + q]);
            }
    }
    __syncthreads();  // dred is written again below
    const double dz = 1e-8 * (1.0 + cmax);
    double dv[2] = {0.0, 0.0}, op[2] = {0.0, 0.0}, od[2] = {0.0, 0.0};
    bool unb[2] = {false, false};
    for (int s = wp; works && 32 * s < I.n; s += nw) {
        const int q = 32 * s + lane;
        const int j = q < I.n ? (MODE <= kHeldOut ? W.cid32[q] : (int)W.cid[q]) : I.n;
        for (int v = 0; v < 2; ++v) {
            const Acc<float> ad = any_dot<MODE <= kHeldOut, LONG>(W.cbase, W.ci, W.cv, ys[v], s, I.n, sh.longs[0]);
            if (j >= I.n) continue;
            const double dcj = I.dc[j], cj = I.c[j];
            const double aty = I.atyh[j] + ad.result_d();
            const double d = cj + div_by(aty, dcj, I.rdc[j]);
            const double lo = I.cl[j], hi = I.cu[j];
            const float xv = xs[v][j];
            const double x = xv == W.scl()[j] ? lo : (xv == W.scu()[j] ? hi : (I.xh[j] + (double)xv) * dcj);
            const double bnd = dabs(dfinite(hi) ? hi : lo);
            const double tol = 1e-9 * (1.0 + bnd);
            const double lob = lo + tol, hib = hi - tol;
            const bool pos = blt(0.0, d), neg = blt(d, 0.0);
            // (x <= lob is not lob < x, but for a NaN, which is not at a bound)
            const bool real = blt(x, CUDART_INF) || blt(-CUDART_INF, x);
            const bool at_lo = pos && real && lob == lob && !blt(lob, x);
            const bool at_hi = neg && real && hib == hib && !blt(x, hib);
            if (!at_lo && !at_hi) dv[v] = bmax(dv[v], dabs(d));
            op[v] += cj * x;
            if (!neg) {
                if (dfinite(lo)) od[v] += d * lo;
                else if (blt(dz, d)) unb[v] = true;
            } else {
                if (dfinite(hi)) od[v] += d * hi;
                else if (blt(dz, -d)) unb[v] = true;
            }
        }
    }
    for (int i = t; i < I.m; i += workers)
        for (int v = 0; v < 2; ++v) {
            const double yv = div_by(I.yh[i] + (double)ys[v][i], I.dr[i], I.rdr[i]);
            if (blt(yz[v], yv)) {
                if (dfinite(I.rmax[i])) od[v] -= yv * I.rmax[i];
                else unb[v] = true;
            } else if (blt(yv, -yz[v])) {
                if (dfinite(I.rmin[i])) od[v] -= yv * I.rmin[i];
                else unb[v] = true;
            }
        }
    if (works)
        for (int v = 0; v < 2; ++v) {
            const double r = warp_bmax(dv[v]), so = warp_sum(op[v]), sd = warp_sum(od[v]);
            const bool u = __any_sync(kFull, unb[v]);
            if (lane == 0) {
                double* P = sh.dred + wp * 8 + 4 * v;
                P[0] = r;
                P[1] = so;
                P[2] = sd;
                P[3] = u ? 1.0 : 0.0;
            }
        }
    __syncthreads();
    if (!works && lane == 0)
        for (int v = 0; v < 2; ++v) {
            double r = 0.0, so = 0.0, sd = 0.0, u = 0.0;
            for (int k = 0; k < nw; ++k) {
                const double* P = sh.dred + k * 8 + 4 * v;
                r = bmax(r, P[0]);
                so += P[1];
                sd += P[2];
                u = bmax(u, P[3]);
            }
            BMetrics mt;
            mt.pinf = top[v][0] / (1.0 + top[v][1]);
            mt.prow = top[v][2];
            mt.dinf = r / (1.0 + cmax);
            mt.op = so;
            const bool bounded = !(u > 0.0);
            mt.od = bounded ? sd : -CUDART_INF;
            mt.gap = bounded ? smax(0.0, mt.op - mt.od) / (1.0 + fabs(mt.op)) : CUDART_INF;
            mt.finite = isfinite(mt.pinf) && isfinite(mt.dinf);
            mt.err = smax(mt.pinf, smax(mt.dinf, isfinite(mt.gap) ? mt.gap : 0.0));
            out[v] = mt;
        }
}

// A restart: the chosen candidate becomes the new FP64 anchor and the deltas
// restart at zero; the warps' squared movements of the anchor go to sh.dred.
template <int MODE>
__device__ __noinline__ void re_anchor(const BatchArgs& a, const BatchDesc* d, int pc, int use_avg,
                                       int t, int workers) {
    BatchShared& sh = b_shared();
    const Inst I = make_inst(a, *d);
    const Held<MODE> W = make_work<MODE>(a, *d);
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    float *x = W.x(pc), *xa = W.xa(pc), *g = W.g(pc);
    float *y = W.y(pc), *ya = W.ya(pc), *axc = W.axc(pc);
    double dn[2] = {0.0, 0.0};
    for (int j = t; j < I.n; j += workers) {
        const double nx = full_x<MODE>(I, W, j, use_avg ? xa[j] : x[j]);
        const double dd = nx - I.pesx[j];
        dn[0] = fma(dd, dd, dn[0]);
        I.pesx[j] = I.xh[j] = nx;
        x[j] = xa[j] = g[j] = 0.f;  // g = A~^T 0
    }
    for (int i = t; i < I.m; i += workers) {
        const double ny = I.yh[i] + (double)(use_avg ? ya[i] : y[i]);
        const double dd = ny - I.pesy[i];
        dn[1] = fma(dd, dd, dn[1]);
        I.pesy[i] = I.yh[i] = ny;
        y[i] = ya[i] = axc[i] = 0.f;
    }
    for (int v = 0; v < 2; ++v) {
        dn[v] = warp_sum(dn[v]);
        if (lane == 0 && wp < workers / 32) sh.dred[2 * wp + v] = dn[v];
    }
}

// ---- one LP --------------------------------------------------------------
// An iteration is bound by latency: the phases' instruction streams and
// dependent loads, and above all the step decision, a chain of FP64 operations
// (60 cycles each, a division 575) in one thread. So the decision has a warp
// of its own, which holds the controller's state in registers, and while it
// runs the workers form A~^T y of the dual just computed: the next attempt
// needs it if the step is accepted (after a rejected one the accepted dual's
// product is still there). Four barriers per attempt:
//   workers                                  decision warp
//   primal step (columns t, t + kBT, ..)     --
//   sums of its dx^2; A~ xbar (by slices)    factors of the next decision
//   dual step (rows t, t + kBT, ..), sums    merges the warps' dx^2
//   A~^T y' (by slices)                      merges the rest, decides
// One iteration of an LP of 113 x 282: 6.2 us with the whole CTA waiting for
// one thread's decision and a lane walking each row, now 3.4; 650 x 1,625
// (10,476 nonzeros) 18.7 -> 7.7; 792 x 1,980 (15,561; iterates and residual
// data do not fit beside the matrix) 22.1 -> 11.9.
__device__ __forceinline__ void cta_sync() {
    __syncwarp();
    asm volatile("barrier.sync 0;" ::: "memory");
}

// Merge of the warps' partials acc[0], acc[3], ... in their order.
__device__ __forceinline__ double merge_warps(const Acc<float>* acc, int warps) {
    Acc<float> s = acc[0];
#pragma unroll 1
    for (int k = 1; k < warps; ++k) s.merge(acc[3 * k]);
    return s.result_d();
}

// Acc merged over the lanes of a warp, as block_merge does.
template <int NV>
__device__ __forceinline__ void lanes_merge(Acc<float> (&v)[NV]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q].shfl_xor(kFull, o, 32);
}

// Products of the staged rows: out[id] = row id times v, in the order of its
// entries (compensated FP32), a warp per slice.
// Slices laid in steps by the warps that found them empty (kept out of the other
// slices' loop).
template <class Idx>
__device__ __noinline__ void long_products(const int* base, const uint16_t* id16, const int* id32,
                                           const Idx* idx, const float* val, const float* v, float* out,
                                           int rows, int longs) {
    const int lane = threadIdx.x & 31, warps = (blockDim.x >> 5) - 1, wp = threadIdx.x >> 5;
    const float* table = val + 32LL * base[slices_of(rows)];
    for (int i = 0; i < longs; ++i) {
        const int s = __float_as_int(table[2 * i]);
        if (s % warps != wp) continue;
        const int q = 32 * s + lane;
        const Acc<float> acc = stepped_dot(idx, val, v, 32LL * __float_as_int(table[2 * i + 1]));
        if (q < rows) out[id16 ? (int)id16[q] : id32[q]] = acc.result();
    }
}

template <bool OUT, bool LONG, class Idx>
__device__ __forceinline__ void slice_products(const int* base, const uint16_t* id16,
                                               const int* id32, const Idx* idx, const float* val,
                                               const float* __restrict__ v, float* out,
                                               int rows, int longs) {
    const int lane = threadIdx.x & 31, warps = (blockDim.x >> 5) - 1;
    for (int s = threadIdx.x >> 5; 32 * s < rows; s += warps) {
        const int q = 32 * s + lane;
        const int row = q < rows ? (id16 ? (int)id16[q] : id32[q]) : -1;
        const Acc<float> acc = padded_dot<OUT>(idx, val, v, base[s], base[s + 1]);
        if (row >= 0) out[row] = acc.result();
    }
    if constexpr (LONG) long_products(base, id16, id32, idx, val, v, out, rows, longs);
}

// LONG: the instance has slices laid in steps.
template <int MODE, bool LONG>
__device__ __forceinline__ void worker_loop(const BatchArgs& a, const BatchDesc* d,
                                            const Held<MODE>& W, int workers, double cmax) {
    BatchShared& sh = b_shared();
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int t = (int)threadIdx.x < workers ? (int)threadIdx.x : 1 << 30;
    const int m = W.m, n = W.n;
    for (;;) {
        const int p = sh.step.parity, q = p ^ 1;
        const float tau = sh.step.tau, sigma = sh.step.sigma, w = sh.step.w;
        Acc<float> dx2[1];
        {   // primal step from g = A~^T y (thread per column), on the deltas
            const float *__restrict__ sc = W.sc(), *__restrict__ gp = W.g(p);
            const float *__restrict__ xp = W.x(p), *__restrict__ xap = W.xa(p);
            const float *__restrict__ lo = W.scl(), *__restrict__ hi = W.scu();
            float *__restrict__ xq = W.x(q), *__restrict__ xaq = W.xa(q);
            float* __restrict__ xbar = W.xbar;
            // (short code: unrolled by 2 or 4, an iteration takes 5-15 % longer)
#pragma unroll 1
            for (int j = t; j < n; j += workers) {
                const float g = sc[j] + gp[j];
                const float xv = xp[j], av = xap[j];
                const float xn = fminf(fmaxf(fmaf(-tau, g, xv), lo[j]), hi[j]);
                xq[j] = xn;
                xbar[j] = fmaf(2.f, xn, -xv);
                const float dx = xn - xv;
                dx2[0].add(dx, dx);
                xaq[j] = fmaf(w, xn - av, av);
            }
        }
        cta_sync();
        if (t < workers) {
            lanes_merge(dx2);
            if (lane == 0) sh.acc[wp * 3] = dx2[0];
        }
        slice_products<MODE <= kHeldOut, LONG>(W.rbase, W.rid, W.rid32, W.ri, W.rv, W.xbar, W.ab, m,
                                               LONG ? sh.longs[1] : 0);
        cta_sync();
        {   // dual step; the projection acts on the full value, so the anchor
            // enters its argument
            const float *__restrict__ yp = W.y(p), *__restrict__ axp = W.axc(p);
            const float *__restrict__ yap = W.ya(p), *__restrict__ ab_ = W.ab;
            const float *__restrict__ yh = W.yh32(), *__restrict__ lo = W.srmin();
            const float* __restrict__ hi = W.srmax();
            float *__restrict__ yq = W.y(q), *__restrict__ axq = W.axc(q);
            float* __restrict__ yaq = W.ya(q);
            Acc<float> dots[2];
#pragma unroll 1
            for (int i = t; i < m; i += workers) {
                const float ab = ab_[i], yv = yp[i], ax = axp[i], av = yap[i];
                const float tt = fmaf(sigma, ab, yv);
                const float arg = (tt + yh[i]) / sigma;
                const float yn = fmaf(-sigma, fminf(fmaxf(arg, lo[i]), hi[i]), tt);
                yq[i] = yn;
                const float dy = yn - yv;
                const float adx = 0.5f * (ab - ax);
                axq[i] = ax + adx;
                dots[0].add(dy, dy);
                dots[1].add(dy, adx);
                yaq[i] = fmaf(w, yn - av, av);
            }
            if (t < workers && 32 * wp < m) {  // (warp-uniform)
                __syncwarp();
                lanes_merge(dots);
                if (lane == 0) {
                    sh.acc[wp * 3 + 1] = dots[0];
                    sh.acc[wp * 3 + 2] = dots[1];
                }
            }
        }
        cta_sync();
        slice_products<MODE <= kHeldOut, LONG>(W.cbase, W.cid, W.cid32, W.ci, W.cv, W.y(q), W.g(q), n,
                                               LONG ? sh.longs[0] : 0);
        cta_sync();
        if (sh.step.done) return;
        if (!sh.step.check) continue;
        const int pc = sh.step.parity;
        metrics<MODE, LONG>(a, d, pc, t, workers, cmax, nullptr);
        cta_sync();
        if (sh.step.done) return;
        if (sh.step.restart) {
            re_anchor<MODE>(a, d, pc, sh.step.use_avg, t, workers);
            cta_sync();
            anchor_data<MODE, LONG>(a, d, t, workers);  // ends with a barrier
        }
    }
}

// The decision warp's side of the same loop. Its first lane holds the state.
template <int MODE, bool LONG>
__device__ __forceinline__ void decision_loop(const BatchArgs& a, const BatchDesc* d, int workers,
                                              double cmax, double eta, double omega, BatchOut& o) {
    BatchShared& sh = b_shared();
    const int lane = threadIdx.x & 31;
    const int warps_c = min(workers, d->n + 31) / 32, warps_r = min(workers, d->m + 31) / 32;
    BatchRare& c = sh.rare;
    double romega = 1.0 / omega;
    long long k = 1, hn = 0, attempts = 0;
    int until = a.check, retries = 0;
    if (lane == 0) {
        c.epoch_kkt = -1.0;
        c.prev_cand = CUDART_INF;
        c.epoch_start = c.restarts = 0;
        c.status = IGAOS_STATUS_ITERATION_LIMIT;
        c.asked = c.handed = c.have_pe = 0;
        c.last.pinf = c.last.dinf = c.last.gap = c.last.prow = CUDART_INF;
        c.last.op = 0.0;
    }
    // the averaging weight 2 / (h + 2), rounded from FP64; for h below 2^24 the
    // FP32 quotient is the same number (a quotient of such integers is never
    // within an FP64 rounding of the middle of two floats)
    auto weight = [](long long h) {
        return h < (1 << 24) - 2 ? 2.f / (float)(int)(h + 2) : (float)(2.0 / ((double)h + 2.0));
    };
    // factors 1 - k^-0.3 and 1 + k^-0.6 (src/pdhg/pdhg.cu:778-782), those of
    // the next iteration loaded while this one runs
    auto factors = [&](long long i, float& lo, float& hi) {
        lo = i < kFacTab ? a.fac[2 * i] : 1.f - powf((float)i, -0.3f);
        hi = i < kFacTab ? a.fac[2 * i + 1] : 1.f + powf((float)i, -0.6f);
    };
    float lo_now, hi_now, lo_next, hi_next;
    factors(1, lo_now, hi_now);
    factors(2, lo_next, hi_next);
    for (;;) {
        const float w_next = weight(hn + 1);
        const double flo = lo_now, fhi_eta = (double)hi_now * eta;
        cta_sync();
        cta_sync();
        // fixed-order merges over the warps that hold columns (rows), one
        // quantity per lane
        const double dx2 = merge_warps(sh.acc, warps_c);
        cta_sync();
        const double dot = merge_warps(sh.acc + 1 + (lane & 1), warps_r);
        const double dy2 = dot, cross = __shfl_sync(kFull, dot, 1);
        if (lane == 0) {
            // step decision (src/pdhg/pdhg.cu:770-794). num, cross, etabar and
            // the step sizes compare as integers: all are >= 0 there
            ++attempts;
            auto less_pos = [](double u, double v) {
                return __double_as_longlong(u) < __double_as_longlong(v);
            };
            const double num = fma(omega, dx2, div_by(dy2, omega, romega));
            const bool sound = dfinite(dx2) && dfinite(dy2) && dfinite(cross);
            double etabar = CUDART_INF, eta_new = CUDART_INF;
            const bool curved = sound && dfinite(num) && dgt0(num) && dgt0(cross);
            if (curved) {
                etabar = num / (2.0 * cross);
                const double up = flo * etabar;
                if (dfinite(etabar)) eta_new = less_pos(fhi_eta, up) ? fhi_eta : up;
            }
            const bool accept = !curved || !less_pos(etabar, eta) || retries >= 20;
            const bool usable = dfinite(eta_new) && less_pos(1e-12, eta_new);
            const double capped = less_pos(1e12, eta_new) ? 1e12 : eta_new;
            eta = usable ? (accept ? capped : eta_new) : (accept ? eta : fmax(eta_new, 1e-12));
            BatchStep& s = sh.step;
            if (!sound) {
                s.done = 1;
                c.status = IGAOS_STATUS_ERROR;
            }
            until -= accept;
            const int check = accept && sound && (until == 0 || k >= a.maxit);
            until = until == 0 ? a.check : until;
            retries = accept ? 0 : retries + 1;
            hn += accept;
            k += accept;
            if (accept) {
                s.parity ^= 1;
                s.w = w_next;
                lo_now = lo_next;
                hi_now = hi_next;
            }
            s.check = check;
            s.tau = (float)div_by(eta, omega, romega);
            s.sigma = (float)(eta * omega);
            if (accept) factors(k + 1, lo_next, hi_next);
        }
        cta_sync();
        if (sh.step.done) break;
        if (!sh.step.check) continue;
        const int pc = sh.step.parity;
        metrics<MODE, LONG>(a, d, pc, 1 << 30, workers, cmax, c.now);
        if (lane == 0) {
            const BMetrics &mc = c.now[0], &ma = c.now[1];
            const long long kd = k - 1;  // index of the iteration just accepted
            auto passes = [&](const BMetrics& u) {
                return u.pinf <= a.tol && u.dinf <= a.tol && u.prow <= a.tol && isfinite(u.gap) &&
                       u.gap <= a.tol;
            };
            const double ec = mc.finite ? mc.err : CUDART_INF;
            const double ea = ma.finite ? ma.err : CUDART_INF;
            BatchStep& s = sh.step;
            c.last = (ec <= ea) ? mc : ma;
            s.use_avg = ea < ec;
            s.restart = 0;
            if (passes(mc)) {
                c.last = mc;
                s.use_avg = 0;
                s.done = 1;
                c.status = IGAOS_STATUS_NEAR_OPTIMAL;
            } else if (passes(ma)) {
                c.last = ma;
                s.use_avg = 1;
                s.done = 1;
                c.status = IGAOS_STATUS_NEAR_OPTIMAL;
            } else if (kd >= a.maxit) {
                s.done = 1;
            } else if (kd >= a.handoff_at && !c.asked &&
                       (c.asked = 1, atomicAdd(a.handoff_count, 1u) < (unsigned)a.handoff_max)) {
                s.done = 1;  // left for the FP64 finish
                c.handed = 1;
            } else {
                const double cand = fmin(ec, ea);
                if (c.epoch_kkt < 0.0) {
                    c.epoch_kkt = cand;
                    c.prev_cand = cand;
                }
                const long long te = kd - c.epoch_start;
                s.restart = (isfinite(cand) && isfinite(c.epoch_kkt) && c.epoch_kkt > 0.0 &&
                             (cand <= 0.2 * c.epoch_kkt ||
                              (cand <= 0.8 * c.epoch_kkt && isfinite(c.prev_cand) && cand > c.prev_cand))) ||
                            (double)te >= 0.36 * (double)kd;
                c.prev_cand = cand;
                if (s.restart) {
                    hn = 0;
                    c.epoch_start = kd;
                    c.epoch_kkt = cand;
                    c.prev_cand = CUDART_INF;
                    ++c.restarts;
                }
            }
        }
        cta_sync();
        if (sh.step.done) break;
        if (sh.step.restart) {
            cta_sync();  // the anchor's movement is in sh.dred
            if (lane == 0) {
                double dxn = 0.0, dyn = 0.0;
                for (int v = 0; v < workers / 32; ++v) {
                    dxn += sh.dred[2 * v];
                    dyn += sh.dred[2 * v + 1];
                }
                if (c.have_pe && dxn > 1e-24 && dyn > 1e-24) {  // primal weight
                    const double om = sqrt(omega * sqrt(dyn / dxn));
                    if (isfinite(om) && om > 0.0) omega = fmin(fmax(om, 1e-6), 1e6);
                }
                c.have_pe = 1;
                romega = 1.0 / omega;
                sh.step.tau = (float)(eta / omega);
                sh.step.sigma = (float)(eta * omega);
                sh.step.w = weight(hn);
            }
            cta_sync();
        }
    }
    o.status = c.status;
    o.handed = c.handed;
    o.objective = c.last.op;
    o.pinf = c.last.pinf;
    o.dinf = c.last.dinf;
    o.gap = c.last.gap;
    o.prow = c.last.prow;
    o.iterations = k - 1;
    o.attempts = attempts;
    o.restarts = c.restarts;
}

template <int MODE, bool LONG>
__device__ __forceinline__ void solve_one(const BatchArgs& a, int b) {
    const long long t_begin = global_ns();
    BatchShared& sh = b_shared();
    const BatchDesc* dp = a.desc + b;
    const BatchDesc d = *dp;
    const int workers = min((int)blockDim.x - 32, kBT);
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool decider = threadIdx.x >= blockDim.x - 32;
    const int t = (int)threadIdx.x < workers ? (int)threadIdx.x : 1 << 30;
    const int m = d.m, n = d.n;
    const Held<MODE> W = make_work<MODE>(a, d);
    __shared__ float s_eta0, s_omega0;
    __shared__ double s_cmax;
    {
        const Inst I = make_inst(a, d);
        for (int j = t; j < n; j += workers) I.xh[j] = I.pesx[j] = 0.0;
        for (int i = t; i < m; i += workers) I.yh[i] = I.pesy[i] = 0.0;
    }
    if (threadIdx.x < 2) sh.longs[threadIdx.x] = threadIdx.x ? d.long_r : d.long_c;
    setup<LONG>(a, dp, t, workers, s_eta0, s_omega0);
    fill_work<MODE, LONG>(a, dp, workers);
    anchor_data<MODE, LONG>(a, dp, t, workers);
    {
        double cm = 0.0;
        for (int j = t; j < n; j += workers) cm = bmax(cm, fabs(a.c[d.col_off + j]));
        cm = warp_bmax(cm);
        if (lane == 0 && t < workers) sh.dred[wp] = cm;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < workers / 32; ++k) cm = bmax(cm, sh.dred[k]);
            s_cmax = cm;
        }
    }
    for (int j = t; j < n; j += workers) {
        W.x(0)[j] = W.xa(0)[j] = 0.f;
        W.g(0)[j] = 0.f;  // A~^T 0
    }
    for (int i = t; i < m; i += workers) W.y(0)[i] = W.ya(0)[i] = W.axc(0)[i] = 0.f;
    const double eta = s_eta0, omega = s_omega0;
    if (threadIdx.x == 0) {
        sh.step.tau = (float)(eta / omega);
        sh.step.sigma = (float)(eta * omega);
        sh.step.w = 1.f;
        sh.step.parity = sh.step.done = sh.step.check = sh.step.restart = sh.step.use_avg = 0;
    }
    __syncthreads();
    if (decider) {
        BatchOut o;
        decision_loop<MODE, LONG>(a, dp, workers, s_cmax, eta, omega, o);
        if (lane == 0) {
            o.ns = global_ns() - t_begin;
            a.out[b] = o;
        }
    } else {
        worker_loop<MODE, LONG>(a, dp, W, workers, s_cmax);
        const Inst I = make_inst(a, d);
        // answer: anchor + delta of the chosen candidate, original units
        const int pf = sh.step.parity;
        const float* xs = sh.step.use_avg ? W.xa(pf) : W.x(pf);
        const float* ys = sh.step.use_avg ? W.ya(pf) : W.y(pf);
        double* xo = a.x_out + d.col_off;
        double* yo = a.y_out + d.row_off;
        for (int j = t; j < n; j += workers) {
            const float xv = xs[j];
            xo[j] = xv == W.scl()[j]
                        ? I.cl[j]
                        : (xv == W.scu()[j] ? I.cu[j] : (I.xh[j] + (double)xv) * (double)I.dc[j]);
        }
        for (int i = t; i < m; i += workers) yo[i] = (I.yh[i] + (double)ys[i]) / (double)I.dr[i];
    }
    __syncthreads();
}

// Classes of instances: threads, CTAs per SM the kernel is compiled
// for, and the shared memory that leaves that many resident. An instance goes
// to the first class whose threads reach its columns and rows (or are kBT) and
// whose shared memory holds it; kTight takes the matrices without their vectors
// too, and the last class the instances in global memory: apart, because its
// CTAs leave their SM's memory to L1, which serves them. In one class with
// instances of 226 KB, 4,096 LPs of 20 to 2,000 rows took 18.5 s, 14.4 before
// classes; 11.6 now (an iteration of an LP of 1,886 rows 98 us before, now 52).
// Instances with long rows (LONG: slices laid in steps, rows that a warp takes in the
// setup) have the same classes again, as kernels of their own: in one kernel with the
// others, their code cost the others' loops registers (150 LPs of 30 to 400 rows 182
// -> 190 ms).
struct BatchClass {
    int threads, ctas;  // threads: without the decision warp
    size_t smem;
};
constexpr int kShapes = 5, kTight = 3, kClasses = 2 * kShapes;
constexpr BatchClass kClass[kShapes] = {{128, 6, 36 * 1024},
                                         {256, 4, 55 * 1024},
                                         {512, 2, 112 * 1024},
                                         {512, 1, 226 * 1024},
                                         {512, 1, 110 * 1024}};

size_t held_bytes(const BatchDesc& d, int mode) {
    return kSharedHead +
           (mode == kHeldWide  ? 0
            : mode == kHeldOut ? 4 * ((size_t)d.n + 2 * (size_t)d.m)
                               : matrix_bytes(d) + (mode == kHeldAll ? state_bytes(d) : 0));
}

// Rows by decreasing length into `order` (counting sort, stable), the first
// staged entry of each slice of 32 (then the total), in units of 32, onto `bases`,
// the slices laid in steps (where pads would take twice as much, if `steps`) onto
// `longs`; returns the entries.
long long sort_slices(const std::vector<int>& len, int* order, std::vector<int>& bases,
                      std::vector<int>& longs, bool steps) {
    const int rows = (int)len.size();
    int longest = 0;
    for (int l : len) longest = std::max(longest, l);
    std::vector<int> start(longest + 2, 0);
    for (int l : len) ++start[longest - l + 1];
    for (int k = 0; k <= longest; ++k) start[k + 1] += start[k];
    for (int r = 0; r < rows; ++r) order[start[longest - len[r]]++] = r;
    int run = 0;
    const size_t first = longs.size();
    std::vector<int> units;  // of the slices laid in steps
    for (int q = 0; q < rows; q += 32) {
        const int in = std::min(32, rows - q), padded = len[order[q]];
        bases.push_back(run);
        if (steps) {
            long long entries = 0;
            for (int st = 0, k = 0; st < kSteps; ++st) {
                const int lane = step_lane(st), to = lane < in ? len[order[q + lane]] : 0;
                entries += (long long)(32 >> st) * (to - k);
                k = to;
            }
            const long long u = 1 + (entries + 31) / 32;
            if (2 * u <= padded) {
                longs.push_back(q / 32);
                longs.push_back(0);
                units.push_back((int)u);
                continue;
            }
        }
        run += padded;
    }
    bases.push_back(run);
    run += (int)((longs.size() - first + 31) / 32);  // the table
    for (size_t i = 0; i < units.size(); ++i) {
        longs[first + 2 * i + 1] = run;
        run += units[i];
    }
    return 32LL * run;
}

// How a batch is staged and dealt to the classes: each instance's sorted slices,
// its mode and class.
struct BatchPlan {
    std::vector<int> order_c, order_r, bases, longs, cls;
    long long out_entries = 0;  // staged in global memory
    size_t smem[kClasses] = {};
};
BatchPlan plan_batch(const int* ap, const int* ai, std::vector<BatchDesc>& desc, long long rows,
                     long long cols) {
    BatchPlan P;
    P.order_c.resize(cols);
    P.order_r.resize(rows);
    P.cls.resize(desc.size());
    std::vector<int> len_c, len_r;
    for (size_t b = 0; b < desc.size(); ++b) {
        BatchDesc& d = desc[b];
        len_c.assign(d.n, 0);
        for (int p = 0; p < d.nnz; ++p) ++len_c[ai[d.nz_off + p]];
        len_r.resize(d.m);
        for (int i = 0; i < d.m; ++i) len_r[i] = ap[d.ap_off + i + 1] - ap[d.ap_off + i];
        auto longer = [](const std::vector<int>& len) {
            return (int)std::count_if(len.begin(), len.end(), [](int l) { return l > kLongRow; });
        };
        d.longer_c = longer(len_c);
        d.longer_r = longer(len_r);
        d.base_off = (long long)P.bases.size();
        d.long_c_at = (long long)P.longs.size();
        auto stage = [&](bool steps) {
            P.bases.resize(d.base_off);
            P.longs.resize(d.long_c_at);
            d.pad_c = sort_slices(len_c, P.order_c.data() + d.col_off, P.bases, P.longs, steps);
            d.long_r_at = (long long)P.longs.size();
            d.pad_r = sort_slices(len_r, P.order_r.data() + d.row_off, P.bases, P.longs, steps);
            d.long_c = (int)(d.long_r_at - d.long_c_at) / 2;
            d.long_r = (int)((long long)P.longs.size() - d.long_r_at) / 2;
        };
        const int reach = std::max(d.m, d.n);
        auto deal = [&]() {  // its mode, and the class returned
            int k = 0;
            d.mode = kHeldAll;
            while (k < kTight && ((reach > kClass[k].threads && kClass[k].threads < kBT) ||
                                  held_bytes(d, kHeldAll) > kClass[k].smem))
                ++k;
            while (held_bytes(d, d.mode) > kClass[k].smem) --d.mode;
            if (d.mode > kHeldOut) return k;
            k = kShapes - 1;
            if (held_bytes(d, kHeldOut) > kClass[k].smem || reach > 0xffff) d.mode = kHeldWide;
            return k;
        };
        // Steps only where pads cost a mode, an SM to itself or space and loads in
        // global memory (a 500 x 1,250 LP of 7,500 nonzeros with one full row: 112
        // KB, 335 with pads, which no CTA has; its iteration 60 us with pads, 34 in
        // steps): a short step costs a warp more than its pads. 512 LPs of 20 to 120
        // rows with one full row: 40 ms padded, at two CTAs per SM, 43 in steps, at
        // four.
        stage(true);
        int k = deal();
        if (d.long_c + d.long_r > 0) {
            const int mode = d.mode;
            stage(false);
            const int padded = deal();
            const bool alone = kClass[padded].ctas == 1 && kClass[k].ctas > 1;
            if (d.mode < mode || d.mode <= kHeldOut || alone) stage(true);
            k = deal();
        }
        if (d.mode <= kHeldOut) {
            d.out_off = P.out_entries;
            P.out_entries += d.pad_c + d.pad_r;
        }
        if (d.longer_c + d.longer_r + d.long_c + d.long_r > 0) k += kShapes;
        P.cls[b] = k;
        P.smem[k] = std::max(P.smem[k], held_bytes(d, d.mode));
    }
    return P;
}

template <int K>
__global__ void __launch_bounds__(kClass[K % kShapes].threads + 32, kClass[K % kShapes].ctas)
    k_batch(const __grid_constant__ BatchArgs a) {
    BatchShared& sh = b_shared();
    for (;;) {
        if (threadIdx.x == 0) sh.inst = (int)atomicAdd(a.queue, 1u);
        __syncthreads();
        const int qi = sh.inst;
        __syncthreads();
        if (qi >= a.count) break;
        const int b = a.order[qi];
        if (a.desc[b].m <= 0 || a.desc[b].n <= 0) continue;
        constexpr int S = K % kShapes;
        constexpr bool LONG = K >= kShapes;
        if constexpr (S < kTight) {
            solve_one<kHeldAll, LONG>(a, b);
        } else if constexpr (S == kTight) {
            if (a.desc[b].mode == kHeldAll) solve_one<kHeldAll, LONG>(a, b);
            else solve_one<kHeldMatrix, LONG>(a, b);
        } else {
            if (a.desc[b].mode == kHeldOut) solve_one<kHeldOut, LONG>(a, b);
            else solve_one<kHeldWide, LONG>(a, b);
        }
    }
}

__global__ void k_to_float(long long n, const double* __restrict__ in, float* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

}  // namespace
}  // namespace igx

// Class, mode (kHeldWide ..) and staged entries of each instance of a batch. For
// tests; not in the public header.
extern "C" void igx_batch_plan(int count, const int* m, const int* n, const int* ap, const int* ai,
                               int* cls, int* mode, long long* entries) {
    using namespace igx;
    std::vector<BatchDesc> desc(count);
    long long ap_off = 0, nz = 0, rows = 0, cols = 0;
    for (int b = 0; b < count; ++b) {
        BatchDesc& d = desc[b];
        d = BatchDesc{};
        d.m = m[b];
        d.n = n[b];
        d.nnz = ap[ap_off + m[b]];
        d.ap_off = ap_off;
        d.nz_off = nz;
        d.row_off = rows;
        d.col_off = cols;
        ap_off += d.m + 1;
        nz += d.nnz;
        rows += d.m;
        cols += d.n;
    }
    const BatchPlan plan = plan_batch(ap, ai, desc, rows, cols);
    for (int b = 0; b < count; ++b) {
        cls[b] = plan.cls[b];
        mode[b] = desc[b].mode;
        entries[b] = desc[b].pad_c + desc[b].pad_r;
    }
}

// ---------------------------------------------------------------- C ABI
extern "C" int igaos_pdhg_solve_batch(int count, const int* m, const int* n, const int* ap,
                                      const int* ai, const double* ax, const double* c,
                                      const double* cl, const double* cu, const double* rmin,
                                      const double* rmax, const igaos_pdhg_options* opt,
                                      igaos_pdhg_batch_result* res, double* x, double* y) {
    using namespace igx;
    if (count <= 0 || !m || !n || !ap || !ai || !ax || !c || !cl || !cu || !rmin || !rmax || !res)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "count must be positive and arrays non-NULL");
    igaos_pdhg_options o;
    if (opt) o = *opt;
    else igaos_pdhg_default_options(&o);
    if (!(o.tolerance > 0)) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "tolerance must be positive");
    try {
        auto t_start = std::chrono::steady_clock::now();
        // host descriptors, validation
        std::vector<BatchDesc> desc(count);
        long long ap_off = 0, nz = 0, rows = 0, cols = 0;
        for (int b = 0; b < count; ++b) {
            if (m[b] < 0 || n[b] < 0)
                return igx_set_error(IGAOS_PDHG_ERR_INVALID, "negative instance size");
            BatchDesc& d = desc[b];
            d.m = m[b];
            d.n = n[b];
            const int* bap = ap + ap_off;
            if (bap[0] != 0)
                return igx_set_error(IGAOS_PDHG_ERR_INVALID, "each instance's row pointer must start at 0");
            for (int i = 0; i < d.m; ++i)
                if (bap[i + 1] < bap[i])
                    return igx_set_error(IGAOS_PDHG_ERR_INVALID, "row pointer must be non-decreasing");
            d.nnz = bap[d.m];
            for (int p = 0; p < d.nnz; ++p) {
                const int j = ai[nz + p];
                if (j < 0 || j >= d.n)
                    return igx_set_error(IGAOS_PDHG_ERR_INVALID, "column index out of range");
                if (!std::isfinite(ax[nz + p]))
                    return igx_set_error(IGAOS_PDHG_ERR_INVALID, "matrix values must be finite");
            }
            d.ap_off = ap_off;
            d.cp_off = cols + b;
            d.nz_off = nz;
            d.row_off = rows;
            d.col_off = cols;
            ap_off += d.m + 1;
            nz += d.nnz;
            rows += d.m;
            cols += d.n;
        }
        for (long long j = 0; j < cols; ++j) {
            if (!std::isfinite(c[j])) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "cost must be finite");
            if (std::isnan(cl[j]) || std::isnan(cu[j]) || cl[j] > cu[j])
                return igx_set_error(IGAOS_PDHG_ERR_INVALID, "bad column bounds");
        }
        for (long long i = 0; i < rows; ++i)
            if (std::isnan(rmin[i]) || std::isnan(rmax[i]) || rmin[i] > rmax[i])
                return igx_set_error(IGAOS_PDHG_ERR_INVALID, "bad row bounds");
        if (igaos_pdhg_device_count() == 0)
            return igx_set_error(IGAOS_PDHG_ERR_NODEVICE, "no CUDA device: PDHG engine unavailable");
        if (o.device >= 0) CU(cudaSetDevice(o.device));
        // largest instances first
        std::vector<int> order(count);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int p1, int p2) {
            return (long long)desc[p1].nnz + desc[p1].m + desc[p1].n >
                   (long long)desc[p2].nnz + desc[p2].m + desc[p2].n;
        });
        // sorted slices and classes, each in that order
        const BatchPlan plan = plan_batch(ap, ai, desc, rows, cols);
        std::vector<int> cls_order;
        int cls_count[kClasses] = {}, cls_first[kClasses] = {};
        for (int k = kClasses - 1; k >= 0; --k) {
            cls_first[k] = (int)cls_order.size();
            for (int b : order)
                if (plan.cls[b] == k) cls_order.push_back(b);
            cls_count[k] = (int)cls_order.size() - cls_first[k];
        }
        // constants, the same for every call: 131,072 powers take 5 ms
        static const std::vector<float> fac = [] {
            std::vector<float> f(2 * kFacTab);
            for (int k = 0; k < kFacTab; ++k) {
                const double kk = k < 1 ? 1.0 : (double)k;
                f[2 * k] = (float)(1.0 - std::pow(kk, -0.3));
                f[2 * k + 1] = (float)(1.0 + std::pow(kk, -0.6));
            }
            return f;
        }();
        cudaStream_t st;
        CU(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        struct StreamGuard {
            cudaStream_t s;
            ~StreamGuard() { cudaStreamDestroy(s); }
        } sg{st};
        Arena ar;
        // 40 bytes per entry, 128 per column and 112 per row, the staged entries, the
        // tables; 50 roundings
        ar.expect((size_t)nz * 40 + (size_t)cols * 128 + (size_t)rows * 112 +
                  (size_t)plan.out_entries * 8 + (plan.bases.size() + plan.longs.size()) * sizeof(int) +
                  (size_t)count * (sizeof(BatchDesc) + sizeof(BatchOut) + 16) +
                  sizeof(float) * fac.size() + 64 * 256);
        auto up = [&](const auto* h, size_t len) {
            using V = std::remove_const_t<std::remove_pointer_t<decltype(h)>>;
            V* dp = ar.alloc<V>(len);
            CU(cudaMemcpyAsync(dp, h, sizeof(V) * len, cudaMemcpyHostToDevice, st));
            return dp;
        };
        BatchArgs A{};
        const int* d_order = up(cls_order.data(), cls_order.size());
        A.desc = up(desc.data(), desc.size());
        unsigned int* queue = ar.alloc<unsigned int>(kClasses);
        CU(cudaMemsetAsync(queue, 0, kClasses * sizeof(unsigned int), st));
        A.ap = up(ap, (size_t)ap_off);
        A.ai = up(ai, (size_t)nz);
        double* axd = up(ax, (size_t)nz);
        float* axf = ar.alloc<float>(nz);
        k_to_float<<<1216, 256, 0, st>>>(nz, axd, axf);
        A.ax = axf;
        A.axd = axd;
        A.c = up(c, cols);
        A.cl = up(cl, cols);
        A.cu = up(cu, cols);
        A.rmin = up(rmin, rows);
        A.rmax = up(rmax, rows);
        A.cp = ar.alloc<int>(cols + count);
        A.ci = ar.alloc<int>(nz);
        A.cnt = ar.alloc<int>(cols);
        A.cax = ar.alloc<float>(nz);
        A.cax64 = ar.alloc<double>(nz);
        A.sax = ar.alloc<float>(nz);
        A.scax = ar.alloc<float>(nz);
        float** colv[] = {&A.dc, &A.sc, &A.scl, &A.scu, &A.x[0], &A.x[1], &A.xa[0], &A.xa[1],
                          &A.xbar, &A.vt, &A.g[0], &A.g[1]};
        A.order_c = up(plan.order_c.data(), plan.order_c.size());
        A.order_r = up(plan.order_r.data(), plan.order_r.size());
        A.bases = up(plan.bases.data(), plan.bases.size());
        A.longs = up(plan.longs.data(), plan.longs.size());
        A.out_val = ar.alloc<float>(plan.out_entries);
        A.out_idx = ar.alloc<int>(plan.out_entries);
        for (float** v : colv) *v = ar.alloc<float>(cols);
        float** rowv[] = {&A.dr, &A.srmin, &A.srmax, &A.yh32, &A.y[0], &A.y[1], &A.ya[0],
                          &A.ya[1], &A.axc[0], &A.axc[1], &A.mt, &A.ab};
        for (float** v : rowv) *v = ar.alloc<float>(rows);
        double** col64[] = {&A.xh, &A.pesx, &A.atyh, &A.rdc};
        for (double** v : col64) *v = ar.alloc<double>(cols);
        double** row64[] = {&A.yh, &A.pesy, &A.axh, &A.rdr};
        for (double** v : row64) *v = ar.alloc<double>(rows);
        A.fac = up(fac.data(), fac.size());
        A.tol = o.tolerance;
        // per-instance iteration cap (the kernel has no wall clock)
        A.maxit = (long long)std::max<int64_t>(1, o.max_iterations);
        // hand-off: 100,000 iterations and 16 instances unless overridden
        // (IGAOS_PDHG_BATCH_HANDOFF=iterations, 0 = never;
        // IGAOS_PDHG_BATCH_HANDOFF_MAX=instances)
        {
            const char* e = std::getenv("IGAOS_PDHG_BATCH_HANDOFF");
            const long long h = e && *e ? std::atoll(e) : 100000;
            A.handoff_at = h > 0 ? h : A.maxit;
            const char* em = std::getenv("IGAOS_PDHG_BATCH_HANDOFF_MAX");
            A.handoff_max = em && *em ? std::max(0, std::atoi(em)) : 16;
        }
        A.handoff_count = ar.alloc<unsigned int>(1);
        CU(cudaMemsetAsync(A.handoff_count, 0, sizeof(unsigned int), st));
        A.check = o.check_period > 0 ? o.check_period : 64;
        // every instance's answer (the FP64 finish starts from it)
        A.x_out = ar.alloc<double>(cols);
        A.y_out = ar.alloc<double>(rows);
        A.out = ar.alloc<BatchOut>(count);
        int sms = 0, dev = 0;
        CU(cudaGetDevice(&dev));
        CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        // one persistent launch per class, the largest instances' first; the
        // others beside it on their own streams, taking the SMs it leaves
        struct Fork {
            cudaStream_t s[kClasses] = {};
            cudaEvent_t e[kClasses + 2] = {};
            ~Fork() {
                for (auto& v : s)
                    if (v) cudaStreamDestroy(v);
                for (auto& v : e)
                    if (v) cudaEventDestroy(v);
            }
        } fk;
        CU(cudaEventCreate(&fk.e[kClasses]));
        CU(cudaEventCreate(&fk.e[kClasses + 1]));
        CU(cudaEventRecord(fk.e[kClasses], st));
        void (*const kernels[kClasses])(BatchArgs) = {
            k_batch<0>, k_batch<1>, k_batch<2>, k_batch<3>, k_batch<4>,
            k_batch<5>, k_batch<6>, k_batch<7>, k_batch<8>, k_batch<9>};
        bool first = true;
        for (int i = 0; i < kClasses; ++i) {
            const int k = kShapes - 1 - i / 2 + (i % 2 ? 0 : kShapes);
            if (cls_count[k] == 0) continue;
            cudaStream_t sk = st;
            if (!first) {
                CU(cudaStreamCreateWithFlags(&fk.s[k], cudaStreamNonBlocking));
                sk = fk.s[k];
                CU(cudaStreamWaitEvent(sk, fk.e[kClasses], 0));
            }
            const BatchClass& shape = kClass[k % kShapes];
            const int threads = shape.threads + 32;
            int per_sm = 0;
            CU(cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)shape.smem));
            CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernels[k], threads,
                                                             plan.smem[k]));
            BatchArgs Ak = A;
            Ak.count = cls_count[k];
            Ak.order = d_order + cls_first[k];
            Ak.queue = queue + k;
            const int grid = std::min(cls_count[k], sms * std::max(1, per_sm));
            kernels[k]<<<grid, threads, plan.smem[k], sk>>>(Ak);
            CU(cudaGetLastError());
            if (!first) {
                CU(cudaEventCreateWithFlags(&fk.e[k], cudaEventDisableTiming));
                CU(cudaEventRecord(fk.e[k], sk));
                CU(cudaStreamWaitEvent(st, fk.e[k], 0));
            }
            first = false;
        }
        CU(cudaEventRecord(fk.e[kClasses + 1], st));
        std::vector<BatchOut> out(count);
        CU(cudaMemcpyAsync(out.data(), A.out, sizeof(BatchOut) * count, cudaMemcpyDeviceToHost, st));
        std::vector<double> xk, yk;  // the launch's answers when the caller wants none
        if (!x) {
            xk.resize(cols);
            x = xk.data();
        }
        if (!y) {
            yk.resize(rows);
            y = yk.data();
        }
        CU(cudaMemcpyAsync(x, A.x_out, sizeof(double) * cols, cudaMemcpyDeviceToHost, st));
        CU(cudaMemcpyAsync(y, A.y_out, sizeof(double) * rows, cudaMemcpyDeviceToHost, st));
        CU(cudaStreamSynchronize(st));
        float kms = 0.f;
        CU(cudaEventElapsedTime(&kms, fk.e[kClasses], fk.e[kClasses + 1]));
        // Instances the launch handed off or left at the cap are solved again,
        // alone, by the single-LP engine in FP64 through the public entry
        // points, from the launch's answer (igaos_pdhg_set_start), with the
        // same tolerance and cap; up to 8 at once, each on its own host
        // thread, engine and stream.
        std::vector<igaos_pdhg_result> fin(count);
        std::vector<char> redo(count, 0);
        std::vector<double> fin_ms(count, 0.0);
        std::vector<int> todo;
        for (int b = 0; b < count; ++b)
            if (out[b].status == IGAOS_STATUS_ITERATION_LIMIT && desc[b].m > 0 && desc[b].n > 0)
                todo.push_back(b);
        std::vector<int> fin_rc(count, IGAOS_PDHG_OK);
        std::vector<std::string> fin_msg(count);
        std::atomic<size_t> next{0};
        auto finish = [&]() {
            CU(cudaSetDevice(dev));
            for (size_t t; (t = next.fetch_add(1)) < todo.size();) {
                const int b = todo[t];
                const BatchDesc& d = desc[b];
                igaos_pdhg_options o64 = o;
                o64.precision = IGAOS_PDHG_FP64;
                o64.time_limit_s = 1e9;  // the cap binds, as in the launch
                o64.pdhg_presolve = 0;
                o64.crossover = 0;
                const auto t1 = std::chrono::steady_clock::now();
                igaos_pdhg_problem* P = nullptr;
                int rc = igaos_pdhg_create(&P, d.m, d.n, d.nnz, ap + d.ap_off, ai + d.nz_off,
                                           ax + d.nz_off, nullptr, nullptr, nullptr, c + d.col_off,
                                           cl + d.col_off, cu + d.col_off, rmin + d.row_off,
                                           rmax + d.row_off, 0.0, &o64);
                if (rc == IGAOS_PDHG_OK)
                    rc = igaos_pdhg_set_start(P, x + d.col_off, y + d.row_off);
                if (rc == IGAOS_PDHG_OK)
                    rc = igaos_pdhg_solve(P, &o64, &fin[b], x + d.col_off, y + d.row_off);
                igaos_pdhg_destroy(P);
                fin_rc[b] = rc;
                if (fin_rc[b] != IGAOS_PDHG_OK) {
                    char msg[512];
                    igaos_pdhg_last_error(msg, sizeof(msg));
                    fin_msg[b] = msg;
                }
                fin_ms[b] = std::chrono::duration<double, std::milli>(
                                std::chrono::steady_clock::now() - t1).count();
                redo[b] = 1;
            }
        };
        int nthreads = 8;
        if (const char* e = std::getenv("IGAOS_PDHG_BATCH_FINISH_THREADS"))
            nthreads = std::max(1, std::atoi(e));
        nthreads = (int)std::min<size_t>((size_t)nthreads, todo.size());
        if (nthreads == 1) {
            finish();
        } else if (nthreads > 1) {
            std::vector<std::thread> pool;
            std::vector<std::exception_ptr> errs(nthreads);
            for (int i = 0; i < nthreads; ++i)
                pool.emplace_back([&, i] {
                    try {
                        finish();
                    } catch (...) {
                        errs[i] = std::current_exception();
                    }
                });
            for (auto& th : pool) th.join();
            for (auto& e : errs)
                if (e) std::rethrow_exception(e);
        }
        for (int b : todo)
            if (fin_rc[b] != IGAOS_PDHG_OK) return igx_set_error(fin_rc[b], fin_msg[b].c_str());
        const double wall = std::chrono::duration<double, std::milli>(
                                std::chrono::steady_clock::now() - t_start).count();
        for (int b = 0; b < count; ++b) {
            igaos_pdhg_batch_result& r = res[b];
            const BatchOut& q = out[b];
            r.status = (desc[b].m > 0 && desc[b].n > 0) ? q.status : IGAOS_STATUS_ERROR;
            r.finished_fp64 = 0;
            r.objective = q.objective;
            r.pinf = q.pinf;
            r.dinf = q.dinf;
            r.rel_gap = q.gap;
            r.prow = q.prow;
            r.iterations = q.iterations;
            r.attempts = q.attempts;
            r.restarts = q.restarts;
            r.kernel_time_ms = kms;
            r.total_time_ms = wall;
            r.instance_time_ms = 1e-6 * (double)q.ns;
            if (redo[b]) {
                const igaos_pdhg_result& f = fin[b];
                r.finished_fp64 = 1;
                r.status = f.status;
                r.objective = f.objective;
                r.pinf = f.pinf;
                r.dinf = f.dinf;
                r.rel_gap = f.rel_gap;
                r.prow = f.prow;
                r.iterations += f.iterations;
                r.attempts += f.attempts;
                r.restarts += f.restarts;
                r.instance_time_ms += fin_ms[b];
            }
        }
    } catch (const CudaError& e) {
        return igx_set_error(e.code, e.what());
    } catch (const std::exception& e) {
        return igx_set_error(IGAOS_PDHG_ERR_CUDA, e.what());
    }
    return igx_set_error(IGAOS_PDHG_OK, "");
}
