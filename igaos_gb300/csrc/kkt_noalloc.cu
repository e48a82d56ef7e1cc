// Allocation-free FP64 KKT evaluation (igaos_pdhg_evaluate_noalloc).
//
// For callers that cannot call cudaMalloc: code whose device memory is owned
// by a framework allocator or a fixed pool sized up front, or that runs where
// an allocation (which can synchronise the device) is not acceptable, such
// as a latency-bound serving loop. They pass every input and the output as
// device buffers they already own; the kernels' scratch (per-CTA partials,
// the metric accumulators, the last-CTA counters) lives in one file-scope
// __device__ array that every GPU loading this library holds until the
// process exits.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

#include "device.cuh"
#include "engine.hpp"

namespace igx {
namespace {

constexpr int kNaMaxCtas = 1024;  // resident ones take rows and columns in strides
constexpr int kNaMaxDim = 1 << 22;  // a limit of the interface, not of the scratch

struct NaScratch {
    double part[kNaMaxCtas * 8];  // per-CTA partials of the current pass
    DevMetrics met;               // accumulated metrics
    double cmax;                  // max |c_j|
    unsigned int ticket[2];       // last-CTA counters (must start at zero)
};

// 64 KiB + a few bytes of device memory, per device that loads the library.
static __device__ __align__(256) NaScratch g_na_scratch;

constexpr int kMaxDevices = 64;
std::mutex g_na_mu;
NaScratch* g_na_ptr[kMaxDevices] = {};
int g_na_sms[kMaxDevices] = {};

// a < b and max(a, b) with the outcome of the FP64 instructions for every
// operand (false, and a, when either is NaN) on the integer pipe: the FP64
// pipe (2 operations per clock per SM) is what the products need.
__device__ __forceinline__ bool na_nan(double a) {
    return ((unsigned long long)__double_as_longlong(a) << 1) > 0xffe0000000000000ULL;
}
__device__ __forceinline__ bool na_lt(double a, double b) {
    return dlt(a, b) && !na_nan(a) && !na_nan(b);
}
__device__ __forceinline__ double na_max(double a, double b) { return na_lt(a, b) ? b : a; }
__device__ __forceinline__ double na_min(double a, double b) { return na_lt(b, a) ? b : a; }

// One pass over the rows of a warp: G = 2^lg lanes share a row with entries
// [b, e), `steps` entries per lane (uniform in the warp, so that no FP64
// instruction is issued for slots past the longest row), four loads of each
// kind in flight. Every lane of a group gets its row's sum.
__device__ __forceinline__ double na_dot(const int* __restrict__ idx,
                                         const double* __restrict__ val,
                                         const double* __restrict__ x, int b, int e, int lg,
                                         int steps) {
    const int G = 1 << lg, gl = (threadIdx.x & 31) & (G - 1);
    double s = 0.0;
    int p = b + gl;
    for (int k = 0; k < steps; k += 4, p += 4 * G) {
        const int left = steps - k;
        double a[4], xv[4];
        int j[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int q = p + u * G;
            j[u] = q < e ? __ldcs(idx + q) : -1;
            a[u] = q < e ? __ldcs(val + q) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) xv[u] = j[u] >= 0 ? __ldg(x + j[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (u < left) s = fma(a[u], xv[u], s);
    }
    for (int o = G >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
    return s;
}

struct NaRow {
    int row;     // index in [0, nr), or -1
    double sum;  // of that row
};

// Row sums of rows [r0, r0 + nr), nr <= 32, by one warp: lane i gets the sum
// of the i-th longest. An FP64 instruction occupies the FP64 pipe for the
// whole warp whatever its active lanes, so rows of like length go together:
// the warp sorts its rows by length (integer keys) and takes them longest
// first, G lanes per row from the longest row of the pass at about eight
// entries per lane. In file order with one G per warp, columns of mixed length
// (a Zipf tail among short ones) issued more of them: 128 us against 86 us for
// 500,000 columns of 5 M entries (80 us with the block sums as they are now).
__device__ __forceinline__ NaRow na_row_sums(const int* __restrict__ ptr,
                                             const int* __restrict__ idx,
                                             const double* __restrict__ val,
                                             const double* __restrict__ x, int r0, int nr) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    int b = 0, e = 0;
    if (lane < nr) {
        b = __ldg(ptr + r0 + lane);
        e = __ldg(ptr + r0 + lane + 1);
    }
    // bitonic sort, longest first; lanes without a row (key -1) come last
    long long key = lane < nr ? ((long long)(e - b) << 5 | lane) : -1;
    for (int k = 2; k <= 32; k <<= 1)
        for (int o = k >> 1; o > 0; o >>= 1) {
            const long long other = __shfl_xor_sync(full, key, o);
            const bool larger = ((lane & o) == 0) == ((lane & k) == 0);
            key = larger == (key > other) ? key : other;
        }
    const int row = key < 0 ? -1 : (int)(key & 31);
    const int len = key < 0 ? 0 : (int)(key >> 5);
    b = __shfl_sync(full, b, row & 31);
    NaRow r{row, 0.0};
    for (int q0 = 0; q0 < nr;) {
        const int longest = __shfl_sync(full, len, q0);
        if (longest == 0) break;
        int lg = 0;
        while (lg < 5 && (8 << lg) < longest) ++lg;
        const int q = q0 + (lane >> lg);
        const int qb = __shfl_sync(full, b, q & 31), ql = __shfl_sync(full, len, q & 31);
        const int qe = q < nr ? qb + ql : qb;
        const double s = na_dot(idx, val, x, qb, qe, lg, (longest + (1 << lg) - 1) >> lg);
        const double v = __shfl_sync(full, s, ((lane - q0) << lg) & 31);
        const int per = 32 >> lg;
        if (lane >= q0 && lane < q0 + per) r.sum = v;
        q0 += per;
    }
    return r;
}

// Row pass: A x in original units -> pinf numerator/normaliser, prow,
// max |y|; also max |c| (grid-stride over columns).
// Bound by the random gathers of x through L2 (one 32-byte sector per entry)
// and the FP64 pipe (53 % busy here, 70 % in the column pass). A warp used to
// take a row with all its lanes and 32 rows in series, one dependent load
// chain after another: on a 200,000 x 500,000 LP of 5 M entries 569 us, and
// 691 us for the column pass; now 57 and 80 us, and a call 1,286 -> 122 us.
__global__ void __launch_bounds__(kThreads, 4) na_rows(int m, int n, int per_warp,
                                                    const int* __restrict__ ap,
                                                    const int* __restrict__ ai,
                                                    const double* __restrict__ ax,
                                                    const double* __restrict__ x,
                                                    const double* __restrict__ y,
                                                    const double* __restrict__ c,
                                                    const double* __restrict__ rmin,
                                                    const double* __restrict__ rmax,
                                                    NaScratch* s) {
    __shared__ double red[kWarps * 8];
    // the column pass may start as this one drains: it waits before it uses
    // anything written here
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    double pv = 0.0, pa = 0.0, prow = 0.0, ymax = 0.0, cmax = 0.0;
    const int step = gridDim.x * kWarps * per_warp;
    for (int r0 = (blockIdx.x * kWarps + (int)(threadIdx.x >> 5)) * per_warp; r0 < m; r0 += step) {
        const NaRow R = na_row_sums(ap, ai, ax, x, r0, min(per_warp, m - r0));
        if (R.row >= 0) {
            const int i = r0 + R.row;
            const double Ax = R.sum;
            const double lo = rmin[i], hi = rmax[i];
            const double vi = na_max(lo - Ax, Ax - hi);
            pv = na_max(pv, vi);
            pa = na_max(pa, dabs(na_min(na_max(Ax, lo), hi)));
            if (na_lt(0.0, vi)) {  // the FP64 division only where it can count
                double sc = dabs(Ax);
                if (dfinite(lo)) sc = na_max(sc, dabs(lo));
                if (dfinite(hi)) sc = na_max(sc, dabs(hi));
                prow = na_max(prow, vi / (1.0 + sc));
            }
            ymax = na_max(ymax, dabs(y[i]));
        }
    }
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        cmax = na_max(cmax, dabs(c[j]));
    double r[5] = {pv, pa, prow, ymax, cmax};
    block_dmax<5>(r, red);
    if (threadIdx.x == 0)
        for (int q = 0; q < 5; ++q) s->part[blockIdx.x * 8 + q] = r[q];
    if (!last_cta(&s->ticket[0])) return;
    double t[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads)
        for (int q = 0; q < 5; ++q) t[q] = dmax(t[q], s->part[b * 8 + q]);
    block_dmax<5>(t, red);
    if (threadIdx.x == 0) {
        s->met.pv = t[0];
        s->met.pa = t[1];
        s->met.pinf = smax(t[0], 0.0) / (1.0 + t[1]);
        s->met.prow = t[2];
        s->met.ymax = t[3];
        s->cmax = t[4];
        s->ticket[1] = 0u;  // whatever calls that overlapped have left there
    }
}

// Column pass: d = c + A^T y -> dinf, c^T x, column part of the dual bound;
// then the row part of the bound (its noise threshold needs max |y|) and, in
// the last CTA, the final metrics.
__global__ void __launch_bounds__(kThreads, 4) na_cols(int m, int n, int per_warp,
                                                    const int* __restrict__ cp,
                                                    const int* __restrict__ ci,
                                                    const double* __restrict__ acx,
                                                    const double* __restrict__ x,
                                                    const double* __restrict__ y,
                                                    const double* __restrict__ c,
                                                    const double* __restrict__ cl,
                                                    const double* __restrict__ cu,
                                                    const double* __restrict__ rmin,
                                                    const double* __restrict__ rmax, NaScratch* s,
                                                    double* out6) {
    __shared__ double red[kWarps * 8];
    const int step = gridDim.x * kWarps * per_warp;
    int j0 = (blockIdx.x * kWarps + (int)(threadIdx.x >> 5)) * per_warp;
    NaRow C{-1, 0.0};
    if (j0 < n) C = na_row_sums(cp, ci, acx, y, j0, min(per_warp, n - j0));
    // the row pass (its maxima, and the partials' space) is complete from here
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0 && threadIdx.x == 0) s->ticket[0] = 0u;
    const double cmax = __ldcg(&s->cmax);
    const double dz = 1e-8 * (1.0 + cmax);
    double dv = 0.0, op = 0.0, od = 0.0, unb = 0.0;
    while (j0 < n) {
        if (C.row >= 0) {
            const int j = j0 + C.row;
            const double d = c[j] + C.sum, xj = x[j], lo = cl[j], hi = cu[j];
            const double bnd = dabs(dfinite(hi) ? hi : lo);
            const double tol = 1e-9 * (1.0 + bnd);
            const double lob = lo + tol, hib = hi - tol;
            const bool at_lo = na_lt(xj, lob) || xj == lob, at_hi = na_lt(hib, xj) || xj == hib;
            if (!(at_lo && na_lt(0.0, d)) && !(at_hi && na_lt(d, 0.0))) dv = na_max(dv, dabs(d));
            op = fma(c[j], xj, op);
            if (d >= 0) {
                if (dfinite(lo)) od = fma(d, lo, od);
                else if (na_lt(dz, d)) unb = 1.0;
            } else {
                if (dfinite(hi)) od = fma(d, hi, od);
                else if (na_lt(dz, -d)) unb = 1.0;
            }
        }
        j0 += step;
        if (j0 < n) C = na_row_sums(cp, ci, acx, y, j0, min(per_warp, n - j0));
    }
    const double yz = 1e-8 * (1.0 + __ldcg(&s->met.ymax));
    double odr = 0.0, unbr = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const double yi = y[i];
        if (na_lt(yz, yi)) {
            if (dfinite(rmax[i])) odr -= yi * rmax[i];
            else unbr = 1.0;
        } else if (na_lt(yi, -yz)) {
            if (dfinite(rmin[i])) odr -= yi * rmin[i];
            else unbr = 1.0;
        }
    }
    double mx[3] = {dv, unb, unbr};
    block_dmax<3>(mx, red);
    double sm[3] = {op, od, odr};
    block_sum<3>(sm, red);
    if (threadIdx.x == 0) {
        double* P = s->part + blockIdx.x * 8;
        for (int q = 0; q < 3; ++q) {
            P[q] = mx[q];
            P[3 + q] = sm[q];
        }
    }
    if (!last_cta(&s->ticket[1])) return;
    double tm[3] = {0.0, 0.0, 0.0}, ts[3] = {0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads)
        for (int q = 0; q < 3; ++q) {
            tm[q] = dmax(tm[q], s->part[b * 8 + q]);
            ts[q] += s->part[b * 8 + 3 + q];
        }
    block_dmax<3>(tm, red);
    block_sum<3>(ts, red);
    if (threadIdx.x == 0) {
        DevMetrics& o = s->met;
        o.dv = tm[0];
        o.dinf = tm[0] / (1.0 + cmax);
        o.op = ts[0];
        const bool bounded = !(tm[1] > 0.0) && !(tm[2] > 0.0);
        o.od = bounded ? ts[1] + ts[2] : -CUDART_INF;
        o.gap = bounded ? smax(0.0, o.op - o.od) / (1.0 + fabs(o.op)) : CUDART_INF;
        out6[0] = __ldcg(&o.pinf);
        out6[1] = o.dinf;
        out6[2] = o.gap;
        out6[3] = o.op;
        out6[4] = o.od;
        out6[5] = __ldcg(&o.prow);
    }
}

// Rows (columns) per warp item: 32 fill the epilogue's lanes; with fewer than
// that many for every resident warp they are spread wider, since a warp takes
// its rows in series and the longest of these chains is the pass; down to 8
// (20,465 x 44,354, Zipf columns: 8 per warp 41 us a call, 4 per warp 55 us,
// where most lanes sort and reduce for nothing).
int rows_per_warp(int rows, int resident) {
    int r = 32;
    while (r > 8 && (long long)rows < (long long)r * kWarps * resident) r >>= 1;
    return r;
}

// Launch width: CTAs that stay resident (4 per SM, 64 registers) take the
// items in strides, so a CTA's block reductions are paid once.
int na_grid(int rows, int per_warp, int resident) {
    return std::min(resident, (rows + per_warp * kWarps - 1) / (per_warp * kWarps));
}

// Device address of the scratch on the current device. The symbol names a
// host-side stand-in in host code; its device address is looked up once per
// device, with that device current, and cached.
int scratch_for_current_device(NaScratch** out, int* sms) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return igx_set_error(IGAOS_PDHG_ERR_NODEVICE, cudaGetErrorString(e));
    if (dev < 0 || dev >= kMaxDevices)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "device ordinal beyond the scratch table");
    std::lock_guard<std::mutex> lock(g_na_mu);
    if (!g_na_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_na_scratch);
        if (e != cudaSuccess || !p) {
            char buf[256];
            std::snprintf(buf, sizeof(buf), "cudaGetSymbolAddress of the evaluation scratch: %s",
                          cudaGetErrorString(e));
            return igx_set_error(IGAOS_PDHG_ERR_CUDA, buf);
        }
        e = cudaDeviceGetAttribute(&g_na_sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return igx_set_error(IGAOS_PDHG_ERR_CUDA, cudaGetErrorString(e));
        g_na_ptr[dev] = static_cast<NaScratch*>(p);
    }
    *out = g_na_ptr[dev];
    *sms = g_na_sms[dev];
    return IGAOS_PDHG_OK;
}

}  // namespace
}  // namespace igx

extern "C" int igaos_pdhg_evaluate_noalloc(int m, int n, const int* ap, const int* ai,
                                           const double* ax, const int* cp, const int* ci,
                                           const double* acx, const double* c, const double* cl,
                                           const double* cu, const double* rmin,
                                           const double* rmax, const double* x, const double* y,
                                           double* out6, void* stream) {
    using namespace igx;
    if (m <= 0 || n <= 0) return igx_set_error(IGAOS_PDHG_ERR_INVALID, "m and n must be positive");
    if (m > kNaMaxDim || n > kNaMaxDim)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID,
                             "m or n above 4,194,304, the limit of the allocation-free "
                             "evaluation (use igaos_pdhg_evaluate)");
    if (!ap || !ai || !ax || !cp || !ci || !acx || !c || !cl || !cu || !rmin || !rmax || !x ||
        !y || !out6)
        return igx_set_error(IGAOS_PDHG_ERR_INVALID, "NULL device pointer");
    NaScratch* s = nullptr;
    int sms = 1;
    int rc = scratch_for_current_device(&s, &sms);
    if (rc != IGAOS_PDHG_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int resident = std::min(4 * sms, kNaMaxCtas);
    const int pr = rows_per_warp(m, resident), pc = rows_per_warp(n, resident);
    const int gr = na_grid(m, pr, resident), gc = na_grid(n, pc, resident);
    na_rows<<<gr, kThreads, 0, st>>>(m, n, pr, ap, ai, ax, x, y, c, rmin, rmax, s);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        // the products of the column pass need nothing of the row pass, so
        // its CTAs start as the row pass drains (programmatic launch)
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(gc);
        cfg.blockDim = dim3(kThreads);
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, na_cols, m, n, pc, cp, ci, acx, x, y, c, cl, cu, rmin, rmax, s,
                               out6);
    }
    if (e != cudaSuccess) {
        char buf[256];
        std::snprintf(buf, sizeof(buf), "CUDA error in PDHG engine: %s", cudaGetErrorString(e));
        return igx_set_error(IGAOS_PDHG_ERR_CUDA, buf);
    }
    return igx_set_error(IGAOS_PDHG_OK, "");
}
