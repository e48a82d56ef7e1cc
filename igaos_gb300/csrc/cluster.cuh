// Small LPs: the line-search attempts of a chunk in one thread-block cluster.
//
// For an LP of a few thousand rows and columns an attempt is a microsecond of
// work, and the grid-wide kernels spend ten and more on launches, on chains of
// dependent L2 loads (schedule -> row pointer -> entries -> gathers ->
// partials) and on the step decision. One cluster of C CTAs (1 to 16) instead
// runs the whole chunk in one launch, with the LP and its iterates on chip:
//   * each CTA stages its rows of A~ and A~^T (16-bit indices and values, lane
//     by lane) and their vectors (both parity slots of the iterates, bounds,
//     costs) in shared memory once per launch, and writes the accepted
//     iterates back at its end;
//   * every CTA keeps a replica of the gathered vectors (xbar and both parity
//     slots of y); the step of a row writes its new entry to every CTA's
//     through distributed shared memory, and so go the partial sums;
//   * per attempt: primal half, cluster barrier, dual half, cluster barrier,
//     then every CTA takes the same step decision (decide_step) in a warp of
//     its own from the same partials, while its other warps form A~^T y' of
//     the dual just computed: the next attempt starts from it if the step is
//     accepted (else from the accepted dual's, which is kept).
// The sums are those of the kernel each precision would otherwise run, bit for
// bit, whatever C: work is dealt in virtual warps (below) and their partials
// are merged in the same order.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "engine.hpp"
#include "kernels.cuh"

namespace igx {

constexpr int kSmallCluster = 16;       // most CTAs
constexpr int kSmallWarps = 16;         // warps of a CTA that own rows
constexpr int kSmallThreads = 32 * (kSmallWarps + 3);  // and the decision's three
constexpr size_t kSmallSmemMax = 222 * 1024;  // dynamic shared memory per CTA
// FP32: a virtual warp v < kSmallVirtual takes the schedule's items v, v +
// kSmallVirtual, ..., at most kSmallItems of them; its lanes' sums run over
// them. Sixteen virtual warps make a partial, eight partials the total.
constexpr int kSmallVirtual = 128;
constexpr int kSmallItems = 8;
// FP64: a virtual warp is an item; eight make a partial, as in a CTA of the
// grid-wide kernels, and the partials merge as finish_attempt merges them.
constexpr int kSmallMaxItems = kSmallVirtual * kSmallItems;

__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
// All threads of every CTA of the cluster, in two halves; release/acquire at
// cluster scope (global and distributed shared memory). The release alone
// takes about 1,000 cycles after remote stores, 500 without: work that
// nobody waits for goes between the halves. One CTA has no first half.
__device__ __forceinline__ void cluster_arrive(int ctas) {
    __syncwarp();
    if (ctas > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait(int ctas) {
    __syncwarp();
    if (ctas > 1)
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
        __syncthreads();
}
// v into the entry `at` (an address in this CTA's replica) of every CTA's
template <typename T>
__device__ __forceinline__ void cluster_put(T* at, T v, int ctas) {
    if (ctas == 1) {
        *at = v;
        return;
    }
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    for (int r = 0; r < ctas; ++r) *cl.map_shared_rank(at, r) = v;
}

// Writes a row's new entry into the same slot of every CTA's replica.
template <typename T>
struct ClusterBcast {
    T* base;  // this CTA's replica
    int ctas;
    __device__ __forceinline__ void operator()(int i, T v) const { cluster_put(base + i, v, ctas); }
};

// A CTA's items as staged: item = {first row, rows, log2 G, first slot}; entry u
// of a lane (its row's entries gl, gl + G, ...) lies at slot first + 32 u +
// lane, padded with zeros to the longest row's entries per lane (the item's
// count, in the bits of log2 G from 8 up).
template <typename T>
struct Staged {
    const uint16_t* idx;
    const T* val;
};
__host__ __device__ inline int staged_count(int longest, int lg) {
    return (longest + (1 << lg) - 1) >> lg;
}

// row sums of one staged item, handed to the lanes of its rows (the sums and
// their order are those of lane_products and reduce_rows)
template <typename T>
__device__ __forceinline__ Acc<T> staged_sums(const int4 d, const Staged<T>& S,
                                              const T* __restrict__ sx) {
    int at = d.w + (threadIdx.x & 31), left = d.z >> 8;
    Acc<T> acc;
#pragma unroll 1
    for (; left >= 2; left -= 2, at += 64) {
        const T a0 = S.val[at], a1 = S.val[at + 32];
        const int j0 = S.idx[at], j1 = S.idx[at + 32];
        const T x0 = sx[j0], x1 = sx[j1];
        acc.add(a0, x0);
        acc.add(a1, x1);
    }
    if (left) acc.add(S.val[at], sx[S.idx[at]]);
    return reduce_rows<T>(acc, d.z & 0xff);
}

// The sums of a half's virtual warps lie padded with zeros to small_pad.
template <typename T>
__host__ __device__ inline int small_pad(int virt) {
    return std::is_same<T, float>::value ? kSmallVirtual : (virt + 7) & ~7;
}
template <typename T>
__host__ __device__ inline size_t small_bytes(int m, int n, const SmallPlan& p) {
    size_t b = (size_t)(n + 2 * m) * sizeof(T);                                // replicas
    b = (b + 15) & ~(size_t)15;
    if (p.held) {
        b += (size_t)p.cap.items_at * 32 * (7 * sizeof(T) + 2 * sizeof(Acc<T>));  // columns' vectors
        b += (size_t)p.cap.items_a * 32 * 9 * sizeof(T);                          // rows' vectors
    }
    b += (size_t)2 * (small_pad<T>(p.virt_at) + small_pad<T>(p.virt_a)) * sizeof(T);  // partials
    b += (size_t)p.cap.slots * sizeof(T);                                    // values
    b = (b + 15) & ~(size_t)15;
    b += (size_t)(p.cap.items_at + p.cap.items_a) * sizeof(int4);              // items
    b += (size_t)p.cap.slots * 2;                                              // indices
    return b + 32;
}

// (float)(a / b) of the FP64 quotient, ib = 1 / b correctly rounded: the
// product is within two ulps of it, which decides the float unless they
// straddle the middle of two.
__device__ __forceinline__ float float_quotient(double a, double b, double ib) {
    const double q = __dmul_rn(a, ib);
    const unsigned low = (unsigned)__double2loint(q) & 0x1fffffffu;
    const int ex = (__double2hiint(q) >> 20) & 0x7ff;
    const bool clear = low - 0x0ffffff8u > 16u && ex > 1023 - 126 && ex < 1023 + 127;
    return clear ? (float)q : (float)div_exact(a, b, ib);
}

// FP32: the three totals, by one warp: partials of 16 virtual warps, plain
// sums, each in a lane; eight of them merged, compensated.
__device__ __forceinline__ void small_totals(const float* dx, const float* dy, const float* cr,
                                             double* total) {
    const int lane = threadIdx.x & 31, q = lane >> 3;
    const float4* v = reinterpret_cast<const float4*>((q == 0 ? dx : q == 1 ? dy : cr) + 16 * (lane & 7));
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 f = v[k];
        s = s + f.x;
        s = s + f.y;
        s = s + f.z;
        s = s + f.w;
    }
    Acc<float> t;
#pragma unroll
    for (int r = 0; r < kSmallVirtual / 16; ++r) {
        Acc<float> part;
        part.s = __shfl_sync(0xffffffffu, s, (lane & 24) + r);
        t.merge(part);
    }
    const double d = t.result_d();
#pragma unroll
    for (int k = 0; k < 3; ++k) total[k] = __shfl_sync(0xffffffffu, d, 8 * k);
}
// FP64: one total by one warp (three warps side by side): partials of 8, 32
// of them over the lanes (the levels of the tree that only add zeros left
// out), groups of 32 in turn.
__device__ __forceinline__ double small_total(const double* v, int pad) {
    const int lane = threadIdx.x & 31;
    double total = 0.0;
    for (int g = 0; 256 * g < pad; ++g) {
        const int k0 = 8 * (32 * g + lane);
        double s = 0.0;
        if (k0 < pad) {
            const double2* a = reinterpret_cast<const double2*>(v + k0);
            const double2 b0 = a[0], b1 = a[1], b2 = a[2], b3 = a[3];
            s = b0.x + b0.y;
            s = s + b1.x;
            s = s + b1.y;
            s = s + b2.x;
            s = s + b2.y;
            s = s + b3.x;
            s = s + b3.y;
        }
        int o = 16;
        if (pad < 256)
            while (o && 8 * o >= pad) o >>= 1;
        for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        s = __shfl_sync(0xffffffffu, s, 0);
        total = g == 0 ? s : total + s;
    }
    return total;
}

// The attempts of one chunk (up to max_attempts, until the control block's
// stop flag). What an attempt costs is latency: the two barriers, and FP64
// operations of one warp at 60 cycles and more each (its SMSP's unit takes a
// warp through in 64), so only what the next half waits for stands before a
// barrier's arrival: the averages and ||dx||^2 are formed behind it. 2,048 FP32
// iterations of a 2,000 x 5,000 LP: 19.5 -> 12.9 ms (with one deciding CTA, its
// answer published behind a third barrier, the vectors in global memory and
// entries by row pointers).
template <typename T, bool HELD>
__global__ void __launch_bounds__(kSmallThreads, 1)
    k_attempts_cluster(PrimalArgs<T> pa, DualArgs<T> da, int m, int n, int max_attempts,
                       SmallPlan plan) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CtlView<T> sview;
    __shared__ double stotal[2];
    __shared__ int scnt[2][kSmallWarps + 1][2];
    const int rank = cluster_rank(), ctas = plan.ctas;
    const int wi = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31);
    const bool owns = wi < kSmallWarps;
    // columns go to the lower warps first, of these to the SMSPs 1 to 3 (their
    // products run beside the decision's warp, on SMSP 0); rows to the upper
    // ones, over the SMSPs in turn
    const int low = wi & 7;
    const int at_pos = (wi & 8) + ((low & 3) ? (low >> 2) * 3 + (low & 3) - 1 : 6 + (low >> 2));
    const int deal_step = kSmallWarps * ctas;
    const int first_at = at_pos * ctas + rank;
    const int first_a = (kSmallWarps - 1 - wi) * ctas + rank;

    // ---- carve
    const int sat = HELD ? plan.cap.items_at * 32 : 0, sa = HELD ? plan.cap.items_a * 32 : 0;
    const int pad_at = small_pad<T>(plan.virt_at), pad_a = small_pad<T>(plan.virt_a);
    T* sxbar = reinterpret_cast<T*>(smem);
    T* sy[2] = {sxbar + n, sxbar + n + m};
    size_t off = ((size_t)(n + 2 * m) * sizeof(T) + 15) & ~(size_t)15;
    Acc<T>* sg = reinterpret_cast<Acc<T>*>(smem + off);   // A~^T y of both slots
    T* vat = reinterpret_cast<T*>(sg + 2 * sat);  // c, lo, hi, x[2], xavg[2]
    T* va = vat + 7 * sat;                        // rmin, rmax, yhat, y[2], axc[2], yavg[2]
    T* part_dx = va + 9 * sa;                     // of every other attempt
    T *part_dy = part_dx + 2 * pad_at, *part_cr = part_dy + pad_a;
    T* val = part_cr + pad_a;
    off = (size_t)(reinterpret_cast<unsigned char*>(val + plan.cap.slots) - smem);
    off = (off + 15) & ~(size_t)15;
    int4* item = reinterpret_cast<int4*>(smem + off);
    uint16_t* idx = reinterpret_cast<uint16_t*>(item + plan.cap.items_at + plan.cap.items_a);

    // ---- each warp's share of both schedules: items, entries, row pointers
    auto items_of = [&](int o, auto&& f) {  // every item of this warp, in order
        const WarpSched& ws = o ? da.ws : pa.ws;
        const int virt = o ? plan.virt_a : plan.virt_at;
        for (int v = o ? first_a : first_at; v < virt; v += deal_step)
            for (int w = v; w < ws.nwarps; w += virt) f(ws, w);
    };
    if (owns)
        for (int o = 0; o < 2; ++o) {
            const Csr<T>& A = o ? da.A : pa.AT;
            int c = 0, e = 0;
            items_of(o, [&](const WarpSched& ws, int w) {
                const int r0 = __ldg(ws.row + w);
                ++c;  // (rows are sorted by decreasing length)
                e += 32 * staged_count(__ldg(A.ptr + r0 + 1) - __ldg(A.ptr + r0), __ldg(ws.lg + w));
            });
            if (lane == 0) {
                scnt[o][wi + 1][0] = c;
                scnt[o][wi + 1][1] = e;
            }
        }
    for (int i = threadIdx.x; i < 2 * (pad_at + pad_a); i += kSmallThreads) part_dx[i] = T(0);
    __syncthreads();
    if (threadIdx.x < 2) {
        int run = 0;  // rows of A after those of A~^T, in one sequence
        for (int o = 0; o < 2; ++o) {
            scnt[o][0][threadIdx.x] = run;
            for (int k = 1; k <= kSmallWarps; ++k) run = scnt[o][k][threadIdx.x] += run;
        }
    }
    __syncthreads();
    const int p0 = __ldcg(&pa.ctl->parity);
    const int items_at = scnt[1][0][0];  // of this CTA
    const int it0 = owns ? scnt[0][wi][0] : 0, it1 = owns ? scnt[1][wi][0] : 0;
    if (owns)
        for (int o = 0; o < 2; ++o) {
            const Csr<T>& A = o ? da.A : pa.AT;
            int k = scnt[o][wi][0], ce = scnt[o][wi][1];
            items_of(o, [&](const WarpSched& ws, int w) {
                const int r0 = __ldg(ws.row + w), r1 = __ldg(ws.row + w + 1);
                const int lg = __ldg(ws.lg + w), r = r0 + (lane >> lg);
                const int cnt = staged_count(__ldg(A.ptr + r0 + 1) - __ldg(A.ptr + r0), lg);
                int q = 0, e = 0;
                if (r < r1) {
                    q = __ldg(A.ptr + r) + (lane & ((1 << lg) - 1));
                    e = __ldg(A.ptr + r + 1);
                }
                for (int u = 0; u < cnt; ++u, q += 1 << lg) {
                    const bool ok = q < e;
                    idx[ce + 32 * u + lane] = ok ? (uint16_t)__ldg(A.idx + q) : (uint16_t)0;
                    val[ce + 32 * u + lane] = ok ? __ldg(A.val + q) : T(0);
                }
                if (lane == 0) item[k] = make_int4(r0, r1 - r0, lg | cnt << 8, ce);
                const int i = r0 + lane;
                if (HELD && lane < r1 - r0) {
                    if (o == 0) {
                        T* v = vat + 32 * k + lane;
                        v[0] = __ldg(pa.c + i);
                        v[sat] = __ldg(pa.lo + i);
                        v[2 * sat] = __ldg(pa.hi + i);
                        v[(3 + p0) * sat] = pa.x[p0][i];
                        v[(5 + p0) * sat] = pa.xavg[p0][i];
                    } else {
                        T* v = va + 32 * (k - items_at) + lane;
                        v[0] = __ldg(da.rmin + i);
                        v[sa] = __ldg(da.rmax + i);
                        v[2 * sa] = da.yhat ? __ldg(da.yhat + i) : T(0);
                        v[(3 + p0) * sa] = da.y[p0][i];
                        v[(5 + p0) * sa] = da.axc[p0][i];
                        v[(7 + p0) * sa] = da.yavg[p0][i];
                    }
                }
                ce += 32 * cnt;
                ++k;
            });
        }
    for (int i = threadIdx.x; i < m; i += kSmallThreads) sy[p0][i] = pa.y[p0][i];
    // the deciding warp's state (every lane's)
    StepState st{};
    long long attempts = 0, accepted = 0, k_stop = 0;
    int nan_flag = 0;
    double dots[3] = {0.0, 0.0, 0.0};
    if (wi == kSmallWarps) {
        st = load_step(pa.ctl, da.fac, da.n_fac);
        k_stop = pa.ctl->k_stop;
        nan_flag = pa.ctl->nan_flag;
        if (lane == 0) sview = read_ctl<T>(pa.ctl);
    }
    const long long fac_base = pa.ctl->fac_base;
    __syncthreads();
    const Staged<T> S{idx, val};
    // A~^T y of slot q into sg, this warp's items
    auto product_at = [&](int q) {
        int k = it0;
        items_of(0, [&](const WarpSched&, int) {
            sg[q * sat + 32 * k + lane] = staged_sums<T>(item[k], S, sy[q]);
            ++k;
        });
    };
    if (HELD && owns) product_at(p0);
    cluster_arrive(ctas);  // every CTA running and staged before any remote write
    cluster_wait(ctas);

    int att = 0;
    for (; att < max_attempts; ++att) {
        const CtlView<T> cv = sview;
        if (cv.stop) break;  // the same in every CTA
        const int p = cv.parity, q = p ^ 1;
        T* dx_to = part_dx + (att & 1) * pad_at;  // other CTAs may still read the last ones
        if (owns) {  // primal half
            if constexpr (HELD) {
                int k = it0;
                for (int v = first_at; v < plan.virt_at; v += deal_step)
                    for (int w = v; w < pa.ws.nwarps; w += plan.virt_at, ++k) {
                        const int4 d = item[k];
                        if (lane >= d.y) continue;
                        T* z = vat + 32 * k + lane;
                        const T x = z[(3 + p) * sat];
                        const T g = z[0] + sg[p * sat + 32 * k + lane].result();
                        const T xn = primal_step(cv.tau, g, x, z[sat], z[2 * sat]);
                        z[(3 + q) * sat] = xn;
                        cluster_put(sxbar + d.x + lane, fma((T)2, xn, -x), ctas);
                    }
            } else {
                int k = it0;
                PrimalEpi<T, ClusterBcast<T>> epi{pa.c,       pa.lo,      pa.hi,   pa.x[p], pa.xavg[p],
                                                  pa.x[q],    pa.xavg[q], pa.xbar, cv.tau,  cv.w,
                                                  T(0),       ClusterBcast<T>{sxbar, ctas}};
                for (int v = first_at; v < plan.virt_at; v += deal_step) {
                    epi.dx2 = T(0);
                    for (int w = v; w < pa.ws.nwarps; w += plan.virt_at, ++k) {
                        const int4 d = item[k];
                        typename PrimalEpi<T, ClusterBcast<T>>::Pre pre{};
                        if (lane < d.y) pre = epi.load(d.x + lane);
                        const Acc<T> g = staged_sums<T>(d, S, sy[p]);
                        if (lane < d.y) epi.apply(d.x + lane, g, pre);
                    }
                    const T dx2 = lanes_sum(epi.dx2);
                    if (lane == 0) cluster_put(dx_to + v, dx2, ctas);
                }
            }
        }
        cluster_arrive(ctas);
        auto averages_at = [&]() {  // ||dx||^2 and the average
            int k = it0;
            for (int v = first_at; v < plan.virt_at; v += deal_step) {
                T dx2 = T(0);
                for (int w = v; w < pa.ws.nwarps; w += plan.virt_at, ++k) {
                    if (lane >= item[k].y) continue;
                    T* z = vat + 32 * k + lane;
                    const T xn = z[(3 + q) * sat], xa = z[(5 + p) * sat];
                    const T dx = xn - z[(3 + p) * sat];
                    dx2 = fma(dx, dx, dx2);
                    z[(5 + q) * sat] = fma(cv.w, xn - xa, xa);
                }
                __syncwarp();
                dx2 = lanes_sum(dx2);
                if (lane == 0) cluster_put(dx_to + v, dx2, ctas);
            }
        };
        if (HELD && owns && ctas > 1) averages_at();
        cluster_wait(ctas);
        if (HELD && owns && ctas == 1) averages_at();
        if (owns) {  // dual half
            int k = it1;
            DualEpi<T, ClusterBcast<T>> epi{da.rmin,    da.rmax,   da.y[p],    da.axc[p], da.yavg[p], da.yhat,
                                            da.y[q],    da.axc[q], da.yavg[q], cv.sigma,  cv.isigma,
                                            cv.w,       T(0),      T(0),       ClusterBcast<T>{sy[q], ctas}};
            for (int v = first_a; v < plan.virt_a; v += deal_step) {
                epi.dy2 = epi.cross = T(0);
                for (int w = v; w < da.ws.nwarps; w += plan.virt_a, ++k) {
                    const int4 d = item[k];
                    if constexpr (HELD) {
                        const T ab = staged_sums<T>(d, S, sxbar).result();
                        if (lane >= d.y) continue;
                        T* z = va + 32 * (k - items_at) + lane;
                        const T y = z[(3 + p) * sa];
                        const T yn = dual_step(cv.sigma, cv.isigma, ab, y, da.yhat != nullptr, z[2 * sa],
                                               z[0], z[sa]);
                        z[(3 + q) * sa] = yn;
                        cluster_put(sy[q] + d.x + lane, yn, ctas);
                        const T dy = yn - y;
                        const T adx = (T)0.5 * (ab - z[(5 + p) * sa]);
                        z[(5 + q) * sa] = adx;
                        epi.dy2 = fma(dy, dy, epi.dy2);
                        epi.cross = fma(dy, adx, epi.cross);
                    } else {
                        typename DualEpi<T, ClusterBcast<T>>::Pre pre{};
                        if (lane < d.y) pre = epi.load(d.x + lane);
                        const Acc<T> ab = staged_sums<T>(d, S, sxbar);
                        if (lane < d.y) epi.apply(d.x + lane, ab, pre);
                    }
                }
                __syncwarp();
                const T sums = lanes_sum2(epi.dy2, epi.cross);
                if ((lane & 15) == 0) cluster_put((lane ? part_cr : part_dy) + v, sums, ctas);
            }
        }
        cluster_arrive(ctas);
        auto averages_a = [&]() {
            int k = it1;
            items_of(1, [&](const WarpSched&, int) {
                if (lane < item[k].y) {
                    T* z = va + 32 * (k - items_at) + lane;
                    z[(5 + q) * sa] = z[(5 + p) * sa] + z[(5 + q) * sa];
                    const T ya = z[(7 + p) * sa];
                    z[(7 + q) * sa] = fma(cv.w, z[(3 + q) * sa] - ya, ya);
                }
                ++k;
            });
        };
        if (HELD && owns && ctas > 1) averages_a();
        cluster_wait(ctas);
        if (HELD && owns && ctas == 1) averages_a();
        if (owns) {
            if (HELD) product_at(q);
        } else if (wi == kSmallWarps || sizeof(T) == 8) {
            if constexpr (std::is_same<T, double>::value) {
                const double t = wi == kSmallWarps       ? small_total(dx_to, pad_at)
                                 : wi == kSmallWarps + 1 ? small_total(part_dy, pad_a)
                                                         : small_total(part_cr, pad_a);
                if (wi > kSmallWarps && lane == 0) stotal[wi - kSmallWarps - 1] = t;
                asm volatile("bar.sync 1, 96;" ::: "memory");
                dots[0] = t;
                dots[1] = stotal[0];
                dots[2] = stotal[1];
            } else {
                small_totals(dx_to, part_dy, part_cr, dots);
            }
            if (wi == kSmallWarps) {  // as decide_step
                const StepOut o = step_rule<sizeof(T) == 8>(st, dots[0], dots[1], dots[2]);
                const double sigma = __dmul_rn(o.eta, st.omega);
                CtlView<T> nv = cv;
                if constexpr (std::is_same<T, double>::value) {
                    const double out = __ddiv_rn(lane == 1 ? 1.0 : o.eta, lane == 1 ? sigma : st.omega);
                    nv.isigma = __shfl_sync(0xffffffffu, out, 1);
                    nv.tau = out;
                } else {
                    nv.tau = float_quotient(o.eta, st.omega, st.iomega);
                    nv.isigma = 1.0f / (float)sigma;
                }
                nv.sigma = (T)sigma;
                if (!o.sound) nan_flag = 1;
                if (o.accept) {
                    nv.parity = q;
                    nv.w = (T)o.w;
                    nv.stop = st.k >= k_stop || nan_flag;
                }
                if (lane == 0) sview = nv;
                st.eta = o.eta;
                st.retries = o.accept ? 0 : st.retries + 1;
                if (o.accept) {
                    ++accepted;
                    ++st.hn;
                    ++st.k;
                }
                ++attempts;
            }
        }
        __syncthreads();
        if (wi == kSmallWarps)
            step_factors(st, fac_base, da.fac, da.n_fac);  // of the next decision
    }
    // the accepted iterates, for the host's checks
    const int p = sview.parity;
    if (HELD && owns) {
        int k = it0;
        items_of(0, [&](const WarpSched&, int) {
            const int4 d = item[k];
            const T* z = vat + 32 * k + lane;
            if (lane < d.y) {
                pa.x[p][d.x + lane] = z[(3 + p) * sat];
                pa.xavg[p][d.x + lane] = z[(5 + p) * sat];
            }
            ++k;
        });
        k = it1;
        items_of(1, [&](const WarpSched&, int) {
            const int4 d = item[k];
            const T* z = va + 32 * (k - items_at) + lane;
            if (lane < d.y) {
                da.y[p][d.x + lane] = z[(3 + p) * sa];
                da.axc[p][d.x + lane] = z[(5 + p) * sa];
                da.yavg[p][d.x + lane] = z[(7 + p) * sa];
            }
            ++k;
        });
    }
    cluster_arrive(ctas);  // no CTA leaves while another may still write to it
    cluster_wait(ctas);    // (and every CTA has read the control block)
    if (rank == 0 && wi == kSmallWarps && lane == 0 && attempts) {
        DevCtl* c = pa.ctl;
        for (int k = 0; k < 3; ++k) c->dots[k] = dots[k];
        c->eta = st.eta;
        c->k = st.k;
        c->hn = st.hn;
        c->attempts += attempts;
        c->accepted += accepted;
        c->retries = st.retries;
        c->parity = p;
        c->stop = sview.stop;
        c->nan_flag = nan_flag;
        ctl_derive(c);
    }
}

}  // namespace igx
