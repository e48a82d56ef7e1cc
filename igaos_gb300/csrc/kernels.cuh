// Kernels of the GB300 PDHG engine. Reference algorithm: IGAOS
// src/pdhg/pdhg.cu (file:line cited per kernel).
#pragma once

#include "device.cuh"

namespace igx {

// Original-unit column value x = dc * x~ (src/pdhg/pdhg.cu:712). An FP32
// iterate projected onto its FP32-rounded bound is exactly at that bound:
// it maps to the FP64 bound itself (dc * fl32(l/dc) would sit ~6e-8 |l|
// away, outside evaluate()'s 1e-9 "at bound" band). FP64 iterates are
// unscaled as the reference does, without snapping.
__device__ __forceinline__ double unscale_x(double xs, double, double, double dc, double,
                                           double) {
    return xs * dc;
}
__device__ __forceinline__ double unscale_x(float xs, float slo, float shi, double dc, double lo,
                                           double hi) {
    if (xs == slo) return lo;
    if (xs == shi) return hi;
    return (double)xs * dc;
}

template <typename TI>
__global__ void k_unscale_cols(int n, const TI* __restrict__ xs, const TI* __restrict__ slo,
                               const TI* __restrict__ shi, const double* __restrict__ dc,
                               const double* __restrict__ lo, const double* __restrict__ hi,
                               double* __restrict__ out) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
        out[j] = unscale_x(xs[j], slo[j], shi[j], dc[j], lo[j], hi[j]);
}

// The caller's numbering and the device's: device entry i is the caller's
// perm[i]. Answers go back in original units: x = dc x~ (op 1), y = y~ / dr
// (op 2), or as they are. (On the host, behind a copy of its own, this took 3 of
// the 25.5 ms of 256 iterations of a multicommodity LP of 4 million columns and
// rows.)
__global__ void k_from_user(int n, const double* __restrict__ in, const int* __restrict__ perm,
                            double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = in[perm[i]];
}
template <typename T>
__global__ void k_to_user(int n, const T* __restrict__ in, int op, const double* __restrict__ d,
                          const int* __restrict__ perm, double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = (double)in[i];
        out[perm[i]] = op == 1 ? __dmul_rn(v, d[i]) : op == 2 ? __ddiv_rn(v, d[i]) : v;
    }
}

// ------------------------------------------------------------ attempt state
// Per-launch view of the control block, read once per CTA.
template <typename T>
struct CtlView {
    int parity, stop;
    T tau, sigma, w, isigma;
};
template <typename T>
__device__ __forceinline__ CtlView<T> read_ctl(const DevCtl* c);
template <>
__device__ __forceinline__ CtlView<double> read_ctl<double>(const DevCtl* c) {
    return CtlView<double>{c->parity, *(volatile const int*)&c->stop, c->tau, c->sigma, c->w,
                           c->isigma};
}
template <>
__device__ __forceinline__ CtlView<float> read_ctl<float>(const DevCtl* c) {
    return CtlView<float>{c->parity, *(volatile const int*)&c->stop, c->tau_f, c->sigma_f, c->w_f,
                          c->isigma_f};
}

// The attempt kernels follow one another by programmatic launches: a kernel's
// CTAs take their places as the last one's leave and wait here for its
// results; in FP64 they first load what does not change (schedule, row
// pointers; in FP32 that cost the large LPs more in registers than it gave).
// A kernel lets the next one start when its products are done: from its
// start on, waiting CTAs slowed FP32 attempts of large LPs by 8 %. 1,024 FP64
// iterations of a 2,000 x 5,000 LP: 17.7 -> 15.7 ms; of an 8,000 x 20,000 LP in
// FP32 16.1 -> 14.9; 256 of the 200,000 x 500,000 LP in FP64 28.6 -> 28.4.
// (One resident launch per chunk with grid-wide barriers was slower than
// either: 30.8 ms against 28.4 for 1,024 iterations of a 20,000 x 50,000 LP.)
__device__ __forceinline__ void follow_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void let_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename T>
struct PrimalArgs {
    WarpSched ws;
    Csr<T> AT;              // A~^T (rows = columns of A)
    const T* y[2];          // dual iterate slots
    const T* c;             // scaled cost
    const T* lo;            // scaled column bounds
    const T* hi;
    T* x[2];
    T* xavg[2];
    T* xbar;
    Acc<T>* part;           // per-CTA ||dx||^2 (compensated in FP32 kernels)
    DevCtl* ctl;
};

// Primal half of one line-search attempt, fused into the A^T y SpMV:
//   g = c + A^T y;  x' = P_[l,u](x - tau g);  xbar = 2x' - x;  dx = x' - x
// (kern_primal, src/pdhg/pdhg.cu:33-45) plus the candidate Halpern average
// xavg' = xavg + w (x' - xavg), w = 2/(hn+2) (kern_mix2, :129-141, :795-799),
// written to the other parity slot so that a rejected attempt leaves the
// accepted state untouched.
template <typename T>
__device__ __forceinline__ T primal_step(T tau, T g, T x, T lo, T hi) {
    return clamp_val(fma(-tau, g, x), lo, hi);
}
// Hook called with each row's new gathered-vector entry (xbar_j, y'_i):
// nothing for the grid-wide kernels.
struct NoBcast {
    template <typename U>
    __device__ __forceinline__ void operator()(int, U) const {}
};

template <typename T, class B = NoBcast>
struct PrimalEpi {
    const T *c, *lo, *hi, *xc, *xa;
    T *xn_out, *xa_out, *xbar;
    T tau, w, dx2;
    B bc{};
    struct Pre {
        T c, lo, hi, x, xa;
    };
    __device__ __forceinline__ Pre load(int j) const {
        return Pre{__ldg(c + j), __ldg(lo + j), __ldg(hi + j), xc[j], xa[j]};
    }
    __device__ __forceinline__ void apply(int j, const Acc<T>& acc, const Pre& v) {
        const T g = v.c + acc.result();
        const T xn = primal_step(tau, g, v.x, v.lo, v.hi);
        xn_out[j] = xn;
        const T xb = fma((T)2, xn, -v.x);
        xbar[j] = xb;
        bc(j, xb);
        const T dx = xn - v.x;
        dx2 = fma(dx, dx, dx2);
        xa_out[j] = fma(w, xn - v.xa, v.xa);
    }
};

// OCC: resident CTAs per SM the kernel is compiled for (its register
// budget); FP64 attempts come in two (3 and 4), chosen by the autotuner.
template <typename T, int OCC = HotCtas<T>::value>
__global__ void __launch_bounds__(kThreads, OCC) k_primal(PrimalArgs<T> a) {
    __shared__ __align__(16) double smred[kWarps * 4];
    FirstItem first;
    if constexpr (sizeof(T) == 8) first = first_item<T>(a.ws, a.AT);
    follow_previous();
    const CtlView<T> cv = read_ctl<T>(a.ctl);
    if (cv.stop) return;
    if constexpr (sizeof(T) == 4) first = first_item<T>(a.ws, a.AT);
    const int p = cv.parity, q = p ^ 1;
    PrimalEpi<T> epi{a.c, a.lo, a.hi, a.x[p], a.xavg[p], a.x[q], a.xavg[q], a.xbar,
                     cv.tau, cv.w, (T)0};
    warp_rows_from<T>(a.ws, a.AT, a.y[p], epi, first);
    let_next();
    const T dx2 = epi.dx2;
    T v[1] = {dx2};
    block_sum_t<T, 1>(v, reinterpret_cast<T*>(smred));
    if (threadIdx.x == 0) {
        Acc<T> e;
        e.s = v[0];
        a.part[blockIdx.x] = e;
    }
}

template <typename T>
struct DualArgs {
    WarpSched ws;
    Csr<T> A;
    const T* xbar;
    const T* rmin;          // scaled row bounds
    const T* rmax;
    T* y[2];
    T* axc[2];              // A x of the accepted iterate
    T* yavg[2];
    Acc<T>* part;           // per-CTA (||dy||^2, dy'A dx)
    const Acc<T>* part_primal;
    const T* yhat;          // anchor of anchored iterations (rounded), or nullptr
    const double* fac;      // (1 - k^-0.3, 1 + k^-0.6) for k = ctl->fac_base + i
    int n_fac;
    int n_primal;
    DevCtl* ctl;
};

// Anchored iterations (FP32 + FP64 refinement) hold y = yhat + dy with an
// FP64 anchor yhat; the dual projection must act on the full value, so the
// clamp argument is (t + yhat)/sigma with t = dy + sigma A dxbar and the row
// bounds shifted by the anchor's activity. yhat == nullptr: plain iterates.
// The quotient u / sigma (u = t, or t + yhat) is formed from the correctly
// rounded reciprocal 1/sigma of the step decision by one remainder
// correction (Markstein): q0 = u (1/sigma), r = fma(-sigma, q0, u),
// q = fma(r, 1/sigma, q0). q is the correctly rounded quotient except in
// rare cases (where it is one ulp off); an IEEE FP64 division costs about
// ten FP64 instructions, and FP64's pipe (2 per clock per SM on this GPU)
// bounds the FP64 attempt. The rest is the reference's formula (kern_dual,
// src/pdhg/pdhg.cu:49-61), y' = fma(-sigma, clamp(q, lo, hi), t), so an
// in-range row keeps the reference's rounding residue, which the line search
// sees through dy. (An oracle run with this quotient took the same
// iterations to the same objective, bit for bit, on the 14 golden LPs, six
// Netlib LPs and a 1 x 1 LP; giving in-range rows an exact 0 instead froze
// the 1 x 1 LP's step size: with dy = 0 the line search sees no curvature.)
template <typename T>
__device__ __forceinline__ T dual_step(T sigma, T isigma, T ab, T y, bool anchored, T yh, T lo, T hi) {
    const T t = fma(sigma, ab, y);
    const T u = anchored ? t + yh : t;
    const T q0 = u * isigma;
    const T q = fma(fma(-sigma, q0, u), isigma, q0);
    return fma(-sigma, clamp_val(q, lo, hi), t);
}
template <typename T, class B = NoBcast>
struct DualEpi {
    const T *rmin, *rmax, *yc, *axc, *ya, *yhat;
    T *yn_out, *axc_out, *ya_out;
    T sigma, isigma, w, dy2, cross;
    B bc{};
    struct Pre {
        T lo, hi, y, ax, ya, yh;
    };
    __device__ __forceinline__ Pre load(int i) const {
        return Pre{__ldg(rmin + i), __ldg(rmax + i), yc[i], axc[i], ya[i],
                   yhat ? __ldg(yhat + i) : T(0)};
    }
    __device__ __forceinline__ void apply(int i, const Acc<T>& acc, const Pre& v) {
        const T ab = acc.result();
        const T yn = dual_step(sigma, isigma, ab, v.y, yhat != nullptr, v.yh, v.lo, v.hi);
        yn_out[i] = yn;
        bc(i, yn);
        const T dy = yn - v.y;
        const T adx = (T)0.5 * (ab - v.ax);
        axc_out[i] = v.ax + adx;
        dy2 = fma(dy, dy, dy2);
        cross = fma(dy, adx, cross);
        ya_out[i] = fma(w, yn - v.ya, v.ya);
    }
};

// a / b, correctly rounded, from ib = 1 / b correctly rounded: the product and
// two remainder steps (Markstein 1990: the first leaves an error below an ulp,
// the second rounds correctly). 300 cycles of latency, a division 575.
// Operands far from 1 by hundreds of binades divide.
__device__ __forceinline__ double div_exact(double a, double b, double ib) {
    auto tame = [](double v) {
        const int ex = (__double2hiint(v) >> 20) & 0x7ff;
        return ex > 512 && ex < 1536;
    };
    if (!tame(a) || !tame(b)) return __ddiv_rn(a, b);
    double q = __dmul_rn(a, ib);
    q = fma(fma(-b, q, a), ib, q);
    return fma(fma(-b, q, a), ib, q);
}

// What a step decision reads of the control block, loaded ahead of the dot
// products it waits for (by every lane of the deciding warp).
struct StepState {
    double eta, omega, iomega, f_lo, f_hi;
    long long k, hn;
    int retries;
};
// growth/shrink factors 1 - k^-0.3 and 1 + k^-0.6, tabulated by the host
// (std::pow, as the reference) for the iterations of this chunk
__device__ __forceinline__ void step_factors(StepState& s, long long fac_base, const double* fac,
                                             int n_fac) {
    const long long fi = s.k - fac_base;
    if (fac && fi >= 0 && fi < n_fac) {
        s.f_lo = fac[2 * fi];
        s.f_hi = fac[2 * fi + 1];
    } else {
        const double kk = (double)s.k;
        s.f_lo = __dsub_rn(1.0, pow(kk, -0.3));
        s.f_hi = __dadd_rn(1.0, pow(kk, -0.6));
    }
}
__device__ __forceinline__ StepState load_step(const DevCtl* c, const double* fac, int n_fac) {
    StepState s;
    s.eta = c->eta;
    s.omega = c->omega;
    s.iomega = c->iomega;
    s.k = c->k;
    s.hn = c->hn;
    s.retries = c->retries;
    step_factors(s, c->fac_base, fac, n_fac);
    return s;
}

// Adaptive step decision (src/pdhg/pdhg.cu:770-794) by one warp, every lane
// with the same operands. Host-side arithmetic of the reference has no FMA
// contraction; the explicit _rn intrinsics keep it that way here. The chain of
// FP64 operations (60 cycles each, a comparison 100, a division 575) is the
// serial part of every attempt: comparisons run on the integer pipe, quotients
// by omega on its reciprocal, and the divisions that are left go side by side
// in two lanes: etabar with the next averaging weight, then tau's with
// 1/sigma. With six divisions in one thread, its loads behind the dot products
// and FP64 comparisons, 1,024 FP64 iterations of a 60 x 150 LP took 17.5 ms,
// now 16.0, and of a 2,000 x 5,000 LP 19.6, now 17.9.
struct StepOut {
    double eta, w;  // the next attempt's step size; the averaging weight after an acceptance
    bool accept, sound;
};
// OVER: an infinite product beside finite norms gives etabar 0, a rejected step;
// compensated FP32 sums do not have it (they overflow to NaN), and the four
// instructions cost 70 ns an attempt.
template <bool OVER>
__device__ __forceinline__ StepOut step_rule(const StepState& s, double dx2, double dy2, double cross) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    auto nonneg_less = [](double a, double b) {  // a, b >= 0
        return __double_as_longlong(a) < __double_as_longlong(b);
    };
    const double num = __dadd_rn(__dmul_rn(s.omega, dx2), div_exact(dy2, s.omega, s.iomega));
    const bool sound = dfinite(dx2) && dfinite(dy2) && dfinite(cross);
    const bool curved = (OVER ? number(cross) : sound) && dfinite(num) && dgt0(num) && dgt0(cross);
    // lane 0: etabar; lane 1: the weight 2 / (hn + 2) after an acceptance
    const double den = lane == 1 ? (double)(s.hn + 1) + 2.0 : (curved ? __dmul_rn(2.0, cross) : 1.0);
    const double quo = __ddiv_rn(lane == 1 ? 2.0 : num, den);
    const double etabar = curved ? __shfl_sync(full, quo, 0) : CUDART_INF;
    const double w_next = __shfl_sync(full, quo, 1);
    double eta_new = CUDART_INF;
    if (dfinite(etabar)) {
        const double lo = __dmul_rn(s.f_lo, etabar), hi = __dmul_rn(s.f_hi, s.eta);
        eta_new = nonneg_less(hi, lo) ? hi : lo;
    }
    const bool accept = !nonneg_less(etabar, s.eta) || s.retries >= 20;
    const bool usable = dfinite(eta_new) && nonneg_less(1e-12, eta_new);
    double eta = s.eta;
    if (accept) {
        if (usable) eta = nonneg_less(1e12, eta_new) ? 1e12 : eta_new;
    } else {
        eta = usable ? eta_new : 1e-12;
    }
    return StepOut{eta, w_next, accept, sound};
}
template <bool OVER>
__device__ __forceinline__ void decide_step(DevCtl* c, const StepState& s, double dx2, double dy2,
                                            double cross) {
    const int lane = threadIdx.x & 31;
    const StepOut o = step_rule<OVER>(s, dx2, dy2, cross);
    const double eta = o.eta;
    const double sigma = __dmul_rn(eta, s.omega);
    // lane 0: tau; lane 1: 1 / sigma
    const double out = __ddiv_rn(lane == 1 ? 1.0 : eta, lane == 1 ? sigma : s.omega);
    const double isigma = __shfl_sync(0xffffffffu, out, 1);
    if (lane != 0) return;
    c->dots[0] = dx2;
    c->dots[1] = dy2;
    c->dots[2] = cross;
    if (!o.sound) c->nan_flag = 1;
    c->attempts += 1;
    c->eta = eta;
    if (o.accept) {
        c->parity ^= 1;
        c->hn = s.hn + 1;
        c->accepted += 1;
        c->retries = 0;
        if (s.k >= c->k_stop || c->nan_flag) c->stop = 1;
        c->k = s.k + 1;
        c->w = o.w;
        c->w_f = (float)o.w;
    } else {
        c->retries = s.retries + 1;
    }
    c->tau = out;
    c->sigma = sigma;
    c->tau_f = (float)out;
    c->sigma_f = (float)sigma;
    c->isigma = isigma;
    c->isigma_f = 1.0f / (float)sigma;
}

// The attempt's end, by one CTA that sees every partial: their fixed-order
// compensated merge (of n_primal and `gd` CTAs) and the step decision. A launch
// of at most 32 CTAs has its partials in the first warp's lanes; the other
// warps' zeros would change nothing.
template <typename T>
__device__ __forceinline__ void finish_attempt(const DualArgs<T>& a, int gd, double* smred) {
    StepState st;
    if (threadIdx.x < 32) st = load_step(a.ctl, a.fac, a.n_fac);
    Acc<T> s[3];
    for (int i = threadIdx.x; i < a.n_primal; i += kThreads) s[0].merge(a.part_primal[i]);
    for (int i = threadIdx.x; i < gd; i += kThreads) {
        s[1].merge(a.part[2 * i]);
        s[2].merge(a.part[2 * i + 1]);
    }
    if (a.n_primal <= 32 && gd <= 32) {
        if (threadIdx.x < 32)
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < 3; ++q) s[q].shfl_xor(0xffffffffu, o, 32);
    } else {
        block_merge<T, 3>(s, reinterpret_cast<Acc<T>*>(smred));
    }
    if (threadIdx.x < 32) {
        double d[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) d[q] = __shfl_sync(0xffffffffu, s[q].result_d(), 0);
        decide_step<sizeof(T) == 8>(a.ctl, st, d[0], d[1], d[2]);
    }
}

// Dual half of one attempt, fused into the A xbar SpMV:
//   t = y + sigma A xbar;  y' = t - sigma P_[rmin,rmax](t/sigma);
//   A(x'-x) = (A xbar - A x)/2   (kern_dual, src/pdhg/pdhg.cu:49-61),
// the candidate averages/commits of kern_mix2 (:129-141), the dot partials of
// kern_dots (:67-97), and -- in the last CTA to finish -- the fixed-order
// reduction of all partials (kern_dotfin, :99-125) and the step decision that
// the reference made on the host after a blocking copy (:768-794).
template <typename T, int OCC = HotCtas<T>::value>
__global__ void __launch_bounds__(kThreads, OCC) k_dual(DualArgs<T> a) {
    __shared__ __align__(16) double smred[kWarps * 4];
    FirstItem first;
    if constexpr (sizeof(T) == 8) first = first_item<T>(a.ws, a.A);
    follow_previous();
    const CtlView<T> cv = read_ctl<T>(a.ctl);
    if (cv.stop) return;
    if constexpr (sizeof(T) == 4) first = first_item<T>(a.ws, a.A);
    const int p = cv.parity, q = p ^ 1;
    DualEpi<T> epi{a.rmin, a.rmax, a.y[p], a.axc[p], a.yavg[p], a.yhat, a.y[q], a.axc[q], a.yavg[q],
                   cv.sigma, cv.isigma, cv.w, (T)0, (T)0};
    warp_rows_from<T>(a.ws, a.A, a.xbar, epi, first);
    let_next();
    T v[2] = {epi.dy2, epi.cross};
    block_sum_t<T, 2>(v, reinterpret_cast<T*>(smred));
    if (threadIdx.x == 0) {
        Acc<T> e0, e1;
        e0.s = v[0];
        e1.s = v[1];
        a.part[2 * blockIdx.x] = e0;
        a.part[2 * blockIdx.x + 1] = e1;
    }
    if (!last_cta(&a.ctl->ticket)) return;
    finish_attempt(a, gridDim.x, smred);
}

// ------------------------------------------------------------- plain SpMV
// y = A x (Spmv::mv, src/pdhg/pdhg.cu:143-157).
template <typename T, typename TO>
__global__ void __launch_bounds__(kThreads, HotCtas<T>::value)
    k_spmv(WarpSched ws, Csr<T> A, const T* x, TO* y) {
    follow_previous();
    auto f = [&](int r, const Acc<T>& acc) { y[r] = (TO)acc.result_d(); };
    PlainEpi<decltype(f)> epi{f};
    warp_rows_all<T>(ws, A, x, epi);
    let_next();
}

// -------------------------------------------------------- Ruiz equilibration
// src/pdhg/pdhg.cu:474-481: dr_i *= sqrt(max_j |a_ij| dc_j / dr_i), and
// :482-490: dc_j /= sqrt(max_i |a_ij| / dr_i * dc_j), over the warp schedule
// of the length-sorted matrix (G lanes per row). The max is order-free, and a
// rounded product or quotient with a positive constant is monotone, so the
// row's own factor is applied once, to the max; the columns' quotients by dr_i
// take its reciprocal and are correctly rounded (div_exact). The factors are
// bit-identical to the sequential host loops. With a division per entry and
// FP64 comparisons the FP64 pipe bound the sweeps: scaling a 200,000 x 500,000 LP
// (5 million nonzeros) took 4.9 ms, now 3.3; a 20,000 x 50,000 LP 0.67, now 0.47.
__device__ __forceinline__ double ruiz_max(double mx, double v) {  // both >= 0; a NaN v is left out
    const long long a = __double_as_longlong(mx), b = __double_as_longlong(v);
    return b > a && b <= 0x7ff0000000000000LL ? v : mx;
}
__global__ void __launch_bounds__(kThreads) k_ruiz_rows(WarpSched ws, const int* __restrict__ ap,
                                                          const int* __restrict__ ai,
                                                          const double* __restrict__ ax,
                                                          const double* dc, double* dr,
                                                          double* idr) {
    follow_previous();
    const int lane = threadIdx.x & 31;
    for (int w = blockIdx.x * kWarps + (threadIdx.x >> 5); w < ws.nwarps; w += gridDim.x * kWarps) {
        const int r0 = __ldg(ws.row + w), r1 = __ldg(ws.row + w + 1);
        const int lg = __ldg(ws.lg + w), G = 1 << lg, gl = lane & (G - 1);
        const int i = r0 + (lane >> lg);
        double mx = 0.0;
        if (i < r1)
            for (int p = ap[i] + gl; p < ap[i + 1]; p += G)
                mx = ruiz_max(mx, __dmul_rn(dabs(ax[p]), dc[ai[p]]));
        for (int o = G >> 1; o > 0; o >>= 1) mx = ruiz_max(mx, __shfl_xor_sync(0xffffffffu, mx, o, G));
        if (i < r1 && gl == 0) {
            double d = dr[i];
            mx = ruiz_max(0.0, __ddiv_rn(mx, d));
            if ((mx > 0) && isfinite(mx)) d = __dmul_rn(d, __dsqrt_rn(mx));
            dr[i] = d;
            idr[i] = __drcp_rn(d);
        }
    }
    let_next();
}

__global__ void __launch_bounds__(kThreads) k_ruiz_cols(WarpSched ws, const int* __restrict__ cp,
                                                          const int* __restrict__ ci,
                                                          const double* __restrict__ acx,
                                                          const double* dr, const double* idr,
                                                          double* dc) {
    follow_previous();
    const int lane = threadIdx.x & 31;
    for (int w = blockIdx.x * kWarps + (threadIdx.x >> 5); w < ws.nwarps; w += gridDim.x * kWarps) {
        const int r0 = __ldg(ws.row + w), r1 = __ldg(ws.row + w + 1);
        const int lg = __ldg(ws.lg + w), G = 1 << lg, gl = lane & (G - 1);
        const int j = r0 + (lane >> lg);
        double mx = 0.0;
        if (j < r1)
            for (int p = cp[j] + gl; p < cp[j + 1]; p += G) {
                const int i = ci[p];
                mx = ruiz_max(mx, div_exact(dabs(acx[p]), dr[i], idr[i]));
            }
        for (int o = G >> 1; o > 0; o >>= 1) mx = ruiz_max(mx, __shfl_xor_sync(0xffffffffu, mx, o, G));
        if (j < r1 && gl == 0) {
            const double d = dc[j];
            mx = ruiz_max(0.0, __dmul_rn(mx, d));
            if ((mx > 0) && isfinite(mx)) dc[j] = __ddiv_rn(d, __dsqrt_rn(mx));
        }
    }
    let_next();
}

// Pock-Chambolle pass (alpha = 1) after Ruiz, opt-in (no reference
// counterpart: the reference scales by Ruiz alone, src/pdhg/pdhg.cu:472-498).
// sum[r] = sum over row r of |a_rj| dc_j / dr_r for rows of A (rowmajor = 1)
// or over column r of |a_ir| dc_r / dr_i (rowmajor = 0), on the warp schedule
// of that orientation; both sums come from the same scaled matrix.
__global__ void __launch_bounds__(kThreads) k_pc_sums(WarpSched ws, const int* __restrict__ ptr,
                                                        const int* __restrict__ idx,
                                                        const double* __restrict__ val,
                                                        const double* __restrict__ dr,
                                                        const double* __restrict__ dc, int rowmajor,
                                                        double* __restrict__ sum) {
    const int lane = threadIdx.x & 31;
    for (int w = blockIdx.x * kWarps + (threadIdx.x >> 5); w < ws.nwarps; w += gridDim.x * kWarps) {
        const int r0 = __ldg(ws.row + w), r1 = __ldg(ws.row + w + 1);
        const int lg = __ldg(ws.lg + w), G = 1 << lg, gl = lane & (G - 1);
        const int r = r0 + (lane >> lg);
        double s = 0.0;
        if (r < r1) {
            for (int p = ptr[r] + gl; p < ptr[r + 1]; p += G) {
                const int k = idx[p];
                s += rowmajor ? fabs(val[p]) * dc[k] / dr[r] : fabs(val[p]) * dc[r] / dr[k];
            }
        }
        for (int o = G >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
        if (r < r1 && gl == 0) sum[r] = s;
    }
}

// d *= sqrt(sum) (rows, mul = 1) or d /= sqrt(sum) (columns, mul = 0) where
// the sum is positive and finite (empty rows and columns keep their factor).
__global__ void k_pc_apply(int n, const double* __restrict__ sum, int mul, double* __restrict__ d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double s = sum[i];
        if (!(s > 0) || !isfinite(s)) continue;
        d[i] = mul ? d[i] * sqrt(s) : d[i] / sqrt(s);
    }
}

// evaluate()'s at-bound bands per column (src/pdhg/pdhg.cu:206-212), the
// same FP64 operations as the inline test: tol = 1e-9 (1 + |b|), b = cu if
// finite else cl; lob = cl + tol, hib = cu - tol. A free column gives
// inf - inf = NaN there, which the inline test's x <= NaN / x >= NaN never
// passes; -inf / +inf keep that outcome for the integer-pipe compares.
__global__ void k_bands(int n, const double* __restrict__ cl, const double* __restrict__ cu,
                        double* __restrict__ lob, double* __restrict__ hib) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const double l = cl[j], u = cu[j];
        const double tol = 1e-9 * (1.0 + fabs(isfinite(u) ? u : l));
        const double lb = l + tol, hb = u - tol;
        lob[j] = isnan(lb) ? -CUDART_INF : lb;
        hib[j] = isnan(hb) ? CUDART_INF : hb;
    }
}

__global__ void k_fill(int n, double v, double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = v;
}

// :491-492 -- non-finite or non-positive factors fall back to 1.
__global__ void k_fix_scale(int n, double* __restrict__ d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (!(d[i] > 0) || !isfinite(d[i])) d[i] = 1.0;
}

// Scaled values a~_ij = a_ij dc_j / dr_i (src/pdhg/pdhg.cu:505,512), in
// place over the original FP64 values, with an FP32 copy. `rowmajor`
// selects which index array names the column.
__global__ void k_scale_matrix(int rows, const int* __restrict__ ptr, const int* __restrict__ idx,
                               double* __restrict__ val, float* __restrict__ val32,
                               const double* __restrict__ dr, const double* __restrict__ dc,
                               int rowmajor) {
    const int lane = threadIdx.x & 31;
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= rows) return;
    for (int p = ptr[r] + lane; p < ptr[r + 1]; p += 32) {
        double v;
        if (rowmajor) v = __ddiv_rn(__dmul_rn(val[p], dc[idx[p]]), dr[r]);
        else v = __ddiv_rn(__dmul_rn(val[p], dc[r]), dr[idx[p]]);
        val[p] = v;
        val32[p] = (float)v;
    }
}

// The FP32 copy of A into its padded layout (row r in [ptr4[r], ptr4[r+1]),
// a multiple of 4 slots; pads hold value 0 and the row's first index).
__global__ void k_pad4(int rows, const int* __restrict__ ptr, const int* __restrict__ idx,
                       const float* __restrict__ val, const int* __restrict__ ptr4,
                       int* __restrict__ idx4, float* __restrict__ val4) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int b = ptr[r], len = ptr[r + 1] - b, b4 = ptr4[r], len4 = ptr4[r + 1] - b4;
        for (int k = 0; k < len4; ++k) {
            idx4[b4 + k] = idx[b + (k < len ? k : 0)];
            val4[b4 + k] = k < len ? val[b + k] : 0.f;
        }
    }
}

// s = v / d (bounds) or v * d (cost), elementwise, FP64 and FP32 copies.
// out = a - b in FP64 (change between two restart points)
template <typename T>
__global__ void k_ray_diff(int n, const T* __restrict__ a, const T* __restrict__ b,
                           double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = (double)a[i] - (double)b[i];
}

// out = 1 / d (IEEE quotient, as the inline 1.0 / d it replaces)
__global__ void k_recip(int n, const double* __restrict__ d, double* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = __ddiv_rn(1.0, d[i]);
}

__global__ void k_scale_vec(int n, const double* __restrict__ v, const double* __restrict__ d,
                            int mul, double* __restrict__ out, float* __restrict__ out32) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = mul ? __dmul_rn(v[i], d[i]) : __ddiv_rn(v[i], d[i]);
        out[i] = s;
        if (out32) out32[i] = (float)s;
    }
}

// ----------------------------------------------------- reductions / norms
// out[0] = sum v^2 (sqrt if `root`), deterministic fixed-order tree.
struct NormArgs {
    const double* v;
    int n;
    double* part;
    double* out;
    unsigned int* ticket;
};
__global__ void k_sumsq(NormArgs a, int root) {
    __shared__ double red[kWarps * 4];
    follow_previous();
    let_next();
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x)
        s = fma(a.v[i], a.v[i], s);
    double v[1] = {s};
    block_sum<1>(v, red);
    if (threadIdx.x == 0) a.part[blockIdx.x] = v[0];
    if (!last_cta(a.ticket)) return;
    double t[1] = {0.0};
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads) t[0] += a.part[i];
    block_sum<1>(t, red);
    if (threadIdx.x == 0) a.out[0] = root ? sqrt(t[0]) : t[0];
}

// Power-iteration normalisation (src/pdhg/pdhg.cu:617-622): v = w / ||w||
// unless ||w|| < 1e-300, in which case the loop is over (flag latched).
__global__ void k_power_normalise(int n, const double* w, double* v,
                                  const double* nw, int* done) {
    follow_previous();
    let_next();
    if (*(volatile int*)done) return;
    const double nrm = *nw;
    if (nrm < 1e-300) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *done = 1;
        return;
    }
    const double inv = 1.0 / nrm;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[i] = w[i] * inv;
}

// sum (a-b)^2 over two vector pairs (primal-weight update,
// src/pdhg/pdhg.cu:1044-1052), FP64 accumulation.
template <typename T>
__global__ void k_diffnorms(int n, const T* __restrict__ x, const T* __restrict__ px, int m,
                            const T* __restrict__ y, const T* __restrict__ py,
                            double* part, double* out, unsigned int* ticket) {
    __shared__ double red[kWarps * 4];
    double s[2] = {0.0, 0.0};
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        double d = (double)x[i] - (double)px[i];
        s[0] = fma(d, d, s[0]);
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
        double d = (double)y[i] - (double)py[i];
        s[1] = fma(d, d, s[1]);
    }
    block_sum<2>(s, red);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = s[0];
        part[2 * blockIdx.x + 1] = s[1];
    }
    if (!last_cta(ticket)) return;
    double t[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kThreads) {
        t[0] += part[2 * i];
        t[1] += part[2 * i + 1];
    }
    block_sum<2>(t, red);
    if (threadIdx.x == 0) {
        out[0] = t[0];
        out[1] = t[1];
    }
}

template <typename T>
__global__ void k_add_const(int n, T v, T* __restrict__ x) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x[i] += v;
}

template <typename TI, typename TO>
__global__ void k_convert(int n, const TI* __restrict__ in, TO* __restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = (TO)in[i];
}

// --------------------------------------------------------------- KKT pass
// FP64 metrics of candidate pairs (x~, y~) in ORIGINAL units, one fused
// device pass replacing metrics_of + evaluate (src/pdhg/pdhg.cu:698-733,
// 173-254). Candidate v = blockIdx.y. Three launches:
//   prod      : A~ x~ and A~^T y~ over the warp schedules, stored in FP64
//               (scaled units)
//   rows      : one thread per row: pinf numerator/normaliser, prow, max |y|
//   cols      : one thread per column: reduced costs d, dinf, c^T x, the
//               column part of the Lagrangian bound; then one thread per row
//               for its row part (needs max |y| for its noise threshold) and
//               the final metrics.
// The metrics run with every lane of a warp busy (inside the warp schedule
// only 32/G lanes hold a row, and an FP64 instruction issued with partial
// lanes occupies GB300's narrow FP64 pipe as long as a full one), several
// rows or columns per thread, and their maxima reduce on the integer pipe:
// with a row per thread, the FP64 compares of the block reductions cost
// more of that pipe than the metrics themselves.
// In the solve loop the pass is enqueued behind a chunk of attempts before the
// host knows its outcome: the candidates are those of the control block's
// parity, and a chunk that has not stopped (more attempts are to come) makes
// the pass a no-op. What a check of a small LP costs is launches and the
// host's two waits: with the pass launched after the chunk's answer, two
// product kernels and four for the anchored iterates, a check took 143 us of a
// 2,000 x 5,000 LP's solve, now 114.

// One vector of each candidate, by the parity of the accepted iterate.
template <typename T>
struct Candidates {
    const T* at[2][2];  // [parity][candidate]
};
// The parity of the candidates to evaluate: the control block's; 0 without
// one; -1 while its chunk runs on. First in a kernel: waits for its predecessor.
__device__ __forceinline__ int candidate_parity(const DevCtl* ctl) {
    follow_previous();
    if (!ctl) return 0;
    return __ldcg(&ctl->stop) ? __ldcg(&ctl->parity) : -1;
}

template <typename T>
struct KktArgs {
    Candidates<T> x, y;
    const double* ax[2];                      // A~ x~ per candidate (scaled units)
    const double* aty[2];                     // A~^T y~ per candidate (scaled units)
    const double *dr, *dc;
    const double* idr;                        // 1 / dr (IEEE quotients)
    const double* idc;                        // 1 / dc (IEEE quotients)
    // evaluate()'s at-bound bands (src/pdhg/pdhg.cu:206-212), per column:
    // lob = cl + 1e-9 (1 + |b|), hib = cu - 1e-9 (1 + |b|), b = finite cu else cl
    const double *lob, *hib;
    const double *c, *cl, *cu, *rmin, *rmax;  // original units
    const T *slo, *shi;                       // scaled column bounds, iterate precision
    double cmax;
    double* part;   // >= 2 * blocks * 8 doubles
    DevMetrics* out;
    unsigned int* ticket;
    const DevCtl* ctl;  // of the chunk just enqueued, or nullptr
};

// Products of both candidates: out[v] = M v_in[v] in FP64 (the same warp
// traversal and accumulator as every other product of the engine).
template <typename T>
struct KktProdArgs {
    WarpSched ws[2];  // A, A^T
    Csr<T> M[2];
    Candidates<T> in[2];
    double* out[2][2];  // [orientation][candidate]
    int ncand;
    const DevCtl* ctl;
};
// Both candidates' products with A~ and A~^T: blockIdx.y = candidate + ncand * orientation.
template <typename T>
__global__ void __launch_bounds__(kThreads, HotCtas<T>::value) k_kkt_prod(KktProdArgs<T> a) {
    const int o = blockIdx.y >= a.ncand, v = blockIdx.y - o * a.ncand;
    const int p = candidate_parity(a.ctl);
    if (p < 0) return;
    double* __restrict__ out = a.out[o][v];
    auto f = [&](int r, const Acc<T>& acc) { out[r] = acc.result_d(); };
    PlainEpi<decltype(f)> epi{f};
    warp_rows_all<T>(a.ws[o], a.M[o], a.in[o].at[p][v], epi);
    let_next();
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_kkt_rows(KktArgs<T> a, int m) {
    __shared__ __align__(16) double smred[kWarps * 4];
    const int v = blockIdx.y, p = candidate_parity(a.ctl);
    if (p < 0) return;
    let_next();
    const T* __restrict__ yv = a.y.at[p][v];
    const double* __restrict__ axv = a.ax[v];
    double pv = 0.0, pa = 0.0, prow = 0.0, ymax = 0.0;
    // comparisons on the integer pipe (dmax, dmin, ...; see device.cuh)
    // (four rows' loads in flight: a small LP has that many per thread)
    const int step = gridDim.x * blockDim.x;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < m; i0 += 4 * step) {
        double av[4], dr[4], lo4[4], hi4[4], idr[4];
        T y4[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * step < m ? i0 + u * step : i0;
            av[u] = axv[i];
            dr[u] = a.dr[i];
            lo4[u] = a.rmin[i];
            hi4[u] = a.rmax[i];
            y4[u] = yv[i];
            idr[u] = a.idr[i];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (i0 + u * step >= m) break;
            const double Ax = av[u] * dr[u];
            const double lo = lo4[u], hi = hi4[u];
            const double vi = dmax(lo - Ax, Ax - hi);
            pv = dmax(pv, vi);
            pa = dmax(pa, dabs(dmin(dmax(Ax, lo), hi)));
            // vi / (1 + sc) <= vi: the FP64 division only when vi beats this
            // thread's running maximum (with prow = 0 that is vi > 0)
            if (dlt(prow, vi)) {
                double sc = dabs(Ax);
                if (dfinite(lo)) sc = dmax(sc, dabs(lo));
                if (dfinite(hi)) sc = dmax(sc, dabs(hi));
                prow = dmax(prow, vi / (1.0 + sc));
            }
            ymax = dmax(ymax, dabs((double)y4[u] * idr[u]));
        }
    }
    double r[4] = {pv, pa, prow, ymax};
    block_dmax<4>(r, smred);
    const int nt = gridDim.x;
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) a.part[(v * nt + blockIdx.x) * 4 + q] = r[q];
    if (!last_cta(a.ticket)) return;
    for (int cv = 0; cv < (int)gridDim.y; ++cv) {
        double t[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = threadIdx.x; b < nt; b += kThreads)
            for (int q = 0; q < 4; ++q) t[q] = dmax(t[q], a.part[(cv * nt + b) * 4 + q]);
        block_dmax<4>(t, smred);
        if (threadIdx.x == 0) {
            DevMetrics& o = a.out[cv];
            o.pv = t[0];
            o.pa = t[1];
            o.pinf = smax(t[0], 0.0) / (1.0 + t[1]);
            o.prow = t[2];
            o.ymax = t[3];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_kkt_cols(KktArgs<T> a, int n, int m) {
    __shared__ __align__(16) double smred[kWarps * 4];
    const int v = blockIdx.y, p = candidate_parity(a.ctl);
    if (p < 0) return;
    const T* __restrict__ xv = a.x.at[p][v];
    const double* __restrict__ atyv = a.aty[v];
    const double dz = 1e-8 * (1.0 + a.cmax);
    double dv = 0.0, op = 0.0, od = 0.0, unb = 0.0;
    // comparisons on the integer pipe, at-bound bands precomputed (k_bands);
    // the reduced cost multiplies by 1/dc instead of dividing by dc
    struct Col {
        double c, aty, idc, dc, cl, cu, lob, hib;
        T x, slo, shi;
    };
    auto load = [&](int j) {
        return Col{a.c[j],  atyv[j],  a.idc[j], a.dc[j],  a.cl[j], a.cu[j],
                   a.lob[j], a.hib[j], xv[j],    a.slo[j], a.shi[j]};
    };
    const int step = gridDim.x * blockDim.x;
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    Col ahead{};
    if (j < n) ahead = load(j);
    for (; j < n; j += step) {  // the next column's loads in flight
        const Col v = ahead;
        if (j + step < n) ahead = load(j + step);
        const double d = v.c + v.aty * v.idc;
        const double cl = v.cl, cu = v.cu;
        const double x = unscale_x(v.x, v.slo, v.shi, v.dc, cl, cu);
        const bool pos = dgt0(d), neg = dlt0(d);
        const bool excused = (pos && !dlt(v.lob, x)) || (neg && !dlt(x, v.hib));
        if (!excused) dv = dmax(dv, dabs(d));
        op += v.c * x;
        if (!neg) {  // d >= 0
            if (dfinite(cl)) od += d * cl;
            else if (dlt(dz, d)) unb = 1.0;
        } else {
            if (dfinite(cu)) od += d * cu;
            else if (dlt(dz, -d)) unb = 1.0;
        }
    }
    // row part of the Lagrangian bound (src/pdhg/pdhg.cu:232-242)
    const T* __restrict__ yv = a.y.at[p][v];
    const double yz = 1e-8 * (1.0 + a.out[v].ymax);
    double odr = 0.0, unbr = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const double y = (double)yv[i] * a.idr[i];
        if (dlt(yz, y)) {
            if (dfinite(a.rmax[i])) odr -= y * a.rmax[i];
            else unbr = 1.0;
        } else if (dlt(y, -yz)) {
            if (dfinite(a.rmin[i])) odr -= y * a.rmin[i];
            else unbr = 1.0;
        }
    }
    double mx[4] = {dv, unb, unbr, 0.0};
    block_dmax<4>(mx, smred);
    double sm3[4] = {op, od, odr, 0.0};
    block_sum<4>(sm3, smred);
    const int nt = gridDim.x;
    if (threadIdx.x == 0) {
        double* P = a.part + (v * nt + blockIdx.x) * 8;
        P[0] = mx[0];
        P[1] = mx[1];
        P[2] = mx[2];
        P[3] = sm3[0];
        P[4] = sm3[1];
        P[5] = sm3[2];
    }
    if (!last_cta(a.ticket)) return;
    for (int cv = 0; cv < (int)gridDim.y; ++cv) {
        double tm[4] = {0.0, 0.0, 0.0, 0.0}, ts[4] = {0.0, 0.0, 0.0, 0.0};
        for (int b = threadIdx.x; b < nt; b += kThreads) {
            const double* P = a.part + (cv * nt + b) * 8;
            for (int q = 0; q < 3; ++q) {
                tm[q] = dmax(tm[q], P[q]);
                ts[q] += P[3 + q];
            }
        }
        block_dmax<4>(tm, smred);
        block_sum<4>(ts, smred);
        if (threadIdx.x == 0) {
            DevMetrics& o = a.out[cv];
            o.dv = tm[0];
            o.dinf = tm[0] / (1.0 + a.cmax);
            o.unb_col = tm[1] > 0.0;
            o.op = ts[0];
            o.od_col = ts[1];
            o.od_row = ts[2];
            o.unb_row = tm[2] > 0.0;
            const bool bounded = !o.unb_col && !o.unb_row;
            o.od = bounded ? o.od_col + o.od_row : -CUDART_INF;
            o.gap = bounded ? smax(0.0, o.op - o.od) / (1.0 + fabs(o.op)) : CUDART_INF;
            o.finite = isfinite(o.pinf) && isfinite(o.dinf);
            const double g = isfinite(o.gap) ? o.gap : 0.0;
            o.err = smax(o.pinf, smax(o.dinf, g));
        }
    }
}

// ------------------------------------------------------ anchored iterations
// The LP seen from an FP64 anchor (x^, y^) in scaled units, rounded to FP32
// for the FP32 iteration on the deltas (x = x^ + dx, y = y^ + dy):
//   columns: c' = c~ + A~^T y^ (the reduced cost at the anchor),
//            l' = l~ - x^, u' = u~ - x^;
//   rows:    [rmin~, rmax~] - A~ x^, and y^ itself for the dual projection.
// Each value is formed in FP64 and rounded once, so it carries FP32 relative
// error of the residual, not of the original data.
__global__ void k_anchor_cols(int n, const double* __restrict__ sc, const double* __restrict__ scl,
                              const double* __restrict__ scu, const double* __restrict__ aty,
                              const double* __restrict__ xh, float* __restrict__ fc,
                              float* __restrict__ fcl, float* __restrict__ fcu) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        fc[j] = (float)(sc[j] + aty[j]);
        fcl[j] = (float)(scl[j] - xh[j]);
        fcu[j] = (float)(scu[j] - xh[j]);
    }
}

__global__ void k_anchor_rows(int m, const double* __restrict__ srmin,
                              const double* __restrict__ srmax, const double* __restrict__ ax,
                              const double* __restrict__ yh, float* __restrict__ frmin,
                              float* __restrict__ frmax, float* __restrict__ yh32) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        frmin[i] = (float)(srmin[i] - ax[i]);
        frmax[i] = (float)(srmax[i] - ax[i]);
        yh32[i] = (float)yh[i];
    }
}

// Full FP64 iterates anchor + delta of the current and the averaged one (v =
// blockIdx.y). A primal delta sitting on its FP32 shifted bound is exactly at
// the bound (the same rule as unscale_x).
struct AnchorFullArgs {
    int n, m;
    const double *xh, *yh;
    Candidates<float> dx, dy;
    const float *flo, *fhi;
    const double *scl, *scu;
    double *x[2], *y[2];
    const DevCtl* ctl;
};
__global__ void __launch_bounds__(kThreads) k_anchor_full(AnchorFullArgs a) {
    const int v = blockIdx.y, p = candidate_parity(a.ctl);
    if (p < 0) return;
    let_next();
    const float* __restrict__ dx = a.dx.at[p][v];
    const float* __restrict__ dy = a.dy.at[p][v];
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < a.n; j += gridDim.x * blockDim.x) {
        const float d = dx[j];
        a.x[v][j] = d == a.flo[j] ? a.scl[j] : (d == a.fhi[j] ? a.scu[j] : a.xh[j] + (double)d);
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.m; i += gridDim.x * blockDim.x)
        a.y[v][i] = a.yh[i] + (double)dy[i];
}

}  // namespace igx
