// Device state of VAJRA_ALGO_HALPERN and the epilogues its two iteration kernels fuse into
// the SpMVs (x+ / x_bar / Halpern for the primal half, y+ / Halpern for the dual half).
#pragma once

#include "common.cuh"

namespace vajra {

constexpr int kHist = 32;

struct HState {
    double omega, eta, tau, sigma;
    double inv_sigma;   // 1 / sigma, kept with sigma so the dual prox multiplies
    double gamma_now;   // reflection coefficient of the running phase (set by the control)
    double kkt_start, kkt_prev;
    double rel_p, rel_d, rel_gap, rel_kkt, pobj, dobj;
    double bnorm, cnorm, offset_min;
    double viol_p_rel, viol_p_abs, viol_d_abs;   // status-guard maxima of the last check
    double hist[kHist];
    long long k_base;
    long long total;
    long long phase_iters[2];
    long long stop_iter;
    int hist_n;
    int phase;          // 0: FP32 phase of the mixed mode, 1: FP64
    int stop;
    int status;
    int restart_count;
    int restart_flag;
    int switch_flag;
    int pad;
    // first iteration of every chunk of the cluster path: nanoseconds of its two halves
    double t_primal_ns[2], t_dual_ns[2];   // per phase
    long long t_samples[2];
};

constexpr int kStatusOptimal = 1;
constexpr int kStatusIterLimit = 6;
constexpr int kStatusTimeLimit = 7;
constexpr int kStatusNumerical = 9;

// One column's primal half: x+ and x_bar from the row sum v = (A^T y)_j, and the Halpern step.
template <typename T>
__device__ __forceinline__ void halpern_primal(T xo, T v, T c, T cl, T cu, T x0, T tau, T w1, T w0, T g, T* xp_out,
                                               T* xb_out, T* x_out) {
    T xp = xo - tau * (c + v);
    xp = xp < cl ? cl : (xp > cu ? cu : xp);
    *xp_out = xp;
    *xb_out = xp + xp - xo;
    *x_out = w1 * ((T(1) + g) * xp - g * xo) + w0 * x0;
}
// One row's dual half: y+ from the row sum w = (A x_bar)_i, and the Halpern step.
template <typename T>
__device__ __forceinline__ void halpern_dual(T yo, T w, T rl, T ru, T y0, T sigma, T inv_sigma, T w1, T w0, T g,
                                             T* yp_out, T* y_out) {
    const T yh = yo + sigma * w;
    T q = yh * inv_sigma;
    q = q < rl ? rl : (q > ru ? ru : q);
    const T yp = yh - sigma * q;
    *yp_out = yp;
    *y_out = w1 * ((T(1) + g) * yp - g * yo) + w0 * y0;
}

// At the last iteration of a chunk (write_cand) the epilogues also keep T(z) (xc, yc) and
// the point it was taken from (xprev, yprev) for the check.
// Both epilogues are two-phase (see spmv.cuh): pre() issues every load that does not need
// the row sum -- the read-only vectors and the device scalars through the read-only path
// (they are written only by other kernels) -- before the SpMV's own loads.
template <typename T>
struct EpiHPrimal {
    const T* c; const T* cl; const T* cu; const T* x0;
    T* x; T* xb; T* xc; T* xprev;
    const HState* st;
    const double* hw;   // Halpern weights of this chunk: hw[2kk] = (k+1)/(k+2), hw[2kk+1] = 1/(k+2)
    int kk, phase, write_cand;
    struct Pre { T xo, c, cl, cu, x0, tau, w1, w0, g; };
    __device__ bool active() const { return st->stop == 0 && st->phase == phase; }
    __device__ Pre pre(int j) const {
        Pre p;
        p.w1 = static_cast<T>(__ldg(hw + 2 * kk));
        p.w0 = static_cast<T>(__ldg(hw + 2 * kk + 1));
        p.tau = static_cast<T>(__ldg(&st->tau));
        p.g = static_cast<T>(__ldg(&st->gamma_now));
        p.xo = x[j];
        p.c = __ldg(c + j);
        p.cl = __ldg(cl + j);
        p.cu = __ldg(cu + j);
        p.x0 = __ldg(x0 + j);
        return p;
    }
    template <typename Acc>
    __device__ void operator()(int j, Acc v, const Pre& p) const {
        T xp, xbn, xn;
        halpern_primal(p.xo, static_cast<T>(v), p.c, p.cl, p.cu, p.x0, p.tau, p.w1, p.w0, p.g, &xp, &xbn, &xn);
        xb[j] = xbn;
        x[j] = xn;
        if (write_cand) { xc[j] = xp; xprev[j] = p.xo; }
    }
    template <typename Acc>
    __device__ void operator()(int j, Acc v) const { (*this)(j, v, pre(j)); }
};

template <typename T>
struct EpiHDual {
    const T* rl; const T* ru; const T* y0;
    T* y; T* yc; T* yprev;
    const HState* st;
    const double* hw;   // Halpern weights of this chunk (as in EpiHPrimal)
    int kk, phase, write_cand;
    struct Pre { T yo, rl, ru, y0, sigma, inv_sigma, w1, w0, g; };
    __device__ bool active() const { return st->stop == 0 && st->phase == phase; }
    __device__ Pre pre(int i) const {
        Pre p;
        p.w1 = static_cast<T>(__ldg(hw + 2 * kk));
        p.w0 = static_cast<T>(__ldg(hw + 2 * kk + 1));
        p.sigma = static_cast<T>(__ldg(&st->sigma));
        p.inv_sigma = static_cast<T>(__ldg(&st->inv_sigma));
        p.g = static_cast<T>(__ldg(&st->gamma_now));
        p.yo = y[i];
        p.rl = __ldg(rl + i);
        p.ru = __ldg(ru + i);
        p.y0 = __ldg(y0 + i);
        return p;
    }
    template <typename Acc>
    __device__ void operator()(int i, Acc w, const Pre& p) const {
        T yp, yn;
        halpern_dual(p.yo, static_cast<T>(w), p.rl, p.ru, p.y0, p.sigma, p.inv_sigma, p.w1, p.w0, p.g, &yp, &yn);
        y[i] = yn;
        if (write_cand) { yc[i] = yp; yprev[i] = p.yo; }
    }
    template <typename Acc>
    __device__ void operator()(int i, Acc w) const { (*this)(i, w, pre(i)); }
};

// The Halpern weights of the next chunk from the current inner counter: one thread per step.
__device__ __forceinline__ void halpern_weights(const HState* st, int len, double* hw, int t, int stride) {
    const long long kb = st->k_base;
    for (int kk = t; kk < len; kk += stride) {
        const double k = static_cast<double>(kb + kk);
        hw[2 * kk] = (k + 1.0) / (k + 2.0);
        hw[2 * kk + 1] = 1.0 / (k + 2.0);
    }
}

static __global__ void k_halpern_weights(const HState* st, int len, double* hw) {
    halpern_weights(st, len, hw, threadIdx.x, blockDim.x);
}

struct EpiStoreActive {
    double* out;
    const HState* st;
    int phase;
    __device__ bool active() const { return st->stop == 0 && st->phase == phase; }
    template <typename Acc> __device__ void operator()(int i, Acc s) const { out[i] = static_cast<double>(s); }
};

}  // namespace vajra
