// k_krylov.cu -- SELL-32 SpMV, fused CG updates with deterministic last-block
// reductions, and level-scheduled ILU(0).
//
// Reductions: every 256 threads write one FP64 partial sum.  Where the next kernel needs the total, each of
// its blocks adds the partials (sum_parts); where the preconditioner must know whether to run (the residual
// norms), the last block to arrive (arrival counter + threadfence) adds them and updates the scalars.
// The order is fixed and the same either way, so results are run-to-run reproducible.  At 255k unknowns the
// sums of p.q and z.r with their fences and arrivals took 9.2 and 7.0 us, now 5.9 and 3.3, and the kernels that
// add the partials 1 to 4 us more than before; a CG iteration 143 us, now 139, in FP64 on 38k unknowns 138, now 128.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "bulk.cuh"
#include "krylov.h"
#include "sell.cuh"

namespace porsol {

namespace {

constexpr int RB = 256;           // threads per block of the plain vector kernels
constexpr int RED_THREADS = 1024;   // of the reducing kernels at most

// Launch shape of the reducing kernels: at most two blocks per SM (the partials the next kernel adds), of 256
// threads while those cover n (every SM works on small systems), of up to 1024 beyond, then grid-stride.
// The shape depends only on n and the device, so the summation order stays fixed.
struct RedShape {
    int blocks, threads;
    int partials() const { return blocks * (threads / RB); }
};
RedShape red_shape(int n)
{
    static int cap = 0;
    if (cap == 0) {
        int dev = 0, sms = 0;
        PORSOL_CUDA(cudaGetDevice(&dev));
        PORSOL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        cap = std::max(1, 2 * sms);
    }
    int t = 256;
    while (t < RED_THREADS && div_up(std::max(n, 1), t) > cap) t *= 2;
    return {std::min(div_up(std::max(n, 1), t), cap), t};
}

template <class V>
__device__ __forceinline__ V warp_sum(V v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One partial sum per 256 threads (RB), written to part.  The per-thread value type V is the vector type: FP32
// vectors are summed in FP32 within a warp (32 terms) and in FP64 from there on, so the FP64 unit (a small
// fraction of GB300's FP32 rate) only sees one value per warp.
template <int K = 0, class V>
__device__ __forceinline__ void block_partials(V v0, double* __restrict__ part)
{
    __shared__ double ws[RED_THREADS / 32];
    const double v = double(warp_sum<V>(v0));
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double t = threadIdx.x < (blockDim.x >> 5) ? ws[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x < (blockDim.x >> 5) && threadIdx.x % 8 == 0)
            part[blockIdx.x * (blockDim.x / RB) + threadIdx.x / 8] = t;
    }
}

// Total of the preceding kernel's partials (same launch shape), in thread 0: the partials over RB threads, a
// tree per warp, the warps in order.  Thread 0 goes on to form the scalars the block needs from it and hands
// them over in shared memory: a warp's FP64 instruction holds the FP64 pipe of the SM for 16 cycles, so a
// quotient in each of 64 warps would cost more than the whole vector operation (9 us against 4 at 255k unknowns).
template <int K = 0>   // a kernel's sums: K of each its own (their shared memory then needs no barrier between)
__device__ __forceinline__ double sum_parts(const volatile double* part)
{
    __shared__ double ws[RB / 32];
    if (threadIdx.x < RB) {
        const int n = int(gridDim.x * (blockDim.x / RB));
        double s = 0.0;
        for (int b = threadIdx.x; b < n; b += RB) s += part[b];
        s = warp_sum<double>(s);
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    }
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
#pragma unroll
        for (int w = 0; w < RB / 32; ++w) t += ws[w];
    return t;
}

// Partials, and their total in the last block to arrive.  Returns true in thread 0 of that block.
template <class V>
__device__ bool block_reduce_last(V v0, double* partial, unsigned int* counter, double* total)
{
    __shared__ bool amlast;
    block_partials(v0, partial);
    if (threadIdx.x < 32) {
        __threadfence();
        __syncwarp();
        if (threadIdx.x == 0) amlast = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!amlast) return false;
    __threadfence();
    *total = sum_parts(partial);
    if (threadIdx.x == 0) *counter = 0u;
    return threadIdx.x == 0;
}

// Row r of a SELL matrix times x, accumulated in the vector type TX (FP32 rows stay on the
// FP32 pipe).
template <class TV, class TX, class CI>
__device__ __forceinline__ TX sell_row(const int* __restrict__ sp, const CI* __restrict__ col,
                                       const TV* __restrict__ val, const TX* __restrict__ x, int r)
{
    return sell_dot<TX>(sp, col, val, r, [x](int j) { return x[j]; });
}

template <class TV, class TX>
__global__ void k_spmv(int n, const int* __restrict__ sp, const int* __restrict__ col, const TV* __restrict__ val,
                       const TX* __restrict__ x, TX* __restrict__ y)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    y[r] = TX(sell_row(sp, col, val, x, r));
}

template <class TV, class TX>
__global__ void k_residual(int n, const int* __restrict__ sp, const int* __restrict__ col,
                           const TV* __restrict__ val, const TX* __restrict__ x, const TX* __restrict__ b,
                           TX* __restrict__ y)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    y[r] = b[r] - sell_row(sp, col, val, x, r);
}

// r = b - A x; def0 = ||r||
template <class TV, class T, class CI>
__global__ void __launch_bounds__(RED_THREADS, 2) k_cg_init(int n, const int* __restrict__ sp, const CI* __restrict__ col,
                                                const TV* __restrict__ val, const T* __restrict__ x,
                                                const T* __restrict__ b, T* __restrict__ r, CgDev* st,
                                                double* partial, unsigned int* counter, CgHostView* hv)
{
    chain_wait();
    T v = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const T ri = b[i] - sell_row(sp, col, val, x, i);
        r[i] = ri;
        v += ri * ri;
    }
    double tot;
    if (block_reduce_last<T>(v, partial, counter, &tot)) {
        const double d0 = sqrt(tot);
        st->def0 = d0;
        st->def = d0;
        st->iter = 0;
        st->breakdown = 0;
        st->converged = (d0 < 1e-30) ? 1 : 0;
        st->stop = st->converged;
        hv->def0 = d0;
        hv->def = d0;
        hv->iter = 0;
        hv->converged = st->converged;
        hv->stop = st->stop;
        hv->breakdown = 0;
    }
}

// partial sums of z . r
template <class T>
__global__ void __launch_bounds__(RED_THREADS, 2) k_dot_zr(int n, const T* __restrict__ z, const T* __restrict__ r,
                                                           const CgDev* st, double* __restrict__ part)
{
    chain_wait();
    if (st->stop) return;
    T v = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v += z[i] * r[i];
    block_partials(v, part);
}

// q = A p; partial sums of p . q
template <class TV, class T, class CI>
__global__ void __launch_bounds__(RED_THREADS, 2) k_spmv_pq(int n, const int* __restrict__ sp, const CI* __restrict__ col,
                                                const TV* __restrict__ val, const T* __restrict__ p,
                                                T* __restrict__ q, const CgDev* st, double* __restrict__ part)
{
    chain_wait();
    if (st->stop) return;
    T v = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const T qi = sell_row(sp, col, val, p, i);
        q[i] = qi;
        v += p[i] * qi;
    }
    block_partials(v, part);
}

// lambda = rho / (p . q); x += lambda p; r -= lambda q; the preconditioner's start from r; def = ||r|| and the
// convergence test
template <class T>
__global__ void __launch_bounds__(RED_THREADS, 2) k_cg_update(int n, T* __restrict__ x, T* __restrict__ r,
                                                  const T* __restrict__ p, const T* __restrict__ q, CgDev* st,
                                                  const double* __restrict__ pq,
                                                  typename Precond<T>::Start start, double* partial,
                                                  unsigned int* counter, CgHostView* hv)
{
    chain_wait();
    if (st->stop) return;
    __shared__ T s_lambda;
    const double alpha = sum_parts(pq);
    if (threadIdx.x == 0) s_lambda = T(st->rho[st->iter & 1] / alpha);
    __syncthreads();
    const T lambda = s_lambda;
    T v = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        x[i] = x[i] + lambda * p[i];
        const T ri = r[i] - lambda * q[i];
        r[i] = ri;
        if (start.dinv) {
            const T s = start.dinv[i] * ri;
            start.r0[i] = s;
            start.d[i] = s * start.inv_theta;
        }
        v += ri * ri;
    }
    double tot;
    if (block_reduce_last<T>(v, partial, counter, &tot)) {
        const double def = sqrt(tot);
        st->def = def;
        st->iter += 1;
        if (!(alpha > 0.0) || !isfinite(def)) st->breakdown = 1;
        if (def < st->def0 * st->tol || def < 1e-30) st->converged = 1;
        st->stop = st->converged || st->breakdown || st->iter >= st->maxit;
        hv->def = def;
        hv->iter = st->iter;
        hv->converged = st->converged;
        hv->breakdown = st->breakdown;
        hv->stop = st->stop;
    }
}

// rho = z . r; beta = rho / last rho; p = z + beta p (first: p = z)
template <class T>
__global__ void __launch_bounds__(RED_THREADS, 2) k_cg_direction(int n, const T* __restrict__ z, T* __restrict__ p,
                                                                 CgDev* st, const double* __restrict__ zr,
                                                                 int first)
{
    chain_wait();
    if (st->stop) return;
    __shared__ T s_beta;
    const double rho = sum_parts(zr);
    const int it = st->iter;
    if (threadIdx.x == 0) s_beta = first ? T(0) : T(rho / st->rho[(it + 1) & 1]);
    __syncthreads();
    const T beta = s_beta;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p[i] = first ? z[i] : z[i] + beta * p[i];
    if (blockIdx.x == 0 && threadIdx.x == 0) st->rho[it & 1] = rho;
}

template <class TA, class TB>
__global__ void k_convert(long long n, const TA* __restrict__ a, TB* __restrict__ b)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) b[i] = TB(a[i]);
}

__global__ void k_axpy_add(int n, const double* __restrict__ y, double* __restrict__ x)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += y[i];
}

__global__ void k_dirichlet_guess(int n, const int* __restrict__ sp, const int* __restrict__ col,
                                  const int* __restrict__ rowlen, const double* __restrict__ val,
                                  const double* __restrict__ b, double* __restrict__ x)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int s = r >> 5, lane = r & 31;
    const int base = sp[s];
    bool isD = true;
    double d = 0.0;
    for (int t = 0; t < rowlen[r]; ++t) {
        const int k = base + t * 32 + lane;
        if (col[k] == r) d = val[k];
        else if (val[k] != 0.0) isD = false;
    }
    x[r] = isD ? b[r] / d : 0.0;
}

template <class T>
__global__ void __launch_bounds__(RED_THREADS, 2) k_norm2(int n, const T* __restrict__ x, double* partial,
                                                          unsigned int* counter, double* out)
{
    T v = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v += x[i] * x[i];
    double tot;
    if (block_reduce_last<T>(v, partial, counter, &tot)) *out = tot;
}

// ---------------- mixed-precision CG with reliable updates ----------------
constexpr int RC_STAGE = 128;   // iterations without a replacement after which the recurrence is guarded

__device__ __forceinline__ void rc_publish(const RcDev* st, CgHostView* hv)
{
    hv->def0 = st->def0;
    hv->def = st->true_def;
    hv->iter = st->iter;
    hv->converged = st->converged;
    hv->breakdown = st->breakdown;
    hv->stop = st->stop;
}

// r64 = b - A x (FP64); def0 = sigma = ||r64||
template <class CI>
__global__ void __launch_bounds__(RED_THREADS, 2) k_rc_init(int n, const int* __restrict__ sp, const CI* __restrict__ col,
                                                const double* __restrict__ val, const double* __restrict__ x,
                                                const double* __restrict__ b, double* __restrict__ r64, RcDev* st,
                                                double* partial, unsigned int* counter, CgHostView* hv)
{
    chain_wait();
    double v = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double ri = b[i] - sell_row(sp, col, val, x, i);
        r64[i] = ri;
        v += ri * ri;
    }
    double tot;
    if (block_reduce_last<double>(v, partial, counter, &tot)) {
        const double d = sqrt(tot);
        st->def0 = st->true_def = st->sigma = d;
        st->isig = d > 0.0 ? 1.0 / d : 0.0;
        st->factor = 1.0f;
        st->iter = st->last = st->nrep = st->replaced = st->breakdown = st->guard = st->restart = 0;
        st->converged = (d < 1e-30) ? 1 : 0;
        st->stop = st->converged || !isfinite(d);
        st->breakdown = !isfinite(d);
        rc_publish(st, hv);
    }
}

// at the start and after a replacement: r = r64 / sigma in FP32, p in the new units, the preconditioner's
// start from r.  A breakdown found by k_rc_update stops the solve here: threads that still read the flag do
// the same work either way.
__global__ void k_rc_rescale(int n, const double* __restrict__ r64, float* __restrict__ r, float* __restrict__ p,
                             RcDev* st, Precond<float>::Start start, int init, CgHostView* hv)
{
    chain_wait();
    const int stop = st->stop, broken = st->breakdown, replaced = st->replaced;
    if (stop || broken || !(init || replaced)) {
        if (broken && !stop && blockIdx.x == 0 && threadIdx.x == 0) {
            st->stop = 1;
            rc_publish(st, hv);
        }
        return;
    }
    const double is = st->isig;
    const float f = st->factor;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float ri = float(r64[i] * is);
        r[i] = ri;
        if (start.dinv) {
            const float s = start.dinv[i] * ri;
            start.r0[i] = s;
            start.d[i] = s * start.inv_theta;
        }
        if (!init) p[i] *= f;
    }
}

// q = A32 p; partial sums of p . q, guarded (RcDev) of p . r too
template <class CI>
__global__ void __launch_bounds__(RED_THREADS, 2) k_rc_pq(int n, const int* __restrict__ sp, const CI* __restrict__ col,
                                              const float* __restrict__ val, const float* __restrict__ p,
                                              const float* __restrict__ r, float* __restrict__ q, const RcDev* st,
                                              double* __restrict__ pq, double* __restrict__ pr)
{
    chain_wait();
    if (st->stop) return;
    float v = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float qi = sell_row(sp, col, val, p, i);
        q[i] = qi;
        v += p[i] * qi;
    }
    block_partials<0>(v, pq);
    if (st->guard) {   // a pass of its own: a branch in the loop above costs 1.6 us of 51.4 at 3M rows
        float w = 0.0f;
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) w += p[i] * r[i];
        block_partials<1>(w, pr);
    }
}

// alpha = rho / (p . q) (guarded: (p . r) / (p . q)); x += sigma alpha p (FP64); r -= alpha q; the
// preconditioner's start from r; partial sums of r . r.  Where the curvature is not positive nothing changes
// (alpha = 0): the direction starts anew from z, guarded.  That happens once: in a direction just started anew, or
// in the guarded form, which keeps the directions conjugate, the matrix itself is not positive definite and the
// solve stops (restarting on and on, indefinite systems ran up to 3000 iterations into an overflow).
__global__ void __launch_bounds__(RED_THREADS, 2) k_rc_update(int n, double* __restrict__ x, float* __restrict__ r,
                                                  const float* __restrict__ p, const float* __restrict__ q,
                                                  RcDev* st, const double* __restrict__ pq,
                                                  const double* __restrict__ pr, Precond<float>::Start start,
                                                  double* __restrict__ part)
{
    chain_wait();
    if (st->stop) return;
    __shared__ double s_sa;
    __shared__ float s_a;
    const int guard = st->guard;
    const double curv = sum_parts<0>(pq);
    const double pr_sum = guard ? sum_parts<1>(pr) : 0.0;
    if (threadIdx.x == 0) {
        const bool ok = curv > 0.0 && isfinite(curv);
        const double alpha = ok ? (guard ? pr_sum : st->rho[st->iter & 1]) / curv : 0.0;
        s_sa = st->sigma * alpha;
        s_a = float(alpha);
        if (blockIdx.x == 0) {
            st->pq = curv;
            st->restart = !ok;
            if (!ok && (st->fresh || guard || !isfinite(curv))) st->breakdown = 1;   // k_rc_rescale stops the solve
        }
    }
    __syncthreads();
    const double sa = s_sa;
    const float a = s_a;
    float v = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        x[i] += sa * double(p[i]);
        const float ri = r[i] - a * q[i];
        r[i] = ri;
        if (start.dinv) {
            const float s = start.dinv[i] * ri;
            start.r0[i] = s;
            start.d[i] = s * start.inv_theta;
        }
        v += ri * ri;
    }
    block_partials(v, part);
}

// Replacement, when the iterated residual has dropped by delta since the last one or its estimate reaches
// the tolerance: r64 = b - A x in FP64, convergence decided on this true residual only; otherwise the kernel
// ends at once.
template <class CI>
__global__ void __launch_bounds__(RED_THREADS) k_rc_true(int n, const int* __restrict__ sp, const CI* __restrict__ col,
                                                const double* __restrict__ val, const double* __restrict__ x,
                                                const double* __restrict__ b, double* __restrict__ r64, RcDev* st,
                                                const double* __restrict__ rr, double* partial,
                                                unsigned int* counter, CgHostView* hv)
{
    chain_wait();
    if (st->stop) return;
    __shared__ int s_replace;
    const double ss = sum_parts(rr);
    if (threadIdx.x == 0) {
        const double defs = sqrt(ss), est = defs * st->sigma;
        s_replace = defs < st->delta || est < st->tol * st->def0 || est < 1e-30 || !isfinite(defs) ||
                    st->iter + 1 >= st->maxit;
        if (!s_replace && blockIdx.x == 0) {
            st->replaced = 0;   // k_rc_zr counts the iteration
            if (st->restart || st->iter + 1 - st->last >= RC_STAGE) st->guard = 1;
        }
    }
    __syncthreads();
    if (!s_replace) return;
    double v = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double ri = b[i] - sell_row(sp, col, val, x, i);
        r64[i] = ri;
        v += ri * ri;
    }
    double tot;
    if (block_reduce_last<double>(v, partial, counter, &tot)) {
        const double d = sqrt(tot);
        const int it = st->iter + 1;
        st->true_def = d;
        st->nrep += 1;
        st->iter = st->last = it;
        st->replaced = 1;
        if (!isfinite(d)) {
            st->breakdown = 1;
            st->stop = 1;
        } else if (d < st->tol * st->def0 || d < 1e-30) {
            st->converged = 1;
            st->stop = 1;
        } else if (it >= st->maxit) {
            st->stop = 1;
        } else {
            // continue on the rescaled system: r and p in units of the new sigma
            const double f = st->sigma / d;
            st->factor = float(f);
            st->rho[(it + 1) & 1] *= f * f;
            st->sigma = d;
            st->isig = 1.0 / d;
        }
        rc_publish(st, hv);
    }
}

// partial sums of z . r (guarded: z . q); counts the iteration where no replacement did
__global__ void __launch_bounds__(RED_THREADS, 2) k_rc_zr(int n, const float* __restrict__ z, const float* __restrict__ r,
                                              const float* __restrict__ q, RcDev* st, double* __restrict__ part,
                                              int init)
{
    chain_wait();
    if (st->stop) return;
    const float* __restrict__ w = st->guard ? q : r;
    float v = 0.0f;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v += z[i] * w[i];
    block_partials(v, part);
    if (blockIdx.x == 0 && threadIdx.x == 0 && !init && !st->replaced) st->iter += 1;
}

// rho = z . r; beta = rho / last rho (guarded: -(z . q) / (p . q), q in the units before a replacement);
// p = z + beta p (at the start and anew: p = z)
__global__ void __launch_bounds__(RED_THREADS, 2) k_rc_direction(int n, const float* __restrict__ z, float* __restrict__ p,
                                                                 RcDev* st, const double* __restrict__ zr, int init)
{
    chain_wait();
    if (st->stop) return;
    __shared__ float s_beta;
    const bool fresh = init || st->restart;
    const double sum = sum_parts(zr);
    if (threadIdx.x == 0) {
        const int it = st->iter;
        const bool guard = !init && st->guard;
        if (fresh) s_beta = 0.0f;
        else if (guard) s_beta = float(-sum / (st->pq * double(st->replaced ? st->factor : 1.0f)));
        else s_beta = float(sum / st->rho[(it + 1) & 1]);
        if (blockIdx.x == 0) {
            st->rho[it & 1] = sum;
            st->fresh = fresh;
        }
    }
    __syncthreads();
    const float beta = s_beta;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        p[i] = fresh ? z[i] : z[i] + beta * p[i];
}

// ---------------- ILU(0) ----------------
__device__ __forceinline__ int sell_slot(const int* sp, int r, int t) { return sp[r >> 5] + t * 32 + (r & 31); }

// Factorisation of one level with a warp per row (rows of at most 32 entries): lane t holds
// entry t of row i.  The finished rows j < i it needs are read lane by entry, two at a time ahead of
// their use, and lane t finds its column in row j among the lanes.  Each entry takes the updates of the
// serial walk in its order.  A level of the 10^3 cube takes about a launch latency instead of the 27 us
// of one thread walking its row's merges load by load.
__global__ void __launch_bounds__(128) k_ilu_factor_warp(int nrows, const int* __restrict__ rows,
                                                         const int* __restrict__ sp, const int* __restrict__ col,
                                                         const int* __restrict__ rowlen,
                                                         const int* __restrict__ diag, double* lu, int* status)
{
    chain_wait();
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= nrows) return;   // whole warps
    const int lane = threadIdx.x & 31;
    const int i = rows[q], len = rowlen[i];
    const int k = sell_slot(sp, i, lane);
    const int ci = lane < len ? col[k] : INT_MAX;
    double a = lane < len ? lu[k] : 0.0;
    const int nl = __popc(__ballot_sync(0xffffffffu, ci < i));   // entries are sorted: the first nl are lower
    auto fetch = [&](int t, int& cj, double& aj, double& pj) {
        const int j = __shfl_sync(0xffffffffu, ci, t);
        const int kj = sell_slot(sp, j, lane);
        const bool in = lane < rowlen[j];
        cj = in ? col[kj] : INT_MAX;
        aj = in ? lu[kj] : 0.0;
        pj = lu[diag[j]];
    };
    int cj = INT_MAX, cn = INT_MAX;
    double aj = 0.0, an = 0.0, pj = 0.0, pn = 0.0;
    if (nl > 0) fetch(0, cj, aj, pj);
    for (int t = 0; t < nl; ++t) {
        if (t + 1 < nl) fetch(t + 1, cn, an, pn);
        if (lane == t) a *= pj;                     // L_ij = a_ij * inv(a_jj)
        const double lij = __shfl_sync(0xffffffffu, a, t);
        // a_ik -= L_ij a_jk for k > j present in both rows
        const int lj = __popc(__ballot_sync(0xffffffffu, cj != INT_MAX));
        for (int u = 0; u < lj; ++u) {
            const int c = __shfl_sync(0xffffffffu, cj, u);
            const double v = __shfl_sync(0xffffffffu, aj, u);
            if (lane > t && lane < len && c == ci) a -= lij * v;
        }
        cj = cn;
        aj = an;
        pj = pn;
    }
    if (ci == i) {
        if (!(fabs(a) > 0.0) || !isfinite(a)) atomicOr(status, ST_NONFINITE);
        a = 1.0 / a;
    }
    if (lane < len) lu[k] = a;
}

// the factor's values into the sweep's step records
__global__ void k_ilu_pack(int nval, const int* __restrict__ pos, const int* __restrict__ slot,
                           const double* __restrict__ lu, double* __restrict__ blob)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nval) blob[pos[e]] = lu[slot[e]];
}

// Steps [s0, s1) of the sweep by one block: a step is (part of) a level, a thread a row, a barrier ends the
// step.  What bounds it is the chain from level to level: the operands from shared memory, the row's five
// dependent FP64 products (a warp's FP64 instruction takes 64 clocks, also when predicated off) and the
// barrier, 0.57 us in all.  The step records do not depend on the sweep, so a warp of its own brings them
// into a ring of nst stages by bulk copies ahead of their use.  With SZ the whole vector lives in shared
// memory, copied in from r and out to z; without, z holds the right-hand side on entry.  The products are
// added in the row's order, as the per-level kernels do; a padding entry multiplies the 0 behind the
// vector.  10^3 cube (3300 rows, 84 + 84 levels): one application takes 99 us in one launch, and took 510 us in
// 168 launches.  Measured and not kept: the records prefetched into registers (130 us), one of the row
// threads issuing the copies (163 us), each row's operands loaded a step ahead by its own thread (117 us).
// Every wait is bounded.  A thread whose wait ran out skips its row and says so in shared memory; all threads
// read that behind the step's barrier and leave together one step later, when the load is long done (a voting
// barrier cost 7 us of the 99): the block sets ST_TIMEOUT and waits (bounded) for its copies.  GATED (the
// self-test): thread `gate` also waits, in the first step, at a barrier for bytes that no copy delivers.
constexpr int ILU_ROWS = 256;              // rows of a step at most: a thread each, and one warp that copies
constexpr int ILU_TB = ILU_ROWS + 32;
constexpr int ILU_AHEAD = 8;               // products of a row whose operands are loaded before the first sum
constexpr unsigned ILU_STAGE = 12 * 1024;  // bytes of a stage: the largest step record
constexpr int ILU_STAGES = 8;
constexpr size_t ILU_SMEM = 220 * 1024;

// acc - sum over the first W columns of v[k] z[c[k]] for one row (operands cp apart), in column order.  W is
// the same for the whole step, so the unused products of shorter bodies are not issued at all.
template <int W, class CI, class Z>
__device__ __forceinline__ double ilu_row(double acc, const double* v, const CI* c, int cp, Z z)
{
    double a[W > 0 ? W : 1], x[W > 0 ? W : 1];
#pragma unroll
    for (int k = 0; k < W; ++k) {
        a[k] = v[k * cp];
        x[k] = z(int(c[k * cp]));
    }
#pragma unroll
    for (int k = 0; k < W; ++k) acc -= a[k] * x[k];
    return acc;
}

// Step record: a header (rows, W, upper, -), W columns of cp doubles (cp: rows rounded up to 8), for the
// upper triangle cp inverted pivots, cp row numbers, W columns of cp column numbers.
// steps: (offset in the records / 16, bytes).
template <class CI, bool SZ, bool GATED = false>
__global__ void __launch_bounds__(ILU_TB) k_ilu_steps(int s0, int s1, const int2* __restrict__ steps,
                                                      const unsigned char* __restrict__ blob,
                                                      const double* __restrict__ r, double* z, int n, int nst,
                                                      const int* stop, int* status, int gate)
{
    chain_wait();
    if (*stop) return;
    extern __shared__ __align__(128) unsigned char sm[];   // the stages' barriers and the gate, the ring, the vector
    unsigned char* ring = sm + 128;
    double* zs = reinterpret_cast<double*>(ring + size_t(nst) * ILU_STAGE);
    const int i = threadIdx.x;
    const bool copier = i == ILU_ROWS;
    const unsigned bars = smem_u32(sm), gate_bar = bars + 8 * ILU_STAGES;
    volatile int* gave_up = reinterpret_cast<volatile int*>(sm + 8 * (ILU_STAGES + 1));   // by the step's parity
    int issued = s0, seen = s0;   // steps whose copies were started and have landed (copier)
    auto issue = [&](const int2& t, int stage) {
        ++issued;
        mbar_expect(bars + 8 * stage, unsigned(t.y));
        bulk_copy(smem_u32(ring + size_t(stage) * ILU_STAGE), blob + 16 * size_t(t.x), unsigned(t.y), bars + 8 * stage);
    };
    const int2 none = make_int2(0, 0);
    int2 next = none;
    if (copier) {
        for (int k = 0; k < nst; ++k) mbar_init(bars + 8 * k);
        if (GATED) mbar_init(gate_bar);
        mbar_init_fence();
        if (GATED) mbar_expect(gate_bar, 16);
        gave_up[0] = gave_up[1] = 0;
        for (int k = 0; k < nst && s0 + k < s1; ++k) issue(steps[s0 + k], k);
        next = s0 + nst < s1 ? steps[s0 + nst] : none;
    }
    if (SZ) {
        for (int k = i; k < n; k += ILU_TB) zs[k] = r[k];
        if (i == 0) zs[n] = 0.0;
    }
    auto value = [&](int j) { return SZ ? zs[j] : (j < n ? z[j] : 0.0); };
    auto leave = [&] {
        if (!copier) return;
        atomicOr(status, ST_TIMEOUT);
        for (int t = seen; t < issued; ++t)   // the copies still in flight
            mbar_wait_bounded(bars + 8 * ((t - s0) % nst), unsigned((t - s0) / nst) & 1u, BULK_WAIT_NS);
    };
    int stage = 0, late = 0;
    unsigned parity = 0;
    __syncthreads();   // barriers initialised, vector in place
    for (int s = s0; s < s1; ++s) {
        bool landed = mbar_wait_bounded(bars + 8 * stage, parity, BULK_WAIT_NS);
        if (GATED && i == gate && s == s0) landed = mbar_wait_bounded(gate_bar, 0, BULK_WAIT_NS) && landed;
        if (landed) seen = s + 1;
        else gave_up[s & 1] = 1;
        const unsigned char* rec = ring + size_t(stage) * ILU_STAGE;
        const int4 h = *reinterpret_cast<const int4*>(rec);
        if (landed && i < h.x) {
            const int W = h.y, up = h.z, cp = (h.x + 7) & ~7;
            const double* v = reinterpret_cast<const double*>(rec + 16) + i;
            const CI* rows = reinterpret_cast<const CI*>(rec + 16 + size_t(W + up) * cp * sizeof(double)) + i;
            const CI* c = rows + cp;
            const int row = int(*rows);
            double acc = SZ ? zs[row] : z[row];
            switch (min(W, ILU_AHEAD)) {
            case 0: break;
            case 1: acc = ilu_row<1>(acc, v, c, cp, value); break;
            case 2: acc = ilu_row<2>(acc, v, c, cp, value); break;
            case 3: acc = ilu_row<3>(acc, v, c, cp, value); break;
            case 4: acc = ilu_row<4>(acc, v, c, cp, value); break;
            case 5: acc = ilu_row<5>(acc, v, c, cp, value); break;
            case 6: acc = ilu_row<6>(acc, v, c, cp, value); break;
            case 7: acc = ilu_row<7>(acc, v, c, cp, value); break;
            default: acc = ilu_row<8>(acc, v, c, cp, value); break;
            }
            for (int k = ILU_AHEAD; k < W; ++k) acc -= v[k * cp] * value(int(c[k * cp]));
            if (up) acc = v[W * cp] * acc;
            if (SZ) zs[row] = acc;
            else z[row] = acc;
        }
        __syncthreads();
        if (late) return leave();
        late = gave_up[s & 1];
        if (copier && landed && s + nst < s1) {   // every thread is done with this stage
            issue(next, stage);
            next = s + nst + 1 < s1 ? steps[s + nst + 1] : none;
        }
        if (++stage == nst) {
            stage = 0;
            parity ^= 1u;
        }
    }
    if (late) return leave();
    if (SZ)
        for (int k = i; k < n; k += ILU_TB) z[k] = zs[k];
}

__global__ void k_ilu_lower_level(int nrows, const int* __restrict__ rows, const int* __restrict__ sp,
                                  const int* __restrict__ col, const int* __restrict__ diag,
                                  const double* __restrict__ lu, const double* __restrict__ r, double* __restrict__ z,
                                  const int* stop)
{
    chain_wait();
    if (*stop) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nrows) return;
    const int i = rows[q];
    double v = r[i];
    const int d = diag[i];
    for (int k = sp[i >> 5] + (i & 31); k < d; k += 32) v -= lu[k] * z[col[k]];
    z[i] = v;
}

__global__ void k_ilu_upper_level(int nrows, const int* __restrict__ rows, const int* __restrict__ sp,
                                  const int* __restrict__ col, const int* __restrict__ rowlen,
                                  const int* __restrict__ diag, const double* __restrict__ lu, double* __restrict__ z,
                                  const int* stop)
{
    chain_wait();
    if (*stop) return;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nrows) return;
    const int i = rows[q];
    const int d = diag[i];
    const int end = sp[i >> 5] + rowlen[i] * 32 + (i & 31);
    double v = z[i];
    for (int k = d + 32; k < end; k += 32) v -= lu[k] * z[col[k]];
    z[i] = lu[d] * v;
}

}  // namespace

// ----------------------------------------------------------------------------
void RedScratch::ensure(int blocks, cudaStream_t s)
{
    if (blocks <= max_blocks) return;
    partial.alloc(blocks);
    counter.alloc(1);
    counter.zero(s);
    max_blocks = blocks;
}

template <class TV, class TX>
void spmv(cudaStream_t s, const SellPattern& P, const TV* val, const TX* x, TX* y)
{
    if (P.n == 0) return;
    PORSOL_LAUNCH(k_spmv<TV, TX><<<div_up(P.n, RB), RB, 0, s>>>(P.n, P.slice_ptr.p, P.col.p, val, x, y));
    PORSOL_CUDA(cudaGetLastError());
}

template <class TV, class TX>
void residual(cudaStream_t s, const SellPattern& P, const TV* val, const TX* x, const TX* b, TX* y)
{
    if (P.n == 0) return;
    PORSOL_LAUNCH(k_residual<TV, TX><<<div_up(P.n, RB), RB, 0, s>>>(P.n, P.slice_ptr.p, P.col.p, val, x, b, y));
    PORSOL_CUDA(cudaGetLastError());
}

template void spmv<double, double>(cudaStream_t, const SellPattern&, const double*, const double*, double*);
template void spmv<float, float>(cudaStream_t, const SellPattern&, const float*, const float*, float*);
template void residual<double, double>(cudaStream_t, const SellPattern&, const double*, const double*,
                                       const double*, double*);
template void residual<float, float>(cudaStream_t, const SellPattern&, const float*, const float*, const float*,
                                     float*);

template <class TV, class T>
void PcgSolver<TV, T>::setup(int n, cudaStream_t s)
{
    if (n == n_ && hview_) return;
    n_ = n;
    r_.alloc(n);
    z_.alloc(n);
    p_.alloc(n);
    q_.alloc(n);
    st_.alloc(1);
    const int nr = red_shape(n).partials();
    red_.ensure(nr, s);
    pq_.alloc(nr);
    zr_.alloc(nr);
    if (!hview_) {
        PORSOL_CUDA(cudaHostAlloc((void**)&hview_, sizeof(CgHostView), cudaHostAllocMapped));
        PORSOL_CUDA(cudaHostGetDevicePointer((void**)&dview_, hview_, 0));
    }
    if (ev_.empty()) {
        ev_.resize(4);
        for (auto& e : ev_) PORSOL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
}

template <class TV, class T>
PcgSolver<TV, T>::~PcgSolver()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (hview_) cudaFreeHost(hview_);
    for (auto& e : ev_) cudaEventDestroy(e);
}

template <class TV, class T>
void PcgSolver<TV, T>::iteration(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, T* x,
                                 Profiler* prof, int prof_kernel)
{
    const int n = P.n;
    const auto [nr, tb] = red_shape(n);
    const int* stop = &st_.p->stop;
    const double spmv_bytes = double(P.nent) * (sizeof(TV) + (P.has_off16() ? 2 : 4)) + 2.0 * n * sizeof(T);
    {
        const bool pf = prof && prof->on && prof_kernel >= 0;
        cudaEvent_t ev = nullptr;
        if (pf) prof->begin(s, prof_kernel, spmv_bytes, &ev);
        if (P.has_off16())
            chain(k_spmv_pq<TV, T, short>, nr, tb, 0, s, n, P.slice_ptr.p, P.off16.p, val, p_.p, q_.p, st_.p, pq_.p);
        else
            chain(k_spmv_pq<TV, T, int>, nr, tb, 0, s, n, P.slice_ptr.p, P.col.p, val, p_.p, q_.p, st_.p, pq_.p);
        if (pf) prof->end(s, prof_kernel, spmv_bytes, ev);
    }
    const typename Precond<T>::Start start = M.start();
    chain(k_cg_update<T>, nr, tb, 0, s, n, x, r_.p, p_.p, q_.p, st_.p, pq_.p, start, red_.partial.p, red_.counter.p,
          dview_);
    if (start.dinv) M.apply_started(s, r_.p, z_.p, stop);
    else M.apply(s, r_.p, z_.p, stop);
    chain(k_dot_zr<T>, nr, tb, 0, s, n, z_.p, r_.p, st_.p, zr_.p);
    chain(k_cg_direction<T>, nr, tb, 0, s, n, z_.p, p_.p, st_.p, zr_.p, 0);
}

template <class TV, class T>
CgResult PcgSolver<TV, T>::solve(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, const T* b,
                                 T* x, double tol, int maxit, Profiler* prof, int prof_kernel)
{
    const int n = P.n;
    ChainPause plain(prof && prof->on);   // events between the kernels time each one
    CgResult res;
    if (n == 0) {
        res.converged = true;
        return res;
    }
    setup(n, s);
    M.set_block_state(nullptr);   // one system: every row works
    const auto [nr, tb] = red_shape(n);
    CgDev init{};
    init.tol = tol;
    init.maxit = maxit;
    PORSOL_CUDA(cudaMemcpyAsync(st_.p, &init, sizeof(CgDev), cudaMemcpyHostToDevice, s));
    if (P.has_off16())
        chain(k_cg_init<TV, T, short>, nr, tb, 0, s, n, P.slice_ptr.p, P.off16.p, val, x, b, r_.p, st_.p,
            red_.partial.p, red_.counter.p, dview_);
    else
        chain(k_cg_init<TV, T, int>, nr, tb, 0, s, n, P.slice_ptr.p, P.col.p, val, x, b, r_.p, st_.p, red_.partial.p,
            red_.counter.p, dview_);
    PORSOL_CUDA(cudaGetLastError());
    const int* stop = &st_.p->stop;
    M.apply(s, r_.p, z_.p, stop);
    chain(k_dot_zr<T>, nr, tb, 0, s, n, z_.p, r_.p, st_.p, zr_.p);
    chain(k_cg_direction<T>, nr, tb, 0, s, n, z_.p, p_.p, st_.p, zr_.p, 1);
    PORSOL_CUDA(cudaGetLastError());
    // One iteration is captured into a CUDA graph (re-captured when the matrix, vectors or
    // preconditioner change) unless per-kernel profiling is on.
    const bool graphs = use_graphs_ && !(prof && prof->on);
    if (graphs) {
        const void* key[5] = {&P, val, x, (const void*)&M, nullptr};
        bool same = exec_ && key_gen_ == M.generation();
        for (int k = 0; k < 4 && same; ++k) same = key_[k] == key[k];
        if (!same) {
            if (exec_) {
                cudaGraphExecDestroy(exec_);
                exec_ = nullptr;
            }
            cudaGraph_t g;
            const long long l0 = g_launches.load();
            PORSOL_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            iteration(s, P, val, M, x, nullptr, -1);
            PORSOL_CUDA(cudaStreamEndCapture(s, &g));
            nodes_ = g_launches.load() - l0;   // captured, not run: counted at each replay
            g_launches.fetch_sub(nodes_);
            PORSOL_CUDA(cudaGraphInstantiate(&exec_, g, 0));
            PORSOL_CUDA(cudaGraphDestroy(g));
            for (int k = 0; k < 4; ++k) key_[k] = key[k];
            key_gen_ = M.generation();
        }
    }
    // Iterations are queued ahead; the host waits on the event of iteration i - LOOKAHEAD
    // and reads the mapped stop flag.  Iterations queued after convergence are no-ops.
    const int LOOKAHEAD = 2;
    int it = 0;
    bool done = false;
    while (!done) {
        if (it < maxit) {
            if (graphs) {
                PORSOL_CUDA(cudaGraphLaunch(exec_, s));
                g_launches.fetch_add(nodes_);
            } else {
                iteration(s, P, val, M, x, prof, prof_kernel);
            }
            PORSOL_CUDA(cudaGetLastError());
            PORSOL_CUDA(cudaEventRecord(ev_[it % ev_.size()], s));
            ++it;
        }
        if (it >= LOOKAHEAD || it >= maxit) {
            const int wait_it = (it >= maxit) ? it - 1 : it - LOOKAHEAD;
            PORSOL_CUDA(cudaEventSynchronize(ev_[wait_it % ev_.size()]));
            if (hview_->stop || it >= maxit) {
                if (it >= maxit) PORSOL_CUDA(cudaStreamSynchronize(s));
                done = hview_->stop || it >= maxit;
            }
        }
    }
    PORSOL_CUDA(cudaStreamSynchronize(s));
    res.iterations = hview_->iter;
    res.def0 = hview_->def0;
    res.def = hview_->def;
    res.converged = hview_->converged != 0;
    res.breakdown = hview_->breakdown != 0;
    res.reduction = res.def0 > 0 ? res.def / res.def0 : 0.0;
    return res;
}

template class PcgSolver<double, double>;

// ---------------- ReliableCg host side ----------------
void ReliableCg::setup(int n, cudaStream_t s)
{
    if (n != n_) {
        r_.alloc(n);
        z_.alloc(n);
        p_.alloc(n);
        q_.alloc(n);
        r64_.alloc(n);
        n_ = n;
    }
    st_.alloc(1);
    const int nr = red_shape(n).partials();
    red_.ensure(nr, s);
    for (DBuf<double>* v : {&pq_, &pr_, &rr_, &zr_}) v->alloc(nr);
    if (!hview_) {
        PORSOL_CUDA(cudaHostAlloc((void**)&hview_, sizeof(CgHostView), cudaHostAllocMapped));
        PORSOL_CUDA(cudaHostGetDevicePointer((void**)&dview_, hview_, 0));
    }
    if (ev_.empty()) {
        ev_.resize(4);
        for (auto& e : ev_) PORSOL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
}

ReliableCg::~ReliableCg()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (hview_) cudaFreeHost(hview_);
    for (auto& e : ev_) cudaEventDestroy(e);
}

void ReliableCg::iteration(cudaStream_t s, const SellPattern& P, const double* val64, const float* val32,
                           Precond<float>& M, const double* b, double* x, Profiler* prof)
{
    const int n = P.n;
    const auto [nr, tb] = red_shape(n);
    const int* stop = &st_.p->stop;
    {
        const bool pf = prof && prof->on;
        const double bytes = double(P.nent) * (P.has_off16() ? 6.0 : 8.0) + 2.0 * n * 4.0;
        cudaEvent_t ev = nullptr;
        if (pf) prof->begin(s, PK_SPMV32, bytes, &ev);
        if (P.has_off16())
            chain(k_rc_pq<short>, nr, tb, 0, s, n, P.slice_ptr.p, P.off16.p, val32, p_.p, r_.p, q_.p, st_.p, pq_.p,
                pr_.p);
        else
            chain(k_rc_pq<int>, nr, tb, 0, s, n, P.slice_ptr.p, P.col.p, val32, p_.p, r_.p, q_.p, st_.p, pq_.p,
                pr_.p);
        if (pf) prof->end(s, PK_SPMV32, bytes, ev);
    }
    const Precond<float>::Start start = M.start();
    chain(k_rc_update, nr, tb, 0, s, n, x, r_.p, p_.p, q_.p, st_.p, pq_.p, pr_.p, start, rr_.p);
    if (P.has_off16())
        chain(k_rc_true<short>, nr, tb, 0, s, n, P.slice_ptr.p, P.off16.p, val64, x, b, r64_.p, st_.p, rr_.p,
              red_.partial.p, red_.counter.p, dview_);
    else
        chain(k_rc_true<int>, nr, tb, 0, s, n, P.slice_ptr.p, P.col.p, val64, x, b, r64_.p, st_.p, rr_.p,
              red_.partial.p, red_.counter.p, dview_);
    chain(k_rc_rescale, nr, tb, 0, s, n, r64_.p, r_.p, p_.p, st_.p, start, 0, dview_);
    if (start.dinv) M.apply_started(s, r_.p, z_.p, stop);
    else M.apply(s, r_.p, z_.p, stop);
    chain(k_rc_zr, nr, tb, 0, s, n, z_.p, r_.p, q_.p, st_.p, zr_.p, 0);
    chain(k_rc_direction, nr, tb, 0, s, n, z_.p, p_.p, st_.p, zr_.p, 0);
}

CgResult ReliableCg::solve(cudaStream_t s, const SellPattern& P, const double* val64, const float* val32,
                           Precond<float>& M, const double* b, double* x, double tol, int maxit, double delta,
                           Profiler* prof)
{
    const int n = P.n;
    ChainPause plain(prof && prof->on);   // events between the kernels time each one
    CgResult res;
    if (n == 0) {
        res.converged = true;
        return res;
    }
    setup(n, s);
    M.set_block_state(nullptr);   // one system: every row works
    const auto [nr, tb] = red_shape(n);
    RcDev init{};
    init.tol = tol;
    init.maxit = maxit;
    init.delta = delta;
    PORSOL_CUDA(cudaMemcpyAsync(st_.p, &init, sizeof(RcDev), cudaMemcpyHostToDevice, s));
    if (P.has_off16())
        chain(k_rc_init<short>, nr, tb, 0, s, n, P.slice_ptr.p, P.off16.p, val64, x, b, r64_.p, st_.p, red_.partial.p,
            red_.counter.p, dview_);
    else
        chain(k_rc_init<int>, nr, tb, 0, s, n, P.slice_ptr.p, P.col.p, val64, x, b, r64_.p, st_.p, red_.partial.p,
            red_.counter.p, dview_);
    const Precond<float>::Start start = M.start();
    chain(k_rc_rescale, nr, tb, 0, s, n, r64_.p, r_.p, p_.p, st_.p, start, 1, dview_);
    const int* stop = &st_.p->stop;
    if (start.dinv) M.apply_started(s, r_.p, z_.p, stop);
    else M.apply(s, r_.p, z_.p, stop);
    chain(k_rc_zr, nr, tb, 0, s, n, z_.p, r_.p, q_.p, st_.p, zr_.p, 1);
    chain(k_rc_direction, nr, tb, 0, s, n, z_.p, p_.p, st_.p, zr_.p, 1);
    PORSOL_CUDA(cudaGetLastError());
    // per-kernel event timing records events inside the V-cycle: no graph capture then
    const bool graphs = !(prof && prof->on);
    const void* key[5] = {&P, val64, val32, (const void*)&M, x};
    bool same = exec_ && key_gen_ == M.generation() && key_[4] == (const void*)b;
    for (int k = 0; k < 4 && same; ++k) same = key_[k] == key[k];
    if (graphs && !same) {
        if (exec_) {
            cudaGraphExecDestroy(exec_);
            exec_ = nullptr;
        }
        cudaGraph_t g;
        const long long l0 = g_launches.load();
        PORSOL_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        iteration(s, P, val64, val32, M, b, x, nullptr);
        PORSOL_CUDA(cudaStreamEndCapture(s, &g));
        nodes_ = g_launches.load() - l0;
        g_launches.fetch_sub(nodes_);
        PORSOL_CUDA(cudaGraphInstantiate(&exec_, g, 0));
        PORSOL_CUDA(cudaGraphDestroy(g));
        for (int k = 0; k < 4; ++k) key_[k] = key[k];
        key_[4] = b;
        key_gen_ = M.generation();
    }
    const int LOOKAHEAD = 2;
    int it = 0;
    bool done = false;
    while (!done) {
        if (it < maxit) {
            if (graphs) {
                PORSOL_CUDA(cudaGraphLaunch(exec_, s));
                g_launches.fetch_add(nodes_);
            } else {
                iteration(s, P, val64, val32, M, b, x, prof);
            }
            PORSOL_CUDA(cudaEventRecord(ev_[it % ev_.size()], s));
            ++it;
        }
        if (it >= LOOKAHEAD || it >= maxit) {
            const int wait_it = (it >= maxit) ? it - 1 : it - LOOKAHEAD;
            PORSOL_CUDA(cudaEventSynchronize(ev_[wait_it % ev_.size()]));
            if (hview_->stop || it >= maxit) {
                if (it >= maxit) PORSOL_CUDA(cudaStreamSynchronize(s));
                done = hview_->stop || it >= maxit;
            }
        }
    }
    RcDev fin{};
    PORSOL_CUDA(cudaMemcpyAsync(&fin, st_.p, sizeof(RcDev), cudaMemcpyDeviceToHost, s));
    PORSOL_CUDA(cudaStreamSynchronize(s));
    nrep_ = fin.nrep;
    guarded_ = fin.guard != 0;
    res.iterations = fin.iter;
    res.def0 = fin.def0;
    res.def = fin.true_def;
    res.converged = fin.converged != 0;
    res.breakdown = fin.breakdown != 0;
    res.reduction = fin.def0 > 0 ? fin.true_def / fin.def0 : 0.0;
    return res;
}

namespace {
// z = D^-1 r, zero in the applications [skip, skip + skips) (counted on the device, so in graphs too)
__global__ void k_test_precond(int n, const float* __restrict__ dinv, const float* __restrict__ r,
                               float* __restrict__ z, const int* __restrict__ count, int skip, int skips,
                               const int* stop)
{
    if (*stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool zero = *count >= skip && *count < skip + skips;
    if (i < n) z[i] = zero ? 0.0f : dinv[i] * r[i];
}
__global__ void k_test_count(int* count, const int* stop)
{
    if (!*stop) ++*count;
}
struct TestPrecond : Precond<float> {
    int n = 0, skip = 0, skips = 0;
    DBuf<float> dinv;
    DBuf<int> count;
    void apply(cudaStream_t s, const float* r, float* z, const int* stop) override
    {
        PORSOL_LAUNCH(k_test_precond<<<div_up(n, RB), RB, 0, s>>>(n, dinv.p, r, z, count.p, skip, skips, stop));
        PORSOL_LAUNCH(k_test_count<<<1, 1, 0, s>>>(count.p, stop));
    }
};
}  // namespace

int mixed_cg_selftest(int n, const int* ptr, const int* col, const double* val, const double* b, double* x, double tol,
                      int maxit, double delta, int skip, int skips, int* iterations, int* guarded)
{
    struct Stream {   // the default stream cannot be captured
        cudaStream_t s = nullptr;
        Stream() { PORSOL_CUDA(cudaStreamCreate(&s)); }
        ~Stream() { cudaStreamDestroy(s); }
    } own;
    const cudaStream_t s = own.s;
    SellPattern P;
    HVec<int> slot;
    build_sell(n, HVec<int>(ptr, ptr + n + 1), HVec<int>(col, col + ptr[n]), P, &slot);
    P.upload(s);
    std::vector<double> v(size_t(P.nent), 0.0);
    std::vector<float> v32(v.size(), 0.0f), d(n, 0.0f);
    for (int i = 0; i < n; ++i)
        for (int k = ptr[i]; k < ptr[i + 1]; ++k) {
            v[size_t(slot[size_t(k)])] = val[k];
            v32[size_t(slot[size_t(k)])] = float(val[k]);
            if (col[k] == i) d[size_t(i)] = float(1.0 / val[k]);
        }
    DBuf<double> a, bd, xd;
    DBuf<float> a32;
    a.upload(v, s);
    a32.upload(v32, s);
    bd.upload(b, n, s);
    xd.alloc(n);
    xd.zero(s);
    TestPrecond M;
    M.n = n;
    M.skip = skip;
    M.skips = skips;
    M.dinv.upload(d, s);
    M.count.alloc(1);
    M.count.zero(s);
    ReliableCg cg;
    const CgResult r = cg.solve(s, P, a.p, a32.p, M, bd.p, xd.p, tol, maxit, delta);
    xd.download(x, n, s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
    *iterations = r.iterations;
    *guarded = cg.guarded() ? 1 : 0;
    if (r.breakdown) throw Error(PORSOL_ERR_NONFINITE, "CG breakdown");
    if (!r.converged) throw Error(PORSOL_ERR_NOT_CONVERGED, "not converged");
    return 0;
}

// ---------------- ILU(0) host side ----------------
void Ilu0::build_levels(const SellPattern& P, cudaStream_t s, bool shared)
{
    P_ = &P;
    const int n = P.n;
    auto slot = [&](int r, int t) { return (long long)P.h_slice_ptr[r / SELL_C] + (long long)t * SELL_C + r % SELL_C; };
    std::vector<int> lev(n, 0);
    int nl = 0;
    for (int i = 0; i < n; ++i) {
        int l = 0;
        for (int t = 0; t < P.h_rowlen[i]; ++t) {
            const int j = P.h_col[slot(i, t)];
            if (j < i) l = std::max(l, lev[j] + 1);
        }
        lev[i] = l;
        nl = std::max(nl, l + 1);
    }
    auto bucket = [&](const std::vector<int>& lv, int nlev, std::vector<int>& ptr, std::vector<int>& rows, bool rev) {
        ptr.assign(nlev + 1, 0);
        for (int i = 0; i < n; ++i) ptr[lv[i] + 1]++;
        for (int l = 0; l < nlev; ++l) ptr[l + 1] += ptr[l];
        rows.assign(n, 0);
        std::vector<int> f(ptr.begin(), ptr.end() - 1);
        if (!rev)
            for (int i = 0; i < n; ++i) rows[f[lv[i]]++] = i;
        else
            for (int i = n - 1; i >= 0; --i) rows[f[lv[i]]++] = i;
    };
    std::vector<int> lrows, urows;
    bucket(lev, nl, h_lptr_, lrows, false);
    std::vector<int> ulev(n, 0);
    int nu = 0;
    for (int i = n - 1; i >= 0; --i) {
        int l = 0;
        for (int t = 0; t < P.h_rowlen[i]; ++t) {
            const int j = P.h_col[slot(i, t)];
            if (j > i) l = std::max(l, ulev[j] + 1);
        }
        ulev[i] = l;
        nu = std::max(nu, l + 1);
    }
    bucket(ulev, nu, h_uptr_, urows, true);
    lrows_.upload(lrows, s);
    urows_.upload(urows, s);
    // two cells of at most 12 faces share a face: 23 entries at most
    for (int i = 0; i < n; ++i) PORSOL_REQUIRE(P.h_rowlen[i] <= 32, PORSOL_ERR_BAD_ARG, "ILU0: row too long");
    // The fused sweep: step records of at most ILU_ROWS rows of one level and ILU_STAGE bytes.  The vector
    // goes to shared memory (16-bit row and column numbers) when all levels can be fused and it fits beside
    // two stages.
    bool all = true;
    for (const std::vector<int>* ptr : {&h_lptr_, &h_uptr_})
        for (size_t l = 0; l + 1 < ptr->size(); ++l) all = all && (*ptr)[l + 1] - (*ptr)[l] <= SHARED_ROWS;
    const size_t zbytes = (size_t(n) + 1) * sizeof(double);
    shared_z_ = shared && all && n < 65535 && 128 + zbytes + 2 * size_t(ILU_STAGE) <= ILU_SMEM;
    stages_ = shared_z_ ? std::min<int>(ILU_STAGES, int((ILU_SMEM - 128 - zbytes) / ILU_STAGE)) : ILU_STAGES;
    const size_t ib = shared_z_ ? 2 : 4;
    const int fused_rows = shared_z_ ? SHARED_ROWS : FUSE_ROWS;
    std::vector<int2> steps;
    std::vector<unsigned char> blob;
    std::vector<int> pos, from;
    runs_.clear();
    auto bytes_of = [&](int cnt, int w, int up) {
        const size_t cp = size_t(cnt + 7) / 8 * 8;
        return 16 + ((w + up) * sizeof(double) + (w + 1) * ib) * cp;
    };
    auto add = [&](const std::vector<int>& ptr, const std::vector<int>& rows, int up) {
        auto in = [&](int i, int j) { return up ? j > i : j < i; };
        auto length = [&](int i) {
            int m = 0;
            for (int t = 0; t < P.h_rowlen[i]; ++t) m += in(i, P.h_col[slot(i, t)]);
            return m;
        };
        for (int l = 0; l + 1 < int(ptr.size()); ++l) {
            if (ptr[l + 1] - ptr[l] > fused_rows) {
                runs_.push_back({false, l, up});
                continue;
            }
            if (runs_.empty() || !runs_.back().fused) runs_.push_back({true, int(steps.size()), int(steps.size())});
            for (int b = ptr[l]; b < ptr[l + 1];) {
                int cnt = 0, w = 0;
                while (b + cnt < ptr[l + 1] && cnt < ILU_ROWS) {
                    const int w1 = std::max(w, length(rows[b + cnt]));
                    if (cnt > 0 && bytes_of(cnt + 1, w1, up) > ILU_STAGE) break;
                    w = w1;
                    ++cnt;
                }
                const size_t cp = size_t(cnt + 7) / 8 * 8, at = blob.size(), sz = bytes_of(cnt, w, up);
                PORSOL_REQUIRE(sz <= ILU_STAGE && at / 16 < (1u << 31), PORSOL_ERR_BAD_ARG, "ILU0: row too long");
                blob.resize(at + sz, 0);
                const int head[4] = {cnt, w, up, 0};
                std::memcpy(blob.data() + at, head, 16);
                auto number = [&](size_t q, int v) {   // q-th row or column number of the record
                    unsigned char* d = blob.data() + at + 16 + (w + up) * cp * sizeof(double) + q * ib;
                    if (ib == 2) {
                        const unsigned short h = (unsigned short)v;
                        std::memcpy(d, &h, 2);
                    } else {
                        std::memcpy(d, &v, 4);
                    }
                };
                for (size_t q = 0; q < cp; ++q) {
                    const int i = q < size_t(cnt) ? rows[b + q] : n;
                    number(q, i);
                    int m = 0;
                    if (i < n)
                        for (int t = 0; t < P.h_rowlen[i]; ++t) {
                            const int k = int(slot(i, t)), j = P.h_col[k];
                            if (!in(i, j)) continue;
                            number(cp + m * cp + q, j);
                            pos.push_back(int(at / 8 + 2 + m * cp + q));
                            from.push_back(k);
                            ++m;
                        }
                    for (; m < w; ++m) number(cp + m * cp + q, n);
                    if (up && i < n) {
                        pos.push_back(int(at / 8 + 2 + w * cp + q));
                        from.push_back(-1 - i);   // the diagonal's slot
                    }
                }
                steps.push_back(make_int2(int(at / 16), int(sz)));
                runs_.back().b = int(steps.size());
                b += cnt;
            }
        }
    };
    add(h_lptr_, lrows, 0);
    add(h_uptr_, urows, 1);
    for (int& k : from)
        if (k < 0) {
            const int i = -1 - k;
            for (int t = 0; t < P.h_rowlen[i]; ++t)
                if (P.h_col[slot(i, t)] == i) k = int(slot(i, t));
            PORSOL_REQUIRE(k >= 0, PORSOL_ERR_BAD_ARG, "ILU0: missing diagonal");
        }
    steps_.upload(steps, s);
    blob_.upload(blob, s);
    pos_.upload(pos, s);
    from_.upload(from, s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
}

void Ilu0::factor(cudaStream_t s, const SellPattern& P, const double* val)
{
    bump_generation();
    lu_.alloc(P.nent);
    PORSOL_CUDA(cudaMemcpyAsync(lu_.p, val, P.nent * sizeof(double), cudaMemcpyDeviceToDevice, s));
    status_.alloc(1);
    status_.zero(s);
    DBuf<int>& status = status_;
    for (size_t l = 0; l + 1 < h_lptr_.size(); ++l) {
        const int cnt = h_lptr_[l + 1] - h_lptr_[l];
        chain(k_ilu_factor_warp, div_up(cnt, 4), 128, 0, s, cnt, lrows_.p + h_lptr_[l], P.slice_ptr.p, P.col.p,
              P.rowlen.p, P.diag.p, lu_.p, status.p);
    }
    PORSOL_CUDA(cudaGetLastError());
    if (pos_.n)
        PORSOL_LAUNCH(k_ilu_pack<<<div_up((long long)pos_.n, RB), RB, 0, s>>>(int(pos_.n), pos_.p, from_.p, lu_.p,
                                                                             reinterpret_cast<double*>(blob_.p)));
    PORSOL_CUDA(cudaGetLastError());
    int st = 0;
    PORSOL_CUDA(cudaMemcpyAsync(&st, status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    PORSOL_CUDA(cudaStreamSynchronize(s));
    PORSOL_REQUIRE(st == 0, PORSOL_ERR_NONFINITE, "ILU0: zero or non-finite pivot");
}

int Ilu0::solve_status(cudaStream_t s) const
{
    int st = 0;
    PORSOL_CUDA(cudaMemcpyAsync(&st, status_.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    PORSOL_CUDA(cudaStreamSynchronize(s));
    return st;
}

size_t Ilu0::steps_shm() const
{
    return 128 + size_t(stages_) * ILU_STAGE + (shared_z_ ? (size_t(P_->n) + 1) * sizeof(double) : 0);
}

int ilu_sweep_selftest(int thread, bool shared, double* z_host)
{
    const int n = 48;
    HVec<int> ptr(size_t(n) + 1, 0), col, slot;
    std::vector<double> a, r(n);
    for (int i = 0; i < n; ++i) {
        for (int j = std::max(0, i - 1); j <= std::min(n - 1, i + 1); ++j) {
            col.push_back(j);
            a.push_back(j == i ? 2.5 : -1.0);
        }
        ptr[size_t(i) + 1] = int(col.size());
        r[size_t(i)] = 1.0 + i / 8.0;
    }
    cudaStream_t s = nullptr;
    SellPattern P;
    build_sell(n, ptr, col, P, &slot);
    P.upload(s);
    std::vector<double> v(size_t(P.nent), 0.0);
    for (size_t k = 0; k < a.size(); ++k) v[size_t(slot[k])] = a[k];
    DBuf<double> val, rd, zd;
    DBuf<int> stop;
    val.upload(v, s);
    rd.upload(r, s);
    zd.alloc(n);
    stop.alloc(1);
    stop.zero(s);
    Ilu0 ilu;
    ilu.build_levels(P, s, shared);
    ilu.factor(s, P, val.p);
    if (thread < 0) {
        ilu.apply(s, rd.p, zd.p, stop.p);
    } else {
        PORSOL_REQUIRE(thread < ILU_TB && ilu.runs_.size() == 1 && ilu.runs_[0].fused, PORSOL_ERR_BAD_ARG, "ILU0 self-test");
        auto* f = ilu.shared_z_ ? k_ilu_steps<unsigned short, true, true> : k_ilu_steps<int, false, true>;
        PORSOL_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ILU_SMEM)));
        device_copy(s, zd.p, rd.p, n * sizeof(double));
        chain(f, 1, ILU_TB, ilu.steps_shm(), s, ilu.runs_[0].a, ilu.runs_[0].b, ilu.steps_.p, ilu.blob_.p, rd.p,
              zd.p, n, ilu.stages_, stop.p, ilu.status_.p, thread);
    }
    const int st = ilu.solve_status(s);
    zd.download(z_host, n, s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
    return st;
}

void Ilu0::apply(cudaStream_t s, const double* r, double* z, const int* stop)
{
    const SellPattern& P = *P_;
    const size_t zbytes = size_t(P.n) * sizeof(double), shm = steps_shm();
    if (!shared_z_) PORSOL_CUDA(cudaMemcpyAsync(z, r, zbytes, cudaMemcpyDeviceToDevice, s));   // the fused steps start from z
    for (const Run& u : runs_) {
        if (u.fused && shared_z_) {
            PORSOL_CUDA(cudaFuncSetAttribute(k_ilu_steps<unsigned short, true>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(ILU_SMEM)));
            chain(k_ilu_steps<unsigned short, true>, 1, ILU_TB, shm, s, u.a, u.b, steps_.p, blob_.p, r, z, P.n, stages_,
                  stop, status_.p, -1);
        } else if (u.fused) {
            PORSOL_CUDA(cudaFuncSetAttribute(k_ilu_steps<int, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(ILU_SMEM)));
            chain(k_ilu_steps<int, false>, 1, ILU_TB, shm, s, u.a, u.b, steps_.p, blob_.p, r, z, P.n, stages_, stop,
                  status_.p, -1);
        } else if (u.b == 0) {
            const int b = h_lptr_[u.a], cnt = h_lptr_[u.a + 1] - b;
            chain(k_ilu_lower_level, div_up(cnt, 128), 128, 0, s, cnt, lrows_.p + b, P.slice_ptr.p, P.col.p, P.diag.p,
                  lu_.p, r, z, stop);
        } else {
            const int b = h_uptr_[u.a], cnt = h_uptr_[u.a + 1] - b;
            chain(k_ilu_upper_level, div_up(cnt, 128), 128, 0, s, cnt, urows_.p + b, P.slice_ptr.p, P.col.p, P.rowlen.p,
                  P.diag.p, lu_.p, z, stop);
        }
    }
    PORSOL_CUDA(cudaGetLastError());
}

// ---------------- helpers ----------------
void device_copy(cudaStream_t s, void* dst, const void* src, size_t bytes)
{
    if (bytes) PORSOL_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s));
}

template <class TA, class TB>
void convert(cudaStream_t s, long long n, const TA* a, TB* b)
{
    if (n == 0) return;
    PORSOL_LAUNCH(k_convert<TA, TB><<<div_up(n, RB), RB, 0, s>>>(n, a, b));
    PORSOL_CUDA(cudaGetLastError());
}
template void convert<double, float>(cudaStream_t, long long, const double*, float*);
template void convert<float, double>(cudaStream_t, long long, const float*, double*);

void axpy_add(cudaStream_t s, int n, const double* y, double* x)
{
    if (n == 0) return;
    PORSOL_LAUNCH(k_axpy_add<<<div_up(n, RB), RB, 0, s>>>(n, y, x));
    PORSOL_CUDA(cudaGetLastError());
}


void dirichlet_guess(cudaStream_t s, const SellPattern& P, const double* val, const double* b, double* x)
{
    if (P.n == 0) return;
    PORSOL_LAUNCH(k_dirichlet_guess<<<div_up(P.n, RB), RB, 0, s>>>(P.n, P.slice_ptr.p, P.col.p, P.rowlen.p, val, b, x));
    PORSOL_CUDA(cudaGetLastError());
}

template <class T>
double norm2(cudaStream_t s, int n, const T* x, RedScratch& red)
{
    if (n == 0) return 0.0;
    const RedShape sh = red_shape(n);
    const int nb = sh.partials();
    red.ensure(nb + 1, s);
    PORSOL_LAUNCH(k_norm2<T><<<sh.blocks, sh.threads, 0, s>>>(n, x, red.partial.p, red.counter.p, red.partial.p + nb));
    PORSOL_CUDA(cudaGetLastError());
    double out = 0.0;
    PORSOL_CUDA(cudaMemcpyAsync(&out, red.partial.p + nb, sizeof(double), cudaMemcpyDeviceToHost, s));
    PORSOL_CUDA(cudaStreamSynchronize(s));
    return std::sqrt(out);
}
template double norm2<double>(cudaStream_t, int, const double*, RedScratch&);
template double norm2<float>(cudaStream_t, int, const float*, RedScratch&);

}  // namespace porsol
