// k_batch.cu -- one preconditioned CG per block of a block-diagonal system: BatchedCg3 for the three
// directions of an upscaling batch at once (AMG), BatchedPcg for one right-hand side (ILU0).
//
// BatchedPcg, per iteration (captured into one CUDA graph): q = A p; per block pq_g and lambda_g =
// rholast_g / pq_g; x += lambda p, r -= lambda q; per block ||r_g|| and the stopping test;
// z = M r; per block rho_g = z_g . r_g and beta_g; p = z + beta p.  Block sums are computed by
// one CTA per block over the block's two unknown ranges in a fixed order, so results are
// reproducible.  The CTA of the last block to finish the residual norms counts the active
// blocks and raises the stop flag (device word read by every kernel, mirrored in mapped host
// memory for the host loop).  A block that meets its tolerance, or whose curvature p.Ap is not
// positive, is frozen (lambda = 0).
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "batch.h"
#include "sell.cuh"

namespace porsol {

namespace {

constexpr int BT = 256;

template <class V>
__device__ __forceinline__ V warp_sum(V v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Threads of the per-block CTAs (one CTA per block sums the block's ranges): a block holds up to
// about 10^5 unknowns, and its CTA alone sets the time of the launch.
constexpr int RT = 1024;

// Sum of a_i * b_i over block g's two ranges in a fixed order; the total is returned in thread 0.
// Thread t keeps four running sums over the elements t + RT (4m + u), u = 0..3, of each range, so
// eight loads are in flight per thread (one running sum put one memory latency on every RT
// elements: 115 us for a 98 k-unknown block).
template <class T>
__device__ double seg_dot(const int* __restrict__ rg, int g, const T* __restrict__ a, const T* __restrict__ b)
{
    __shared__ double ws[RT / 32];
    T v0 = T(0), v1 = T(0), v2 = T(0), v3 = T(0);
    for (int part = 0; part < 2; ++part) {
        const int hi = rg[4 * g + 2 * part + 1];
        int i = rg[4 * g + 2 * part] + threadIdx.x;
        for (; i + 3 * RT < hi; i += 4 * RT) {
            const T a0 = a[i], a1 = a[i + RT], a2 = a[i + 2 * RT], a3 = a[i + 3 * RT];
            const T b0 = b[i], b1 = b[i + RT], b2 = b[i + 2 * RT], b3 = b[i + 3 * RT];
            v0 += a0 * b0;
            v1 += a1 * b1;
            v2 += a2 * b2;
            v3 += a3 * b3;
        }
        for (; i < hi; i += RT) v0 += a[i] * b[i];
    }
    const double w = double(warp_sum<T>((v0 + v1) + (v2 + v3)));
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = w;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < RT / 32; ++k) t += ws[k];
    return t;
}

__device__ __forceinline__ void publish(BatchDev* st, BatchHostView* hv)
{
    hv->iter = st->iter;
    hv->active = st->active;
    hv->breakdown = st->breakdown;
    hv->stop = st->stop;
    __threadfence_system();
}

// After every block has written conv: the last CTA to arrive counts active blocks, updates
// the iteration count and the stop flag.
__device__ void finish_round(int nblk, const int* conv, BatchDev* st, unsigned int* counter, BatchHostView* hv,
                             bool count_iteration)
{
    __shared__ bool last;
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == unsigned(nblk - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int act = 0, brk = 0;
    for (int g = threadIdx.x; g < nblk; g += RT) {
        const int c = ((volatile const int*)conv)[g];
        act += c == 0;
        brk |= c == 2;
    }
    __shared__ int sa[RT / 32], sb[RT / 32];
    const int wa = warp_sum<int>(act), wb = __any_sync(0xffffffffu, brk);
    if ((threadIdx.x & 31) == 0) {
        sa[threadIdx.x >> 5] = wa;
        sb[threadIdx.x >> 5] = wb;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int A = 0, Bk = 0;
        for (int k = 0; k < RT / 32; ++k) {
            A += sa[k];
            Bk |= sb[k];
        }
        if (count_iteration) st->iter += 1;
        st->active = A;
        st->breakdown = Bk;
        st->stop = (A == 0) || st->iter >= st->maxit;
        *counter = 0u;
        publish(st, hv);
    }
}

template <class T>
__global__ void __launch_bounds__(RT) k_b_init(int nblk, const int* __restrict__ rg, const T* __restrict__ r,
                                               double* def0, double* def, int* conv, BatchDev* st,
                                               unsigned int* counter, BatchHostView* hv)
{
    const int g = blockIdx.x;
    const double s = seg_dot<T>(rg, g, r, r);
    if (threadIdx.x == 0) {
        const double d = sqrt(s);
        def0[g] = d;
        def[g] = d;
        conv[g] = !isfinite(d) ? 2 : (d < 1e-30 ? 1 : 0);
    }
    finish_round(nblk, conv, st, counter, hv, false);
}

template <class T>
__global__ void __launch_bounds__(RT) k_b_pq(const int* __restrict__ rg, const T* __restrict__ p,
                                             const T* __restrict__ q, const double* __restrict__ rholast,
                                             int* conv, double* lambda, const BatchDev* st)
{
    if (st->stop) return;
    const int g = blockIdx.x;
    if (conv[g] != 0) {   // frozen block (every thread reads conv[g] before thread 0 may change it)
        if (threadIdx.x == 0) lambda[g] = 0.0;
        return;
    }
    const double s = seg_dot<T>(rg, g, p, q);
    if (threadIdx.x == 0) {
        double l = 0.0;
        if (conv[g] == 0) {
            if (!(s > 0.0) || !isfinite(s)) conv[g] = 2;
            else l = rholast[g] / s;
        }
        lambda[g] = l;
    }
}

template <class T>
__global__ void k_b_update(int n, const int* __restrict__ blk, const double* __restrict__ lambda, T* __restrict__ x,
                           T* __restrict__ r, const T* __restrict__ p, const T* __restrict__ q, const BatchDev* st)
{
    if (st->stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T l = T(lambda[blk[i]]);
    if (l != T(0)) {
        x[i] += l * p[i];
        r[i] -= l * q[i];
    }
}

template <class T>
__global__ void __launch_bounds__(RT) k_b_rr(int nblk, const int* __restrict__ rg, const T* __restrict__ r,
                                             const double* __restrict__ def0, double* def,
                                             const double* __restrict__ tol, int* conv, BatchDev* st,
                                             unsigned int* counter, BatchHostView* hv)
{
    if (st->stop) return;
    const int g = blockIdx.x;
    const bool live = conv[g] == 0;   // uniform in the CTA: read before thread 0 may change it
    const double s = live ? seg_dot<T>(rg, g, r, r) : 0.0;
    if (threadIdx.x == 0 && live) {
        const double d = sqrt(s);
        def[g] = d;
        if (!isfinite(d)) conv[g] = 2;
        else if (d < tol[g] * def0[g] || d < 1e-30) conv[g] = 1;
    }
    finish_round(nblk, conv, st, counter, hv, true);
}

template <class T>
__global__ void __launch_bounds__(RT) k_b_zr(const int* __restrict__ rg, const T* __restrict__ z,
                                             const T* __restrict__ r, double* rholast, double* beta,
                                             const int* __restrict__ conv, int first, const BatchDev* st)
{
    if (st->stop) return;
    const int g = blockIdx.x;
    if (!first && conv[g] != 0) {   // frozen block: its direction is no longer used
        if (threadIdx.x == 0) beta[g] = 0.0;
        return;
    }
    const double s = seg_dot<T>(rg, g, z, r);
    if (threadIdx.x == 0) {
        const double rl = rholast[g];
        beta[g] = (first || conv[g] != 0 || rl == 0.0) ? 0.0 : s / rl;
        rholast[g] = s;
    }
}

template <class T>
__global__ void k_b_direction(int n, const int* __restrict__ blk, const double* __restrict__ beta,
                              const T* __restrict__ z, T* __restrict__ p, const BatchDev* st)
{
    if (st->stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = z[i] + T(beta[blk[i]]) * p[i];
}

template <class TV, class T>
__global__ void k_b_residual(int n, const int* __restrict__ sp, const int* __restrict__ col,
                             const TV* __restrict__ val, const T* __restrict__ x, const T* __restrict__ b,
                             T* __restrict__ r)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = b[i] - sell_dot<T>(sp, col, val, i, [x](int j) { return x[j]; });
}

template <class TV, class T>
__global__ void k_b_spmv(int n, const int* __restrict__ sp, const int* __restrict__ col, const TV* __restrict__ val,
                         const T* __restrict__ p, T* __restrict__ q, const int* __restrict__ blk,
                         const int* __restrict__ conv, const BatchDev* st)
{
    if (st->stop) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || conv[blk[i]] != 0) return;   // a frozen block's q is not used
    q[i] = sell_dot<T>(sp, col, val, i, [p](int j) { return p[j]; });
}

// ---------------- three right-hand sides at once ----------------
// The vectors of BatchedCg3 are cut into chunks of at most CHUNK unknowns of one block.  A chunk is one
// thread block in every kernel; its partial sums are added in chunk order by each reader, so sums do not
// depend on which blocks run when, and no kernel is spent on finishing them.  (One thread block per
// sub-grid left most SMs idle: 126 us of a 611 us iteration on 48 sub-grids.)
constexpr int CT = 256;

__device__ __forceinline__ V3<double> warp_sum3(V3<double> v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += shfl_xor(v, o);
    return v;
}

// sum over the thread block, in thread 0
__device__ __forceinline__ V3<double> block_sum3(const V3<double>& v0)
{
    __shared__ V3<double> ws[CT / 32];
    const V3<double> v = warp_sum3(v0);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    V3<double> t{};
    if (threadIdx.x == 0)
        for (int k = 0; k < CT / 32; ++k) t += ws[k];
    return t;
}

// sum of the partial sums of block g by one warp, in every lane
__device__ __forceinline__ V3<double> chunk_sum(const int* __restrict__ cptr, int g, const V3<double>* __restrict__ part)
{
    V3<double> t{};
    for (int c = cptr[g] + int(threadIdx.x & 31), e = cptr[g + 1]; c < e; c += 32) t += part[c];
    return warp_sum3(t);
}

// chunk: (first unknown, unknowns, block, -)
__global__ void __launch_bounds__(CT) k_b3_residual(const int4* __restrict__ chunks, const int* __restrict__ sp,
                                                    const int* __restrict__ col, const double* __restrict__ val,
                                                    const V3<double>* __restrict__ x, const V3<double>* __restrict__ b,
                                                    V3<double>* __restrict__ r, V3<double>* __restrict__ part)
{
    const int4 c = chunks[blockIdx.x];
    V3<double> v{};
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) {
        const V3<double> ri = b[i] - sell_dot<V3<double>>(sp, col, val, i, [x](int j) { return x[j]; });
        r[i] = ri;
        v += times(ri, ri);
    }
    v = block_sum3(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// q = A p, p . q
__global__ void __launch_bounds__(CT) k_b3_pq(const int4* __restrict__ chunks, const int* __restrict__ sp,
                                              const int* __restrict__ col, const double* __restrict__ val,
                                              const V3<double>* __restrict__ p, V3<double>* __restrict__ q,
                                              const int* __restrict__ conv, V3<double>* __restrict__ part,
                                              const Batch3Dev* st)
{
    if (st->stop) return;
    const int4 c = chunks[blockIdx.x];
    if (conv[c.z] != 0) return;
    V3<double> v{};
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) {
        const V3<double> qi = sell_dot<V3<double>>(sp, col, val, i, [p](int j) { return p[j]; });
        q[i] = qi;
        v += times(p[i], qi);
    }
    v = block_sum3(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}

__device__ __forceinline__ double step_length(double pq, double rho, int done, int* broken)
{
    if (done != 0) return 0.0;
    if (!(pq > 0.0) || !isfinite(pq)) {
        *broken = 1;
        return 0.0;
    }
    return rho / pq;
}

// lambda = rho / p.q per direction; x += lambda p; r -= lambda q; r . r; the preconditioner's FP32 copy of r
template <class T>
__global__ void __launch_bounds__(CT) k_b3_update(const int4* __restrict__ chunks, const int* __restrict__ cptr,
                                                  const V3<double>* __restrict__ part_pq,
                                                  const double* __restrict__ rho, int nblk,
                                                  const int* __restrict__ done, int* broken,
                                                  const int* __restrict__ conv, V3<double>* __restrict__ x,
                                                  V3<double>* __restrict__ r, const V3<double>* __restrict__ p,
                                                  const V3<double>* __restrict__ q, const V3<double>* __restrict__ scale,
                                                  V3<T>* __restrict__ rt, V3<double>* __restrict__ part,
                                                  const Batch3Dev* st)
{
    if (st->stop) return;
    const int4 c = chunks[blockIdx.x];
    const int g = c.z;
    if (conv[g] != 0) return;
    __shared__ V3<double> sl;
    if (threadIdx.x < 32) {
        const V3<double> s = chunk_sum(cptr, g, part_pq);
        if (threadIdx.x == 0) {
            const double* rh = rho + size_t(st->iter & 1) * 3 * nblk + 3 * g;
            int bad[3] = {0, 0, 0};
            sl.a = step_length(s.a, rh[0], done[3 * g], &bad[0]);
            sl.b = step_length(s.b, rh[1], done[3 * g + 1], &bad[1]);
            sl.c = step_length(s.c, rh[2], done[3 * g + 2], &bad[2]);
            if (cptr[g] == int(blockIdx.x))
                for (int d = 0; d < 3; ++d)
                    if (bad[d]) broken[3 * g + d] = 1;
        }
    }
    __syncthreads();
    const V3<double> l = sl, sc = scale[g];
    const bool la = l.a != 0.0, lb = l.b != 0.0, lc = l.c != 0.0;   // a stopped direction keeps its x and r
    V3<double> v{};
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) {
        const V3<double> pi = p[i], qi = q[i];
        V3<double> xi = x[i], ri = r[i];
        if (la) {
            xi.a += l.a * pi.a;
            ri.a -= l.a * qi.a;
        }
        if (lb) {
            xi.b += l.b * pi.b;
            ri.b -= l.b * qi.b;
        }
        if (lc) {
            xi.c += l.c * pi.c;
            ri.c -= l.c * qi.c;
        }
        x[i] = xi;
        r[i] = ri;
        if (sizeof(T) == 4) rt[i] = from_wide<V3<T>>(times(ri, sc));
        v += times(ri, ri);
    }
    v = block_sum3(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// Residual norms and stopping tests of every block and direction (a warp per block); the last thread block
// to arrive counts what is left.  init: the initial norms and the scales of the FP32 copies.
__global__ void __launch_bounds__(CT) k_b3_test(int nblk, const int* __restrict__ cptr,
                                                const V3<double>* __restrict__ part, double tol, int init,
                                                double* def0, double* def, int* done, const int* __restrict__ broken,
                                                int* conv, V3<double>* scale, V3<double>* iscale, Batch3Dev* st,
                                                unsigned int* counter, Batch3HostView* hv)
{
    if (!init && st->stop) return;
    const int g = blockIdx.x * (CT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (g < nblk && (init || conv[g] == 0)) {
        const V3<double> s = chunk_sum(cptr, g, part);
        if (lane == 0) {
            const double v[3] = {s.a, s.b, s.c};
            double sc[3], isc[3];
            int left = 0;
            for (int d = 0; d < 3; ++d) {
                const int k = 3 * g + d;
                const double n = sqrt(v[d]);
                if (init) {
                    def0[k] = def[k] = n;
                    done[k] = !isfinite(n) ? 2 : (n < 1e-30 ? 1 : 0);
                    const bool ok = n > 1e-300 && isfinite(n);
                    sc[d] = ok ? 1.0 / n : 0.0;
                    isc[d] = ok ? n : 0.0;
                } else if (done[k] == 0) {
                    def[k] = n;
                    if (broken[k] || !isfinite(n)) done[k] = 2;
                    else if (n < tol * def0[k] || n < 1e-30) done[k] = 1;
                }
                left |= done[k] == 0;
            }
            if (init) {
                scale[g] = make_v3<double>(sc[0], sc[1], sc[2]);
                iscale[g] = make_v3<double>(isc[0], isc[1], isc[2]);
            }
            conv[g] = left ? 0 : 1;
        }
    }
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    __shared__ int left[3], brk;
    if (threadIdx.x < 3) left[threadIdx.x] = 0;
    if (threadIdx.x == 0) brk = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < 3 * nblk; k += CT) {
        const int c = ((volatile const int*)done)[k];
        if (c == 0) atomicAdd(&left[k % 3], 1);
        if (c == 2) brk = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!init) {
            st->iter += 1;
            for (int d = 0; d < 3; ++d)   // the iteration in which the direction's last block stopped
                if (st->left[d] > 0) st->iters[d] = st->iter;
        }
        int active = 0;
        for (int d = 0; d < 3; ++d) {
            st->left[d] = left[d];
            active += left[d];
            hv->iters[d] = st->iters[d];
        }
        st->stop = active == 0 || st->iter >= st->maxit;
        *counter = 0u;
        hv->active = active;
        hv->breakdown = brk;
        hv->stop = st->stop;
        __threadfence_system();
    }
}

__global__ void __launch_bounds__(CT) k_b3_cast(const int4* __restrict__ chunks, const V3<double>* __restrict__ r,
                                                const V3<double>* __restrict__ scale, V3<float>* __restrict__ rt)
{
    const int4 c = chunks[blockIdx.x];
    const V3<double> sc = scale[c.z];
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) rt[i] = from_wide<V3<float>>(times(r[i], sc));
}

// the preconditioned residual in FP64
template <class T>
__device__ __forceinline__ V3<double> widened(const V3<T>& z, const V3<double>& iscale)
{
    if constexpr (sizeof(T) == 4) return times(to_wide(z), iscale);
    else return z;
}

// z . r
template <class T>
__global__ void __launch_bounds__(CT) k_b3_zr(const int4* __restrict__ chunks, const V3<T>* __restrict__ z,
                                              const V3<double>* __restrict__ r, const V3<double>* __restrict__ iscale,
                                              const int* __restrict__ conv, V3<double>* __restrict__ part,
                                              const Batch3Dev* st)
{
    if (st->stop) return;
    const int4 c = chunks[blockIdx.x];
    if (conv[c.z] != 0) return;
    const V3<double> sc = iscale[c.z];
    V3<double> v{};
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) v += times(widened(z[i], sc), r[i]);
    v = block_sum3(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// beta = rho / last rho per direction (0 at the start); p = z + beta p.  rho alternates between two
// slots: other thread blocks of the block still read the last one.
template <class T>
__global__ void __launch_bounds__(CT) k_b3_direction(const int4* __restrict__ chunks, const int* __restrict__ cptr,
                                                     const V3<double>* __restrict__ part, double* rho, int nblk,
                                                     const int* __restrict__ done, const int* __restrict__ conv,
                                                     const V3<T>* __restrict__ z, const V3<double>* __restrict__ iscale,
                                                     V3<double>* __restrict__ p, int first, const Batch3Dev* st)
{
    if (st->stop) return;
    const int4 c = chunks[blockIdx.x];
    const int g = c.z;
    if (conv[g] != 0) return;
    __shared__ double sb[3];
    if (threadIdx.x < 32) {
        const V3<double> s = chunk_sum(cptr, g, part);
        if (threadIdx.x == 0) {
            const int it = st->iter;
            const double* last = rho + size_t((it + 1) & 1) * 3 * nblk + 3 * g;
            double* now = rho + size_t(it & 1) * 3 * nblk + 3 * g;
            const double v[3] = {s.a, s.b, s.c};
            for (int d = 0; d < 3; ++d) {
                sb[d] = (first || done[3 * g + d] != 0 || last[d] == 0.0) ? 0.0 : v[d] / last[d];
                if (cptr[g] == int(blockIdx.x)) now[d] = v[d];
            }
        }
    }
    __syncthreads();
    const V3<double> be = make_v3<double>(sb[0], sb[1], sb[2]), sc = iscale[g];
    const bool ba = be.a != 0.0, bb = be.b != 0.0, bc = be.c != 0.0;
    for (int i = c.x + threadIdx.x; i < c.x + c.y; i += CT) {
        V3<double> v = widened(z[i], sc);
        const V3<double> pi = p[i];
        if (ba) v.a += be.a * pi.a;
        if (bb) v.b += be.b * pi.b;
        if (bc) v.c += be.c * pi.c;
        p[i] = v;
    }
}

}  // namespace

void BatchRanges::build(const std::vector<int>& four, int n_unknowns, cudaStream_t s)
{
    PORSOL_REQUIRE(four.size() % 4 == 0, PORSOL_ERR_BAD_ARG, "batch ranges: four entries per block");
    nblk = int(four.size() / 4);
    n = n_unknowns;
    h = four;
    std::vector<int> b(n, -1);
    for (int g = 0; g < nblk; ++g)
        for (int k = 0; k < 2; ++k) {
            const int r0 = four[4 * g + 2 * k], r1 = four[4 * g + 2 * k + 1];
            PORSOL_REQUIRE(0 <= r0 && r0 <= r1 && r1 <= n, PORSOL_ERR_BAD_ARG, "batch ranges out of bounds");
            for (int i = r0; i < r1; ++i) {
                PORSOL_REQUIRE(b[i] < 0, PORSOL_ERR_BAD_ARG, "batch ranges overlap");
                b[i] = g;
            }
        }
    for (int i = 0; i < n; ++i) PORSOL_REQUIRE(b[i] >= 0, PORSOL_ERR_BAD_ARG, "batch ranges do not cover every unknown");
    ranges.upload(four, s);
    blk.upload(b, s);
    std::vector<int4> ch;
    std::vector<int> cp{0};
    for (int g = 0; g < nblk; ++g) {
        for (int k = 0; k < 2; ++k)
            for (int i = four[4 * g + 2 * k], e = four[4 * g + 2 * k + 1]; i < e; i += CHUNK)
                ch.push_back(make_int4(i, std::min(CHUNK, e - i), g, 0));
        cp.push_back(int(ch.size()));
    }
    nchunks = int(ch.size());
    chunks.upload(ch, s);
    cptr.upload(cp, s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
}

template <class TV, class T>
void BatchedPcg<TV, T>::setup(int n, int nblk, cudaStream_t s)
{
    if (n != n_) {
        r_.alloc(n);
        z_.alloc(n);
        p_.alloc(n);
        q_.alloc(n);
        n_ = n;
    }
    if (nblk != nblk_) {
        rho_.alloc(nblk);
        rholast_.alloc(nblk);
        lambda_.alloc(nblk);
        beta_.alloc(nblk);
        def0_.alloc(nblk);
        def_.alloc(nblk);
        conv_.alloc(nblk);
        nblk_ = nblk;
    }
    st_.alloc(1);
    if (!counter_.p) {
        counter_.alloc(1);
        counter_.zero(s);
    }
    if (!hview_) {
        PORSOL_CUDA(cudaHostAlloc((void**)&hview_, sizeof(BatchHostView), cudaHostAllocMapped));
        PORSOL_CUDA(cudaHostGetDevicePointer((void**)&dview_, hview_, 0));
    }
    if (ev_.empty()) {
        ev_.resize(4);
        for (auto& e : ev_) PORSOL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
}

template <class TV, class T>
BatchedPcg<TV, T>::~BatchedPcg()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (hview_) cudaFreeHost(hview_);
    for (auto& e : ev_) cudaEventDestroy(e);
}

template <class TV, class T>
void BatchedPcg<TV, T>::iteration(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M,
                                  const BatchRanges& B, T* x, const double* tol)
{
    const int n = P.n, nb = div_up(n, BT), g = B.nblk;
    const int* stop = &st_.p->stop;
    PORSOL_LAUNCH(k_b_spmv<TV, T><<<nb, BT, 0, s>>>(n, P.slice_ptr.p, P.col.p, val, p_.p, q_.p, B.blk.p, conv_.p,
                                                    st_.p));
    PORSOL_LAUNCH(k_b_pq<T><<<g, RT, 0, s>>>(B.ranges.p, p_.p, q_.p, rholast_.p, conv_.p, lambda_.p, st_.p));
    PORSOL_LAUNCH(k_b_update<T><<<nb, BT, 0, s>>>(n, B.blk.p, lambda_.p, x, r_.p, p_.p, q_.p, st_.p));
    PORSOL_LAUNCH(k_b_rr<T><<<g, RT, 0, s>>>(g, B.ranges.p, r_.p, def0_.p, def_.p, tol, conv_.p, st_.p, counter_.p,
                                             dview_));
    M.apply(s, r_.p, z_.p, stop);
    PORSOL_LAUNCH(k_b_zr<T><<<g, RT, 0, s>>>(B.ranges.p, z_.p, r_.p, rholast_.p, beta_.p, conv_.p, 0, st_.p));
    PORSOL_LAUNCH(k_b_direction<T><<<nb, BT, 0, s>>>(n, B.blk.p, beta_.p, z_.p, p_.p, st_.p));
}

template <class TV, class T>
CgResult BatchedPcg<TV, T>::solve(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M,
                                  const BatchRanges& B, const T* b, T* x, const double* tol, int maxit)
{
    const int n = P.n;
    CgResult res;
    PORSOL_REQUIRE(B.n == n && B.nblk > 0, PORSOL_ERR_BAD_ARG, "batched CG: ranges do not match the system");
    setup(n, B.nblk, s);
    // a block-diagonal preconditioner skips the converged blocks' rows (PORSOL_BLOCK_SKIP=0 in the
    // environment: it sweeps every row, with the same results)
    const char* skip_env = std::getenv("PORSOL_BLOCK_SKIP");
    M.set_block_state(skip_env && skip_env[0] == '0' ? nullptr : conv_.p);
    const int nb = div_up(n, BT), g = B.nblk;
    BatchDev init{};
    init.maxit = maxit;
    PORSOL_CUDA(cudaMemcpyAsync(st_.p, &init, sizeof(BatchDev), cudaMemcpyHostToDevice, s));
    p_.zero(s);
    PORSOL_LAUNCH(k_b_residual<TV, T><<<nb, BT, 0, s>>>(n, P.slice_ptr.p, P.col.p, val, x, b, r_.p));
    PORSOL_LAUNCH(k_b_init<T><<<g, RT, 0, s>>>(g, B.ranges.p, r_.p, def0_.p, def_.p, conv_.p, st_.p, counter_.p,
                                               dview_));
    const int* stop = &st_.p->stop;
    M.apply(s, r_.p, z_.p, stop);
    PORSOL_LAUNCH(k_b_zr<T><<<g, RT, 0, s>>>(B.ranges.p, z_.p, r_.p, rholast_.p, beta_.p, conv_.p, 1, st_.p));
    PORSOL_LAUNCH(k_b_direction<T><<<nb, BT, 0, s>>>(n, B.blk.p, beta_.p, z_.p, p_.p, st_.p));
    PORSOL_CUDA(cudaGetLastError());
    const void* key[6] = {&P, val, x, (const void*)&M, (const void*)&B, tol};
    bool same = exec_ && key_gen_ == M.generation();
    for (int k = 0; k < 6 && same; ++k) same = key_[k] == key[k];
    if (!same) {
        if (exec_) {
            cudaGraphExecDestroy(exec_);
            exec_ = nullptr;
        }
        cudaGraph_t gr;
        const long long l0 = g_launches.load();
        PORSOL_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        iteration(s, P, val, M, B, x, tol);
        PORSOL_CUDA(cudaStreamEndCapture(s, &gr));
        nodes_ = g_launches.load() - l0;
        g_launches.fetch_sub(nodes_);
        PORSOL_CUDA(cudaGraphInstantiate(&exec_, gr, 0));
        PORSOL_CUDA(cudaGraphDestroy(gr));
        for (int k = 0; k < 6; ++k) key_[k] = key[k];
        key_gen_ = M.generation();
    }
    // Same host loop as PcgSolver: iterations queued two ahead, stop read from mapped memory.
    const int LOOKAHEAD = 2;
    int it = 0;
    bool done = false;
    while (!done) {
        if (it < maxit) {
            PORSOL_CUDA(cudaGraphLaunch(exec_, s));
            g_launches.fetch_add(nodes_);
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
    res.breakdown = hview_->breakdown != 0;
    res.converged = hview_->active == 0 && !res.breakdown;
    std::vector<double> d0(g), d1(g);
    def0_.download(d0.data(), g, s);
    def_.download(d1.data(), g, s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
    double red = 0.0, s0 = 0.0, s1 = 0.0;
    for (int k = 0; k < g; ++k) {
        if (d0[k] > 0) red = std::max(red, d1[k] / d0[k]);
        s0 += d0[k] * d0[k];
        s1 += d1[k] * d1[k];
    }
    res.reduction = red;
    res.def0 = std::sqrt(s0);
    res.def = std::sqrt(s1);
    return res;
}

template class BatchedPcg<double, double>;

// ---------------- BatchedCg3 ----------------
BatchedCg3::~BatchedCg3()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (hview_) cudaFreeHost(hview_);
    for (auto& e : ev_) cudaEventDestroy(e);
}

void BatchedCg3::setup(const BatchRanges& B, bool fp32, cudaStream_t s)
{
    const size_t n = B.n, nb = B.nblk;
    for (DBuf<V3<double>>* v : {&r_, &p_, &q_}) v->alloc(n);
    if (fp32) {
        r32_.alloc(n);
        z32_.alloc(n);
    } else {
        z64_.alloc(n);
    }
    for (DBuf<V3<double>>* v : {&part_, &part2_}) v->alloc(size_t(B.nchunks));
    for (DBuf<V3<double>>* v : {&scale_, &iscale_}) v->alloc(nb);
    rho_.alloc(6 * nb);
    def0_.alloc(3 * nb);
    def_.alloc(3 * nb);
    done_.alloc(3 * nb);
    broken_.alloc(3 * nb);
    conv_.alloc(nb);
    st_.alloc(1);
    if (!counter_.p) {
        counter_.alloc(1);
        counter_.zero(s);
    }
    if (!hview_) {
        PORSOL_CUDA(cudaHostAlloc((void**)&hview_, sizeof(Batch3HostView), cudaHostAllocMapped));
        PORSOL_CUDA(cudaHostGetDevicePointer((void**)&dview_, hview_, 0));
    }
    if (ev_.empty()) {
        ev_.resize(4);
        for (auto& e : ev_) PORSOL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
}

template <class T>
void BatchedCg3::precondition(cudaStream_t s, Amg<T>& M)
{
    const int* stop = &st_.p->stop;
    if constexpr (sizeof(T) == 4) M.apply3(s, r32_.p, z32_.p, stop);
    else M.apply3(s, r_.p, z64_.p, stop);
}

template <class T>
void BatchedCg3::iteration(cudaStream_t s, const SellPattern& P, const double* val, Amg<T>& M, const BatchRanges& B,
                           V3<double>* x, double tol)
{
    const int nc = B.nchunks, nt = div_up(B.nblk, CT / 32);
    PORSOL_LAUNCH(k_b3_pq<<<nc, CT, 0, s>>>(B.chunks.p, P.slice_ptr.p, P.col.p, val, p_.p, q_.p, conv_.p, part_.p, st_.p));
    PORSOL_LAUNCH(k_b3_update<T><<<nc, CT, 0, s>>>(B.chunks.p, B.cptr.p, part_.p, rho_.p, B.nblk, done_.p, broken_.p,
                                                   conv_.p, x, r_.p, p_.p, q_.p, scale_.p, (V3<T>*)r32_.p, part2_.p,
                                                   st_.p));
    PORSOL_LAUNCH(k_b3_test<<<nt, CT, 0, s>>>(B.nblk, B.cptr.p, part2_.p, tol, 0, def0_.p, def_.p, done_.p, broken_.p,
                                              conv_.p, scale_.p, iscale_.p, st_.p, counter_.p, dview_));
    precondition(s, M);
    direction<T>(s, B, 0);
}

template <class T>
void BatchedCg3::direction(cudaStream_t s, const BatchRanges& B, int first)
{
    const V3<T>* z;
    if constexpr (sizeof(T) == 4) z = z32_.p;
    else z = z64_.p;
    PORSOL_LAUNCH(k_b3_zr<T><<<B.nchunks, CT, 0, s>>>(B.chunks.p, z, r_.p, iscale_.p, conv_.p, part_.p, st_.p));
    PORSOL_LAUNCH(k_b3_direction<T><<<B.nchunks, CT, 0, s>>>(B.chunks.p, B.cptr.p, part_.p, rho_.p, B.nblk, done_.p,
                                                             conv_.p, z, iscale_.p, p_.p, first, st_.p));
}

template <class T>
CgResult BatchedCg3::solve(cudaStream_t s, const SellPattern& P, const double* val, Amg<T>& M, const BatchRanges& B,
                           const double* b3, double* x3, double tol, int maxit)
{
    CgResult res;
    PORSOL_REQUIRE(B.n == P.n && B.nblk > 0, PORSOL_ERR_BAD_ARG, "batched CG: ranges do not match the system");
    setup(B, sizeof(T) == 4, s);
    const V3<double>* b = reinterpret_cast<const V3<double>*>(b3);
    V3<double>* x = reinterpret_cast<V3<double>*>(x3);
    // the preconditioner skips the converged blocks' rows (PORSOL_BLOCK_SKIP=0 in the environment: it
    // sweeps every row, with the same results)
    const char* skip_env = std::getenv("PORSOL_BLOCK_SKIP");
    M.set_block_state(skip_env && skip_env[0] == '0' ? nullptr : conv_.p);
    Batch3Dev init{};
    init.maxit = maxit;
    PORSOL_CUDA(cudaMemcpyAsync(st_.p, &init, sizeof(init), cudaMemcpyHostToDevice, s));
    broken_.zero(s);
    const int nc = B.nchunks;
    PORSOL_LAUNCH(k_b3_residual<<<nc, CT, 0, s>>>(B.chunks.p, P.slice_ptr.p, P.col.p, val, x, b, r_.p, part2_.p));
    PORSOL_LAUNCH(k_b3_test<<<div_up(B.nblk, CT / 32), CT, 0, s>>>(B.nblk, B.cptr.p, part2_.p, tol, 1, def0_.p, def_.p,
                                                                  done_.p, broken_.p, conv_.p, scale_.p, iscale_.p,
                                                                  st_.p, counter_.p, dview_));
    if (sizeof(T) == 4) PORSOL_LAUNCH(k_b3_cast<<<nc, CT, 0, s>>>(B.chunks.p, r_.p, scale_.p, r32_.p));
    precondition(s, M);
    direction<T>(s, B, 1);
    PORSOL_CUDA(cudaGetLastError());
    const void* key[6] = {&P, val, x, (const void*)&M, (const void*)B.chunks.p, (const void*)r32_.p};
    bool same = exec_ && key_gen_ == M.generation() && key_n_[0] == B.nchunks && key_n_[1] == B.nblk && key_tol_ == tol;
    for (int k = 0; k < 6 && same; ++k) same = key_[k] == key[k];
    if (!same) {
        if (exec_) {
            cudaGraphExecDestroy(exec_);
            exec_ = nullptr;
        }
        cudaGraph_t gr;
        const long long l0 = g_launches.load();
        PORSOL_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        iteration(s, P, val, M, B, x, tol);
        PORSOL_CUDA(cudaStreamEndCapture(s, &gr));
        nodes_ = g_launches.load() - l0;
        g_launches.fetch_sub(nodes_);
        PORSOL_CUDA(cudaGraphInstantiate(&exec_, gr, 0));
        PORSOL_CUDA(cudaGraphDestroy(gr));
        for (int k = 0; k < 6; ++k) key_[k] = key[k];
        key_gen_ = M.generation();
        key_n_[0] = B.nchunks;
        key_n_[1] = B.nblk;
        key_tol_ = tol;
    }
    // Same host loop as PcgSolver: iterations queued two ahead, stop read from mapped memory.
    const int LOOKAHEAD = 2;
    int it = 0;
    bool stopped = false;
    while (!stopped) {
        if (it < maxit) {
            PORSOL_CUDA(cudaGraphLaunch(exec_, s));
            g_launches.fetch_add(nodes_);
            PORSOL_CUDA(cudaEventRecord(ev_[it % ev_.size()], s));
            ++it;
        }
        if (it >= LOOKAHEAD || it >= maxit) {
            const int wait_it = (it >= maxit) ? it - 1 : it - LOOKAHEAD;
            PORSOL_CUDA(cudaEventSynchronize(ev_[wait_it % ev_.size()]));
            if (hview_->stop || it >= maxit) {
                if (it >= maxit) PORSOL_CUDA(cudaStreamSynchronize(s));
                stopped = hview_->stop || it >= maxit;
            }
        }
    }
    PORSOL_CUDA(cudaStreamSynchronize(s));
    for (int d = 0; d < 3; ++d) res.iterations += hview_->iters[d];
    res.breakdown = hview_->breakdown != 0;
    res.converged = hview_->active == 0 && !res.breakdown;
    std::vector<double> d0(3 * size_t(B.nblk)), d1(d0.size());
    def0_.download(d0.data(), d0.size(), s);
    def_.download(d1.data(), d1.size(), s);
    PORSOL_CUDA(cudaStreamSynchronize(s));
    for (size_t k = 0; k < d0.size(); ++k)
        if (d0[k] > 0) res.reduction = std::max(res.reduction, d1[k] / d0[k]);
    return res;
}

template CgResult BatchedCg3::solve<float>(cudaStream_t, const SellPattern&, const double*, Amg<float>&,
                                           const BatchRanges&, const double*, double*, double, int);
template CgResult BatchedCg3::solve<double>(cudaStream_t, const SellPattern&, const double*, Amg<double>&,
                                            const BatchRanges&, const double*, double*, double, int);

}  // namespace porsol
