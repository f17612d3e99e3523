// k_tail.cu -- the cluster kernel of the V-cycle's smallest levels (tail.h).
#include <cuda_fp16.h>

#include <algorithm>

#include "bulk.cuh"
#include "cluster.cuh"
#include "tail.h"

namespace porsol {

namespace {

__device__ __forceinline__ void copy16(unsigned dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// ---- setup: one block per owner and level ----
template <class T, bool HALF>
__global__ void __launch_bounds__(TAIL_THREADS) k_tail_pack(int n, int lanes, const int* __restrict__ sp,
                                                            const int* __restrict__ col,
                                                            const int* __restrict__ rowlen,
                                                            const __half* __restrict__ H, const T* __restrict__ A,
                                                            const T* __restrict__ dinv, const T* __restrict__ dv,
                                                            const int* __restrict__ agg, int nn,
                                                            const int* __restrict__ nptr, const int* __restrict__ nidx,
                                                            int all_members, unsigned char* blob)
{
    __shared__ TailHead hd;
    const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    unsigned char* out = blob + size_t(rank) * TAIL_BLOB;
    const int per = tail_per(n), r0 = min(n, rank * per), own = min(n, r0 + per) - r0;
    const int lr = tid / lanes, q = tid % lanes;
    const bool row = lr < own;
    const int r = r0 + lr;
    const int len = row ? rowlen[r] : 0;
    int it = (len + lanes - 1) / lanes;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) it = max(it, __shfl_xor_sync(0xffffffffu, it, o));
    if (lane == 0) hd.iters[w] = it;
    __syncthreads();
    const int pern = tail_per(nn), c0 = all_members ? 0 : min(nn, rank * pern),
              c1 = all_members ? nn : min(nn, c0 + pern);
    const int m0 = nptr[c0], members = nptr[c1] - m0;
    if (tid == 0) {
        int e = 0;
        for (int k = 0; k < TAIL_THREADS / 32; ++k) {
            hd.woff[k] = e;
            e += 32 * hd.iters[k];
        }
        auto up = [](int b) { return (b + 15) & ~15; };
        int at = up(int(sizeof(TailHead)));
        hd.vals = at;
        at = up(at + e * (HALF ? 4 : int(sizeof(T))));
        hd.cols = at;
        if (!HALF) at = up(at + e * 2);
        hd.dinv = at;
        at = up(at + own * int(sizeof(T)));
        hd.diag = at;
        if (HALF) at = up(at + own * int(sizeof(T)));
        hd.agg = at;
        at = up(at + n * 2);
        hd.mptr = at;
        at = up(at + (c1 - c0 + 1) * 2);
        hd.midx = at;
        at = up(at + members * 2);
        hd.bytes = at;
    }
    __syncthreads();
    if (tid < int(sizeof(TailHead) / 4)) reinterpret_cast<int*>(out)[tid] = reinterpret_cast<const int*>(&hd)[tid];
    if (hd.bytes > TAIL_BLOB) return;
    const int e0 = hd.woff[w] + lane;
    const int b = row ? sp[r >> 5] + (r & 31) : 0;
    unsigned* word = reinterpret_cast<unsigned*>(out + hd.vals);
    T* val = reinterpret_cast<T*>(out + hd.vals);
    unsigned short* cl = reinterpret_cast<unsigned short*>(out + hd.cols);
    for (int k = 0; k < hd.iters[w]; ++k) {
        const int t = q + k * lanes;
        const bool in = t < len;
        const int c = in ? col[b + 32 * t] : (row ? r : 0);
        if (HALF) {
            const unsigned short h = in ? __half_as_ushort(H[b + 32 * t]) : (unsigned short)0;
            word[e0 + 32 * k] = unsigned(h) | (unsigned(c) << 16);
        } else {
            val[e0 + 32 * k] = in ? A[b + 32 * t] : T(0);
            cl[e0 + 32 * k] = (unsigned short)c;
        }
    }
    T* di = reinterpret_cast<T*>(out + hd.dinv);
    T* dg = reinterpret_cast<T*>(out + hd.diag);
    for (int k = tid; k < own; k += blockDim.x) {
        di[k] = dinv[r0 + k];
        if (HALF) dg[k] = dv[r0 + k];
    }
    unsigned short* ag = reinterpret_cast<unsigned short*>(out + hd.agg);
    for (int k = tid; k < n; k += blockDim.x) ag[k] = agg[k] < 0 ? (unsigned short)0xFFFF : (unsigned short)agg[k];
    unsigned short* mp = reinterpret_cast<unsigned short*>(out + hd.mptr);
    for (int k = tid; k <= c1 - c0; k += blockDim.x) mp[k] = (unsigned short)(nptr[c0 + k] - m0);
    unsigned short* mi = reinterpret_cast<unsigned short*>(out + hd.midx);
    for (int k = tid; k < members; k += blockDim.x) mi[k] = (unsigned short)nidx[m0 + k];
}

// ---- the cycle ----
// One smoothed level as this thread sees it: its row (all lanes of a row hold the row's values), its
// warp's entries, the whole vectors.
template <class T, bool HALF>
struct Own {
    const unsigned char* part;
    T *f0, *f1;
    int n, lanes, it, i;        // i: the row (clamped to the level)
    bool row;                   // this thread has one
    int q;
    const unsigned* word;       // HALF: (FP16 value, 16-bit column) per entry
    const T* val;
    const unsigned short* col;
    T dinv, diag;
    const TailHead* hd;
    int lr;
    __device__ Own(const TailLevel<T>& L, unsigned char* sm, int rank)
    {
        part = sm + L.blob;
        hd = reinterpret_cast<const TailHead*>(part);
        f0 = reinterpret_cast<T*>(sm + L.f0);
        f1 = reinterpret_cast<T*>(sm + L.f1);
        n = L.n;
        lanes = L.lanes;
        const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int per = tail_per(n), r0 = min(n, rank * per), own = min(n, r0 + per) - r0;
        lr = threadIdx.x / lanes;
        q = threadIdx.x % lanes;
        row = lr < own;
        i = row ? r0 + lr : 0;
        it = hd->iters[w];
        const int e = hd->woff[w] + lane;
        word = reinterpret_cast<const unsigned*>(part + hd->vals) + e;
        val = reinterpret_cast<const T*>(part + hd->vals) + e;
        col = reinterpret_cast<const unsigned short*>(part + hd->cols) + e;
        dinv = row ? reinterpret_cast<const T*>(part + hd->dinv)[lr] : T(0);
        diag = HALF && row ? reinterpret_cast<const T*>(part + hd->diag)[lr] : T(0);
    }
    // (D^-1) A v for this thread's row, the same in all its lanes
    __device__ T product(const T* v) const
    {
        T acc = T(0);
        if (HALF) {
#pragma unroll 4
            for (int k = 0; k < it; ++k) {
                const unsigned u = word[32 * k];
                acc += T(__half2float(__ushort_as_half((unsigned short)(u & 0xFFFFu)))) * v[u >> 16];
            }
        } else {
#pragma unroll 4
            for (int k = 0; k < it; ++k) acc += val[32 * k] * v[col[32 * k]];
        }
        for (int o = lanes >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        return acc;
    }
    // the row's value into the whole vector of every block; to: the blocks' shared memory
    __device__ void share(const unsigned (&to)[TAIL_CTAS], unsigned base, const T* f, T v) const
    {
        if (!row) return;
        const unsigned a = smem_u32(f + i) - base;
        if (lanes == 1) {
#pragma unroll
            for (int k = 0; k < TAIL_CTAS; ++k) put(to[k] + a, v);
        } else if (lanes == 2) {
#pragma unroll
            for (int k = 0; k < TAIL_CTAS; k += 2) put((q ? to[k + 1] : to[k]) + a, v);
        } else {
            for (int k = q; k < TAIL_CTAS; k += lanes) put(map_rank(a + base, unsigned(k)), v);
        }
    }
};

// What bounds it is the chain of phases (7 per smoothed level, 1 for the dense one): each is the entries'
// shared-memory gathers, the lanes' sum, eight remote stores and a cluster barrier, 1.3 us in all.  A
// row's residual, correction and iterate stay in the registers of its lanes from phase to phase.
// Levels of 3182 and 353 rows and a dense one of 80 (FP16 smoother): 26 us from cold caches, where 16 launches
// took 43 us within the graph; a CG iteration on 255k unknowns went from 166 to 144 us, one in FP64 on 38k
// unknowns (982, 224 and 108 rows here) from 153 to 137 us.
template <class T, bool HALF>
__global__ void __launch_bounds__(TAIL_THREADS, 1) k_tail(const __grid_constant__ TailArgs<T> A)
{
    extern __shared__ __align__(128) unsigned char sm[];
    const int tid = threadIdx.x, rank = int(cluster_rank());
    // Everything that the preceding kernel does not write: the level parts, the dense inverse's rows,
    // the member lists of the first restriction.
    for (int l = 0; l < A.levels; ++l) {
        const unsigned char* src = A.blob + (size_t(l) * TAIL_CTAS + rank) * TAIL_BLOB;
        const unsigned dst = smem_u32(sm + A.lv[l].blob);
        for (int k = 16 * tid; k < A.part_bytes[l]; k += 16 * TAIL_THREADS) copy16(dst + k, src + k);
    }
    const int dper = tail_per(A.nd), d0 = min(A.nd, rank * dper), down = min(A.nd, d0 + dper) - d0;
    double* cinv = reinterpret_cast<double*>(sm + A.dinv);
    for (int k = tid; k < down * A.nd; k += TAIL_THREADS) cinv[k] = A.cinv[size_t(d0) * A.nd + k];
    constexpr int NM = 8;
    int mem[NM], nmem = 0, mfirst = 0;
    {
        const int n = A.lv[0].n, per = tail_per(n), r0 = min(n, rank * per), own = min(n, r0 + per) - r0;
        const int lr = tid / A.lv[0].lanes;
        if (lr < own) {
            mfirst = A.rptr[r0 + lr];
            nmem = A.rptr[r0 + lr + 1] - mfirst;
        }
#pragma unroll
        for (int k = 0; k < NM; ++k)
            if (k < nmem) mem[k] = A.ridx[mfirst + k];
    }
    const unsigned base = smem_u32(sm);
    unsigned to[TAIL_CTAS];
#pragma unroll
    for (int k = 0; k < TAIL_CTAS; ++k) to[k] = map_rank(base, unsigned(k));
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_arrive();   // every block of the cluster runs and has its parts
    chain_wait();
    cluster_wait();
    if (*A.stop) return;

    for (int l = 0; l < A.levels; ++l) {
        const TailLevel<T>& L = A.lv[l];
        const Own<T, HALF> o(L, sm, rank);
        // restriction and start from zero
        T b = T(0);
        if (l == 0) {
#pragma unroll
            for (int k = 0; k < NM; ++k)
                if (k < nmem) b += A.rfine[mem[k]];
            for (int k = NM; k < nmem; ++k) b += A.rfine[A.ridx[mfirst + k]];
        } else if (o.row) {
            const TailLevel<T>& F = A.lv[l - 1];
            const TailHead* fh = reinterpret_cast<const TailHead*>(sm + F.blob);
            const unsigned short* mp = reinterpret_cast<const unsigned short*>(sm + F.blob + fh->mptr);
            const unsigned short* mi = reinterpret_cast<const unsigned short*>(sm + F.blob + fh->midx);
            const T* res = reinterpret_cast<const T*>(sm + F.f1);
            for (int k = mp[o.lr]; k < mp[o.lr + 1]; ++k) b += res[mi[k]];
        }
        if (o.row && o.q == 0) reinterpret_cast<T*>(sm + L.bo)[o.lr] = b;
        T r = o.dinv * b, d = r * L.inv_theta;
        o.share(to, base, o.f0, d);
        cluster_sync();
        // two Chebyshev steps
        T acc = o.product(o.f0);
        r -= HALF ? acc : o.dinv * acc;
        T x = d;
        d = L.c1[0] * d + L.c2[0] * r;
        o.share(to, base, o.f1, d);
        cluster_sync();
        acc = o.product(o.f1);
        r -= HALF ? acc : o.dinv * acc;
        x = (x + d) + (L.c1[1] * d + L.c2[1] * r);
        o.share(to, base, o.f0, x);
        cluster_sync();
        // residual
        acc = o.product(o.f0);
        o.share(to, base, o.f1, b - (HALF ? o.diag * acc : acc));
        cluster_sync();
    }
    // the dense level: every block restricts all of it and solves its own rows
    {
        const TailLevel<T>& F = A.lv[A.levels - 1];
        const TailHead* fh = reinterpret_cast<const TailHead*>(sm + F.blob);
        const unsigned short* mp = reinterpret_cast<const unsigned short*>(sm + F.blob + fh->mptr);
        const unsigned short* mi = reinterpret_cast<const unsigned short*>(sm + F.blob + fh->midx);
        const T* res = reinterpret_cast<const T*>(sm + F.f1);
        T* db = reinterpret_cast<T*>(sm + A.db);
        for (int i = tid; i < A.nd; i += TAIL_THREADS) {
            T b = T(0);
            for (int k = mp[i]; k < mp[i + 1]; ++k) b += res[mi[k]];
            db[i] = b;
        }
        __syncthreads();
        const int w = tid >> 5, lane = tid & 31;
        for (int i = w; i < down; i += TAIL_THREADS / 32) {
            double s = 0.0;
            for (int j = lane; j < A.nd; j += 32) s += cinv[i * A.nd + j] * double(db[j]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane < TAIL_CTAS)
                put(map_rank(smem_u32(reinterpret_cast<T*>(sm + A.dx) + d0 + i), unsigned(lane)), T(s));
        }
        cluster_sync();
    }
    for (int l = A.levels - 1; l >= 0; --l) {
        const TailLevel<T>& L = A.lv[l];
        const Own<T, HALF> o(L, sm, rank);
        // y = t + w P xc, by every block for all rows
        const T* xc = reinterpret_cast<const T*>(sm + (l + 1 < A.levels ? A.lv[l + 1].f1 : A.dx));
        const unsigned short* ag = reinterpret_cast<const unsigned short*>(o.part + o.hd->agg);
        for (int i = tid; i < L.n; i += TAIL_THREADS) {
            const int a = ag[i];
            if (a != 0xFFFF) o.f0[i] += A.wp * xc[a];
        }
        const T b = o.row ? reinterpret_cast<const T*>(sm + L.bo)[o.lr] : T(0);
        __syncthreads();
        T x = o.f0[o.i];
        T acc = o.product(o.f0);
        T r = HALF ? o.dinv * b - acc : o.dinv * (b - acc), d = r * L.inv_theta;
        o.share(to, base, o.f1, d);
        cluster_sync();
        acc = o.product(o.f1);
        x += d;
        r -= HALF ? acc : o.dinv * acc;
        d = L.c1[0] * d + L.c2[0] * r;
        o.share(to, base, o.f0, d);
        cluster_sync();
        acc = o.product(o.f0);
        r -= HALF ? acc : o.dinv * acc;
        x = (x + d) + (L.c1[1] * d + L.c2[1] * r);
        if (l > 0) {
            o.share(to, base, o.f1, x);
            cluster_sync();
        } else if (o.row && o.q == 0) {
            A.x[o.i] = x;
        }
    }
}

}  // namespace

int tail_lanes(int n)
{
    int k = 1;
    while (k < 32 && tail_per(n) * 2 * k <= TAIL_LANE_THREADS) k *= 2;
    return k;
}

template <class T>
void tail_pack(cudaStream_t s, int n, const int* sp, const int* col, const int* rowlen, const void* h, const T* A,
               const T* dinv, const T* dv, const int* agg, int nn, const int* nptr, const int* nidx, bool all_members,
               unsigned char* blob)
{
    const int lanes = tail_lanes(n);
    if (h)
        PORSOL_LAUNCH((k_tail_pack<T, true><<<TAIL_CTAS, TAIL_THREADS, 0, s>>>(
            n, lanes, sp, col, rowlen, (const __half*)h, A, dinv, dv, agg, nn, nptr, nidx, all_members ? 1 : 0, blob)));
    else
        PORSOL_LAUNCH((k_tail_pack<T, false><<<TAIL_CTAS, TAIL_THREADS, 0, s>>>(
            n, lanes, sp, col, rowlen, nullptr, A, dinv, dv, agg, nn, nptr, nidx, all_members ? 1 : 0, blob)));
    PORSOL_CUDA(cudaGetLastError());
}

template <class T>
int tail_layout(TailArgs<T>& a)
{
    int at = 0;
    auto take = [&](size_t b) {
        const int p = at;
        at += int((b + 15) / 16 * 16);
        return p;
    };
    for (int l = 0; l < a.levels; ++l) {
        TailLevel<T>& L = a.lv[l];
        L.blob = take(size_t(a.part_bytes[l]));
        L.f0 = take(L.n * sizeof(T));
        L.f1 = take(L.n * sizeof(T));
        const size_t own = tail_per(L.n) * sizeof(T);
        L.bo = take(own);
    }
    a.db = take(a.nd * sizeof(T));
    a.dx = take(a.nd * sizeof(T));
    a.dinv = take(size_t(tail_per(a.nd)) * a.nd * sizeof(double));
    return at;
}

template <class T>
bool tail_fits(bool half)
{
    return half ? cluster_fits(k_tail<T, true>, TAIL_CTAS, TAIL_THREADS, TAIL_SMEM)
                : cluster_fits(k_tail<T, false>, TAIL_CTAS, TAIL_THREADS, TAIL_SMEM);
}

template <class T>
void tail_launch(cudaStream_t s, bool half, const TailArgs<T>& a, int shm)
{
    auto* f = half ? k_tail<T, true> : k_tail<T, false>;
    PORSOL_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_SMEM));
    launch_cluster(f, TAIL_CTAS, TAIL_THREADS, size_t(shm), s, chain_enabled(TAIL_CTAS), a);
}

#define PORSOL_TAIL(T)                                                                                              \
    template void tail_pack<T>(cudaStream_t, int, const int*, const int*, const int*, const void*, const T*,         \
                               const T*, const T*, const int*, int, const int*, const int*, bool, unsigned char*);   \
    template int tail_layout<T>(TailArgs<T>&);                                                                       \
    template void tail_launch<T>(cudaStream_t, bool, const TailArgs<T>&, int);                                       \
    template bool tail_fits<T>(bool);
PORSOL_TAIL(float)
PORSOL_TAIL(double)
#undef PORSOL_TAIL

}  // namespace porsol
