// k_aggregate.cu -- the cluster kernels of aggregate.h.
//
// Arrays that other blocks write within the launch are read past the first-level cache (__ldcg), which is
// not coherent between SMs.  The decisions of a sweep depend on the picks and states of the sweep only and
// the member lists are sorted, so the results are those of the launch-per-step path.
#include <climits>

#include "aggregate.h"
#include "bulk.cuh"
#include "cluster.cuh"
#include "match.cuh"

namespace porsol {

namespace {

struct Part {   // what this block owns of [0, n)
    int lo, hi;
    __device__ Part(int n, int rank)
    {
        const int blocks = gridDim.x, per = (n + blocks - 1) / blocks;
        lo = min(n, rank * per);
        hi = min(n, lo + per);
    }
};

// inclusive sum over the block's threads; *total: the block's sum
__device__ __forceinline__ int block_scan(int v, int* total)
{
    __shared__ int ws[AGG_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    if (w == 0) {
        const int x = ws[lane];
        int s = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        ws[lane] = s;
    }
    __syncthreads();
    const int r = inc + (w ? ws[w - 1] : 0);
    *total = ws[AGG_THREADS / 32 - 1];
    __syncthreads();
    return r;
}

// Exclusive sum of value(i) over [0, n) into put(i, sum), each block its own part: the parts' totals are
// exchanged through tot[0 .. AGG_CTAS).  value() is called twice per element.  Returns the whole sum.
// Every thread of the cluster calls it; it contains one cluster barrier, before the first put().
template <class V, class P>
__device__ int cluster_scan(const Part& p, int rank, int* tot, V value, P put)
{
    int mine = 0, t;
    for (int i = p.lo + threadIdx.x; i < p.hi; i += AGG_THREADS) mine += value(i);
    block_scan(mine, &t);
    if (threadIdx.x == 0) tot[rank] = t;
    cluster_sync();
    int before = 0, all = 0;
    for (int k = 0; k < int(gridDim.x); ++k) {
        const int x = __ldcg(tot + k);
        if (k < rank) before += x;
        all += x;
    }
    for (int base = p.lo; base < p.hi; base += AGG_THREADS) {
        const int i = base + threadIdx.x;
        const int v = i < p.hi ? value(i) : 0;
        const int inc = block_scan(v, &t);
        if (i < p.hi) put(i, before + inc - v);
        before += t;
    }
    return all;
}

// the best candidate over this lane's entries q, q + K, ... of row i
template <int K, class T>
__device__ __forceinline__ void best_entry(const AggArgs<T>& a, int i, int q, int want, bool neg, float floor_s,
                                           float& bs, unsigned& bh, int& bj)
{
    const float ri = __ldcg(a.rs + i);
    const int len = a.rowlen[i], k0 = a.sp[i >> 5] + (i & 31);
    int t = q;
    for (; t + 3 * K < len; t += 4 * K) {
        const int ka = k0 + 32 * t;
        const int j0 = a.col[ka], j1 = a.col[ka + 32 * K], j2 = a.col[ka + 64 * K], j3 = a.col[ka + 96 * K];
        const float v0 = float(a.A[ka]), v1 = float(a.A[ka + 32 * K]), v2 = float(a.A[ka + 64 * K]),
                    v3 = float(a.A[ka + 96 * K]);
        const int s0 = __ldcg(a.state + j0), s1 = __ldcg(a.state + j1), s2 = __ldcg(a.state + j2),
                  s3 = __ldcg(a.state + j3);
        const float r0 = __ldcg(a.rs + j0), r1 = __ldcg(a.rs + j1), r2 = __ldcg(a.rs + j2), r3 = __ldcg(a.rs + j3);
        consider(i, j0, v0, s0, r0, ri, want, neg, floor_s, bs, bh, bj);
        consider(i, j1, v1, s1, r1, ri, want, neg, floor_s, bs, bh, bj);
        consider(i, j2, v2, s2, r2, ri, want, neg, floor_s, bs, bh, bj);
        consider(i, j3, v3, s3, r3, ri, want, neg, floor_s, bs, bh, bj);
    }
    for (; t < len; t += K) {
        const int k = k0 + 32 * t, j = a.col[k];
        consider(i, j, float(a.A[k]), __ldcg(a.state + j), __ldcg(a.rs + j), ri, want, neg, floor_s, bs, bh, bj);
    }
}

// Matching on the couplings of one kind (neg: strong negative ones; else all, with joins): state, partner,
// join of every row.  state as in k_isolated / k_match_wl.
template <int K, class T>
__device__ void match(const AggArgs<T>& a, const Part& p, int* wl, int per, bool neg)
{
    __shared__ int count, left[AGG_CTAS];   // rows still free here and in every block after a sweep
    const int lane = threadIdx.x & 31, tid = threadIdx.x;
    // strengths' scales; rows without a coupling are isolated
    for (int base = (tid & ~31); base < (p.hi - p.lo) * K; base += AGG_THREADS) {
        const int g = base + lane, i = p.lo + g / K, q = g % K;
        const bool valid = i < p.hi;
        bool coupled = false;
        if (valid) {
            const int len = a.rowlen[i], k0 = a.sp[i >> 5] + (i & 31);
            for (int t = q; t < len && !coupled; t += K) {
                const int k = k0 + 32 * t;
                coupled = a.col[k] != i && a.A[k] != T(0);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, coupled);
        const unsigned group = K == 32 ? 0xffffffffu : ((1u << K) - 1u) << (lane / K * K);
        if (valid && q == 0) {
            a.rs[i] = rsqrtf(fabsf(float(a.A[a.diag[i]])));
            a.state[i] = (m & group) ? 0 : 2;
            a.partner[i] = -1;
            a.join[i] = -1;
        }
    }
    const int sweeps = neg ? 4 : 8;
    const float floor_s = neg ? a.theta : 0.0f;
    int todo = p.hi - p.lo;   // this block's rows still free (all of them at first)
    cluster_sync();
    for (int sweep = 0; sweep < sweeps; ++sweep) {
        const int* cur = wl + (sweep & 1) * per;
        int* nxt = wl + ((sweep & 1) ^ 1) * per;
        if (tid == 0) count = 0;
        for (int base = (tid & ~31); base < todo * K; base += AGG_THREADS) {
            const int g = base + lane, at = g / K, q = g % K;
            const bool valid = at < todo;
            const int i = valid ? (sweep ? cur[at] : p.lo + at) : 0;
            const bool active = valid && a.state[i] == 0;   // own row: written by this block only
            float bs = 0.0f;
            unsigned bh = 0u;
            int bj = -1;
            if (active) best_entry<K>(a, i, q, 0, neg, floor_s, bs, bh, bj);
            if (K > 1) best_of_lanes<K>(bs, bh, bj);
            if (valid && q == 0) a.best[i] = active ? bj : -1;
        }
        cluster_sync();
        for (int base = (tid & ~31); base < todo; base += AGG_THREADS) {
            const int at = base + lane;
            bool keep = false;
            int i = 0;
            if (at < todo) {
                i = sweep ? cur[at] : p.lo + at;
                if (a.state[i] == 0) {
                    const int j = a.best[i];
                    if (j >= 0 && __ldcg(a.best + j) == i) {
                        a.state[i] = 1;
                        a.partner[i] = j;
                    } else if (j < 0) {
                        a.state[i] = 3;
                    } else {
                        keep = true;
                    }
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            int o = 0;
            if (lane == 0 && m) o = atomicAdd(&count, __popc(m));
            o = __shfl_sync(0xffffffffu, o, 0);
            if (keep) nxt[o + __popc(m & ((1u << lane) - 1u))] = i;
        }
        __syncthreads();
        if (tid < int(gridDim.x)) put(map_rank(smem_u32(left + cluster_rank()), unsigned(tid)), count);
        cluster_sync();
        todo = count;
        int all = 0;
        for (int k = 0; k < int(gridDim.x); ++k) all += left[k];
        if (all == 0) break;   // the same in every block; further sweeps would change nothing
        __syncthreads();
    }
    if (neg) return;
    // unmatched rows join their strongest paired neighbour
    for (int base = (tid & ~31); base < (p.hi - p.lo) * K; base += AGG_THREADS) {
        const int g = base + lane, i = p.lo + g / K, q = g % K;
        const bool valid = i < p.hi;
        const int st = valid ? a.state[i] : 2;
        const bool active = st == 0 || st == 3;
        float bs = 0.0f;
        unsigned bh = 0u;
        int bj = -1;
        if (active) best_entry<K>(a, i, q, 1, false, 0.0f, bs, bh, bj);
        if (K > 1) best_of_lanes<K>(bs, bh, bj);
        if (active && q == 0) a.join[i] = bj;
    }
    cluster_sync();
}

constexpr int SORT_REG = 12;   // members sorted in registers: rounds of three pairings make about eight

// member lists of agg over nc aggregates: ptr and sorted idx
__device__ void member_lists(const Part& rows, int rank, int nc, const int* agg, int* cnt, int* ptr, int* idx, int* tot)
{
    const Part c(nc, rank);
    for (int k = c.lo + threadIdx.x; k < c.hi; k += AGG_THREADS) cnt[k] = 0;
    cluster_sync();
    for (int i = rows.lo + threadIdx.x; i < rows.hi; i += AGG_THREADS) {
        const int g = __ldcg(agg + i);
        if (g >= 0) atomicAdd(cnt + g, 1);
    }
    cluster_sync();
    const int all = cluster_scan(
        c, rank, tot, [&](int k) { return __ldcg(cnt + k); },
        [&](int k, int at) {
            ptr[k] = at;
            cnt[k] = at;   // the next free place
        });
    if (rank == 0 && threadIdx.x == 0) ptr[nc] = all;
    cluster_sync();
    for (int i = rows.lo + threadIdx.x; i < rows.hi; i += AGG_THREADS) {
        const int g = __ldcg(agg + i);
        if (g >= 0) idx[atomicAdd(cnt + g, 1)] = i;
    }
    cluster_sync();
    for (int k = c.lo + threadIdx.x; k < c.hi; k += AGG_THREADS) {
        const int b = ptr[k], e = __ldcg(cnt + k);
        if (e - b <= SORT_REG) {   // all loads in flight, each member placed by the number of smaller ones
            int v[SORT_REG];
#pragma unroll
            for (int x = 0; x < SORT_REG; ++x) v[x] = b + x < e ? __ldcg(idx + b + x) : INT_MAX;
#pragma unroll
            for (int x = 0; x < SORT_REG; ++x) {
                int at = 0;
#pragma unroll
                for (int y = 0; y < SORT_REG; ++y) at += v[y] < v[x];
                if (b + x < e) __stcg(idx + b + at, v[x]);
            }
            continue;
        }
        for (int x = b + 1; x < e; ++x) {
            const int key = __ldcg(idx + x);
            int y = x - 1;
            for (int v; y >= b && (v = __ldcg(idx + y)) > key; --y) __stcg(idx + y + 1, v);
            __stcg(idx + y + 1, key);
        }
    }
}

// Latency bound: about 30 cluster barriers and as many dependent L2 accesses; the level's entries are
// read by the cluster's SMs once for the isolated rows, once per full sweep and for the rows still free after it.
template <class T, int K>
__global__ void __launch_bounds__(AGG_THREADS, 1) k_aggregate(const AggArgs<T> a)
{
    extern __shared__ int wl[];   // two worklists of this block's rows
    const int rank = int(cluster_rank()), tid = threadIdx.x;
    const int per = (a.n + int(gridDim.x) - 1) / int(gridDim.x);
    const Part p(a.n, rank);
    int* tot = a.scratch + 3;
    if (rank == 0 && tid == 0) a.scratch[2] = 0;
    auto flag = [&](int i) {
        const int st = a.state[i];
        return (((st == 0 || st == 3) && a.join[i] < 0) || (st == 1 && i < a.partner[i])) ? 1 : 0;
    };
    int nc = 0;
    for (int pass = a.neg_first ? 0 : 1; pass < 2; ++pass) {
        match<K>(a, p, wl, per, pass == 0);
        nc = cluster_scan(p, rank, tot + pass * AGG_CTAS, flag, [&](int i, int at) { a.cidx[i] = at; });
        if (pass == 0 && double(nc) <= 0.8 * double(a.n)) break;   // did not stall
    }
    cluster_sync();
    for (int i = p.lo + tid; i < p.hi; i += AGG_THREADS) {
        const int st = a.state[i];
        int g;
        if (st == 2) g = -1;
        else if (flag(i)) g = a.cidx[i];
        else if (st == 1) g = __ldcg(a.cidx + a.partner[i]);
        else {
            const int t = a.join[i];
            g = __ldcg(a.cidx + min(t, __ldcg(a.partner + t)));
        }
        __stcg(a.agg + i, g);
    }
    member_lists(p, rank, nc, a.agg, a.cnt, a.ptr, a.idx, tot + 2 * AGG_CTAS);
    // candidate offsets: goff per aggregate (its members' row lengths), woff per member row
    const Part c(nc, rank);
    auto bound = [&](int k) {
        int b = 0;
        for (int q = a.ptr[k], e = __ldcg(a.cnt + k); q < e; ++q) b += a.rowlen[__ldcg(a.idx + q)];
        return b;
    };
    __syncthreads();   // the block's own member lists are sorted
    int most = 0;
    const int all = cluster_scan(c, rank, tot + 3 * AGG_CTAS, bound, [&](int k, int at) {
        a.goff[k] = at;
        int w = at;
        for (int q = a.ptr[k], e = __ldcg(a.cnt + k); q < e; ++q) {
            const int r = __ldcg(a.idx + q);
            a.woff[r] = w;
            w += a.rowlen[r];
        }
        most = max(most, w - at);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    if ((tid & 31) == 0) atomicMax(a.scratch + 2, most);
    if (rank == 0 && tid == 0) {
        a.goff[nc] = all;
        a.scratch[0] = nc;
        a.scratch[1] = all;
    }
}

__global__ void __launch_bounds__(AGG_THREADS, 1) k_compose_members(int n, int nc, int* agg1, const int* __restrict__ agg2,
                                                                    int* cnt, int* ptr, int* idx, int* scratch)
{
    const int rank = int(cluster_rank());
    const Part p(n, rank);
    for (int i = p.lo + threadIdx.x; i < p.hi; i += AGG_THREADS) {
        const int g = agg1[i];
        __stcg(agg1 + i, g < 0 ? -1 : agg2[g]);
    }
    __syncthreads();
    member_lists(p, rank, nc, agg1, cnt, ptr, idx, scratch + 3);
}

}  // namespace

namespace {

// Bytes of the two worklists of a block.
size_t worklists(int rows, int blocks) { return 2 * sizeof(int) * size_t((rows + blocks - 1) / blocks); }

// Blocks of the cluster: what a level's lanes need at one row (or lane) per thread and sweep, at most 16 (the
// opt-in size; the grid is one cluster), 8 where 16 do not fit the device or the limit; 0: none does.  With fewer
// than that a level of these sizes would be done sooner by a launch per step.
template <class... KA>
int blocks_for(void (*f)(KA...), long long threads, bool lists, int limit)
{
    int b = 1;
    while (b < AGG_CTAS && threads > (long long)b * AGG_THREADS) b *= 2;
    for (; b > 0; b = b > 8 ? 8 : 0) {
        // the largest level that this many blocks may get: up to AGG_ROWS rows for 8 and 16 blocks
        const int rows = b >= 8 ? AGG_ROWS : b * AGG_THREADS;
        if (b <= limit && cluster_fits(f, b, AGG_THREADS, lists ? worklists(rows, b) : 0)) return b;
    }
    return 0;
}

template <class T, int K>
bool agg_launch_lanes(cudaStream_t s, const AggArgs<T>& a, int limit)
{
    const int blocks = blocks_for(k_aggregate<T, K>, (long long)a.n * K, true, limit);
    if (blocks)
        launch_cluster(k_aggregate<T, K>, blocks, AGG_THREADS, worklists(a.n, blocks), s, false, a);
    return blocks != 0;
}

}  // namespace

template <class T>
bool agg_launch(cudaStream_t s, int lanes, const AggArgs<T>& a, int limit)
{
    switch (lanes) {
    case 1: return agg_launch_lanes<T, 1>(s, a, limit);
    case 2: return agg_launch_lanes<T, 2>(s, a, limit);
    case 4: return agg_launch_lanes<T, 4>(s, a, limit);
    case 8: return agg_launch_lanes<T, 8>(s, a, limit);
    default: return agg_launch_lanes<T, 16>(s, a, limit);
    }
}

bool compose_launch(cudaStream_t s, int n, int nc, int* agg1, const int* agg2, int* cnt, int* ptr, int* idx, int* scratch,
                    int limit)
{
    const int blocks = blocks_for(k_compose_members, n, false, limit);
    if (blocks)
        launch_cluster(k_compose_members, blocks, AGG_THREADS, 0, s, false, n, nc, agg1, agg2, cnt, ptr, idx, scratch);
    return blocks != 0;
}

template bool agg_launch<float>(cudaStream_t, int, const AggArgs<float>&, int);
template bool agg_launch<double>(cudaStream_t, int, const AggArgs<double>&, int);

}  // namespace porsol
