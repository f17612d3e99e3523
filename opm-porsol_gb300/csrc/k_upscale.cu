// k_upscale.cu -- PersistentUpscale: the three periodic solves of every sub-grid of a batch in one
// persistent kernel launch.
//
// Work items are sub-grids, taken from device counters, largest first: cluster items (a cluster of
// 2 or 4 CTAs per sub-grid, on as many SMs), then CTA items (a whole CTA per sub-grid), then warp
// items (one warp per sub-grid).  The group that owns an
// item runs a Jacobi-preconditioned CG for the three unit pressure-jump right-hand sides together,
// with FP32 recurrences (matrix copy, vectors and products in FP32: one matrix read feeds three
// products) and reliable updates in FP64 (solution, true residual, convergence test), with
// group-local reductions only (warp shuffles, plus shared memory across the warps of a CTA and
// distributed shared memory across the CTAs of a cluster), so no sub-grid ever waits for another.  A direction stops when its true residual meets
// ||b - A x|| < tol ||b|| or ||b - A x|| < 1e-30 (the per-block test of the batched AMG solve); it
// is frozen from then on.  FP32 matters on this GPU: one SM runs the largest sub-grid alone, and
// with FP64 products its FP64 pipe, not memory, set the time (ncu: 95 % busy).  Every sum runs in a
// fixed order for a given schedule: results are run-to-run reproducible; another CTA size changes
// the summation order.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <numeric>
#include <unordered_map>

#include <cooperative_groups.h>

#include "upscale.h"

namespace porsol {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int UP_MAX_THREADS = 1024;
constexpr int UP_MAX_WARPS = UP_MAX_THREADS / 32;
constexpr int TUNE_ITERS = 48;   // CG iterations of the largest sub-grid in one autotuner trial
namespace cg = cooperative_groups;

// The group of threads that solves one sub-grid: a warp, a CTA, or a cluster of CTAs.
constexpr int G_WARP = 0, G_CTA = 1, G_CLUSTER = 2;

struct UpArgs {
    int trial;            // > 0: a trial; unknowns of the largest sub-grid
    int nitems, ncl, ntile, maxit, n;   // items [0, ncl): clusters; then ntile CTA items; then warp items
    double tol, delta;
    const int* order;     // sub-grid ids: tile items [0, ntile), then warp items
    const int* ranges;    // 4 per sub-grid
    const int* sp;        // SELL-32 union matrix: FP64 values and their FP32 copy
    const int* col;
    const double* val;
    const float* val32;
    const int* diag;
    const double* b3;     // right-hand sides, side by side
    double* x3;           // solutions (FP64)
    double* r64;          // true residuals at replacements (FP64)
    float* r32;           // CG vectors (FP32, in units of the direction's sigma)
    float4* p4;
    float* q32;
    float* dinv;          // 1 / a_ii
    int* iters;           // 3 per sub-grid: iteration at which the direction met its test, -1: never
    double* red;          // 3 per sub-grid: last true ||r|| / ||r0||
    int* counters;        // [0]: next cluster item, [1]: next CTA item, [2]: next warp item
    int* status;
};

// The unknowns of one sub-grid: local index k < n1 is row r0 + k, otherwise row r2 + (k - n1).
struct Rows {
    int r0, n1, r2, n;
    __device__ __forceinline__ int row(int k) const { return k < n1 ? r0 + k : r2 + (k - n1); }
};

// Shared memory of a CTA: the per-warp partials of a reduction, the CTA's totals (read by the other CTAs of a
// cluster; two sets alternate, since a CTA may form its next totals while another still reads these), the
// values handed to all threads.
struct UpShared {
    double part[UP_MAX_WARPS * 6];
    double total[2][6];
    double dval[6];
    float fval[6];
    int mask[2];
};

template <int G>
__device__ __forceinline__ bool leader()
{
    return G == G_WARP || threadIdx.x < 32;
}

// double(v), exact, on the integer pipe for normal values: a conversion takes as long as an FP64 operation
// (16 cycles of the SM for a warp): 192 sub-grids 49.3 -> 44.6 ms.
__device__ __forceinline__ double widen(float v)
{
    const unsigned u = __float_as_uint(v), e = u & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (u << 1) == 0u ? __hiloint2double(int(u), 0) : double(v);
    return __hiloint2double(int((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), int(u << 29));
}
__device__ __forceinline__ double widen(double v) { return v; }

__device__ __forceinline__ bool finite_bits(double v)
{
    return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
}

// Sums over the group: lane l of its leader warp(s) (the first warp of every CTA) gets sum l % 8.  FP32
// partials (the CG's dot products) are summed in FP32 within a warp and in FP64 across warps (eight lanes per
// chunk of the warps, then the chunks) and CTAs (in CTA order), so every leader of the group holds the same
// sums.  One warp adds them: a warp's FP64 instruction holds the SM's FP64 pipe for 16 cycles (a warp issues
// one in 64), and each of 32 warps adding all partials and forming all scalars of the CG cost an iteration 10
// to 20 us.
template <int G, int NV, class T>
__device__ __forceinline__ double group_sum(const T (&v)[NV], UpShared* sh, int& rb)
{
    const int lane = threadIdx.x & 31, i = lane & 7;
    T w[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        w[k] = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w[k] += __shfl_xor_sync(FULL, w[k], o);
    }
    double s = 0.0;
    if constexpr (G == G_WARP) {
        T mine = w[0];
#pragma unroll
        for (int k = 1; k < NV; ++k)
            if (i == k) mine = w[k];
        s = widen(mine);
        __syncwarp();
    } else {
        T* buf = reinterpret_cast<T*>(sh->part);
        const int wi = threadIdx.x >> 5, nw = blockDim.x >> 5;
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < NV; ++k) buf[k * UP_MAX_WARPS + wi] = w[k];
        __syncthreads();
        if (wi == 0) {
            const int c0 = (lane >> 3) * (nw >> 2);   // 8, 16 or 32 warps
            if (i < NV)
                for (int c = c0; c < c0 + (nw >> 2); ++c) s += widen(buf[i * UP_MAX_WARPS + c]);
            __syncwarp();
            s += __shfl_xor_sync(FULL, s, 8);
            s += __shfl_xor_sync(FULL, s, 16);
        }
        if constexpr (G == G_CLUSTER) {
            cg::cluster_group cl = cg::this_cluster();
            double* tot = sh->total[rb];
            rb ^= 1;
            if (threadIdx.x < NV) tot[threadIdx.x] = s;
            cl.sync();
            if (wi == 0) {
                const int nc = int(cl.num_blocks());
                s = 0.0;
                if (i < NV)
                    for (int c = 0; c < nc; ++c) s += cl.map_shared_rank(tot, c)[i];
                __syncwarp();
            }
        }
    }
    return s;
}

// What the leader's lanes 0 .. 2 hold for the three directions, to all threads of the group: put() by the
// leader, then publish() by all, then get().
template <int G, class T>
__device__ __forceinline__ void get3(T v, const T* slot, T (&out)[3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d] = G == G_WARP ? __shfl_sync(FULL, v, d) : slot[d];
}
template <int G, class T>
__device__ __forceinline__ void put3(T v, T* slot)
{
    if (G != G_WARP && threadIdx.x < 3) slot[threadIdx.x] = v;
}
template <int G>
__device__ __forceinline__ void publish()
{
    if (G != G_WARP) __syncthreads();
}
// a bit per direction
template <int G>
__device__ __forceinline__ void put_mask(bool b, int& mine, int* slot)
{
    mine = int(__ballot_sync(FULL, b) & 7u);
    if (G != G_WARP && threadIdx.x == 0) *slot = mine;
}
__device__ __forceinline__ void bits(int m, bool (&b)[3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) b[d] = (m >> d) & 1;
}
template <int G>
__device__ __forceinline__ void group_sync()
{
    if constexpr (G == G_CLUSTER) cg::this_cluster().sync();
    else if constexpr (G == G_CTA) __syncthreads();
    else __syncwarp();
}

// Position of direction d of unknown i in the three-direction vectors: side by side (L = 0,
// 3 i + d: one run per gathered column) or direction-major (L = 1, d n + i: every streamed access
// of a warp is one contiguous run).  The autotuner tries both; they measured within a few per cent
// of each other, either ahead.  Padding all of them to four values measured no faster; the direction p, which
// is gathered, has that layout of its own (ldp).
template <int L>
__device__ __forceinline__ size_t vix(int i, int d, int n)
{
    return L == 0 ? 3 * size_t(i) + d : size_t(d) * size_t(n) + i;
}

// The three values of unknown i, per direction: masked-off directions are neither loaded (read as
// 0) nor stored.  The vectors are written by this kernel (by other CTAs of a cluster, too), so
// their pointers carry no __restrict__: the loads stay ordinary coherent loads, ordered by the
// group's barriers, never the read-only path.
template <int L, class T>
__device__ __forceinline__ void ld3(const T* v, int i, int n, const bool (&m)[3], T (&o)[3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d) o[d] = m[d] ? v[vix<L>(i, d, n)] : T(0);
}
template <int L, class T>
__device__ __forceinline__ void st3(T* v, int i, int n, const bool (&m)[3], const T (&x)[3])
{
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (m[d]) v[vix<L>(i, d, n)] = x[d];
}

// The direction p: four values side by side, the last one unused, so that a gather is one 16-byte load (three
// 4-byte ones at a stride of 12 took twice the passes through the L1).
__device__ __forceinline__ void ldp(const float4* p, int i, float (&o)[3])
{
    const float4 v = p[i];
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
}
__device__ __forceinline__ void stp(float4* p, int i, const float (&x)[3]) { p[i] = make_float4(x[0], x[1], x[2], 0.f); }

// the three values of unknown i of a gathered vector
template <int L>
__device__ __forceinline__ void gather3(const float4* y, int i, int, float (&o)[3])
{
    ldp(y, i, o);
}
template <int L>
__device__ __forceinline__ void gather3(const double* y, int i, int n, double (&o)[3])
{
    constexpr bool all[3] = {true, true, true};
    ld3<L>(y, i, n, all, o);
}

// q = (A y)_r for the three directions (values TV, vector TX, sums TA): the row's SELL-32
// entries read once, two entries' loads in flight before their gathers; products added in entry
// order (padding adds exact zeros).
template <int L, class TA, class TV, class Y>
__device__ __forceinline__ void row_apply3(const int* __restrict__ sp, const int* __restrict__ col,
                                           const TV* __restrict__ val, const Y* y, int n, int r,
                                           TA (&q)[3])
{
    const int s = r >> 5;
    const int b = sp[s], w = (sp[s + 1] - b) >> 5;
    TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
    int k = b + (r & 31), t = 0;
    for (; t + 2 <= w; t += 2, k += 64) {
        const int c0 = col[k], c1 = col[k + 32];
        const TA v0 = TA(val[k]), v1 = TA(val[k + 32]);
        TA y0[3], y1[3];
        gather3<L>(y, c0, n, y0);
        gather3<L>(y, c1, n, y1);
        a0 += v0 * TA(y0[0]);
        a1 += v0 * TA(y0[1]);
        a2 += v0 * TA(y0[2]);
        a0 += v1 * TA(y1[0]);
        a1 += v1 * TA(y1[1]);
        a2 += v1 * TA(y1[2]);
    }
    if (t < w) {
        const int c0 = col[k];
        const TA v0 = TA(val[k]);
        TA y0[3];
        gather3<L>(y, c0, n, y0);
        a0 += v0 * TA(y0[0]);
        a1 += v0 * TA(y0[1]);
        a2 += v0 * TA(y0[2]);
    }
    q[0] = a0;
    q[1] = a1;
    q[2] = a2;
}

// The square of the residual norm, in units of sigma, below which the residual is replaced: dropped by delta,
// or the tolerance reached.
__device__ __forceinline__ double replace_below(const UpArgs& a, double sigma, double def0)
{
    const double l = fmax(a.delta, fmax(a.tol * def0, 1e-30) / sigma);
    return l * l;
}

// The CG of one sub-grid, three directions at once, by a group of nthr threads (tid = rank), with
// FP32 recurrences and reliable updates (residual replacement, Sleijpen and van der Vorst):
//   start   x = 0, sigma = ||b||, r = b / sigma (FP32), p = D^-1 r, rho = r.D^-1 r
//   pass A  q = A32 p (FP32), p.q
//   pass B  x += sigma alpha p (FP64), r -= alpha q; r.D^-1 r, r.r
//   when ||r|| has dropped below delta since the last replacement, or sigma ||r|| reaches the
//   tolerance: pass R, the true residual b - A x in FP64, which alone decides convergence; then
//   pass S, r = (b - A x) / sigma' and p *= sigma / sigma' (the recurrence continues in units of
//   the new sigma), r.D^-1 r again
//   pass C  p = D^-1 r + beta p
// x stays FP64 every iteration: an FP32 increment of x flushed at each replacement (measured) let
// one sub-grid of the 512-sub-grid batch stall at 3.3e-11 against a 1e-11 tolerance, its rounding
// times the condition number bounding the residual each replacement can reach.
// Each pass loads all of a row's values before it stores any, and frozen directions keep their
// values.  The leader's lanes 0 .. 2 keep the per-direction iteration count and reduction in global memory.
// What bounds it (an iteration on 15,606 unknowns by a cluster of two CTAs, 60 us, in thousands of cycles): pass A 59,
// streaming the matrix (the sub-grids at work together exceed the L2; twice as many loads in flight changed
// nothing), pass B 30, the FP64 pipe, pass C 8, the sums, scalars and barriers 27 (53 before one warp did them).
// 192 sub-grids of 5 to 17 cells a side: 86 ms with all threads adding all partials and converting p by FP64
// instructions, 58.5 with one warp's sums, 48 with p as float4 and converted by integers, 44 to 50 with
// clusters of four.  Measured and dropped: r and q in shared memory (64 ms, less L1 for the gathers), x brought up
// to date every second iteration or under pass A (62), six entries a row in flight on 512 threads (65).
template <int G, int L>
__device__ void solve_one(const UpArgs& a, int g, int tid, int nthr, UpShared* sh)
{
    constexpr bool all[3] = {true, true, true};
    const int* rg = a.ranges + 4 * g;
    const Rows R{rg[0], rg[1] - rg[0], rg[2], (rg[1] - rg[0]) + (rg[3] - rg[2])};
    const int n = a.n;
    // the iterations of a solve grow like the side of its sub-grid: so do a trial's
    const int maxit = a.trial > 0 ? max(1, int(float(a.maxit) * cbrtf(float(R.n) / float(a.trial)))) : a.maxit;
    const int dir = min(int(threadIdx.x & 31), 2);   // the direction whose scalars this lane of the leader keeps
    double* const dv0 = G == G_WARP ? nullptr : sh->dval;
    float *const fv0 = G == G_WARP ? nullptr : sh->fval, *const fv1 = G == G_WARP ? nullptr : sh->fval + 3;
    int* const mk = G == G_WARP ? nullptr : sh->mask;
    int rb = 0;
    bool bad = false;
    double v[3] = {0.0, 0.0, 0.0}, sum;
    for (int k = tid; k < R.n; k += nthr) {
        const int r = R.row(k);
        double b[3];
        ld3<0>(a.b3, r, n, all, b);   // right-hand sides: side by side
        const double di = a.val[a.diag[r]];
        bad |= !(di > 0.0);
        a.dinv[r] = float(1.0 / di);
        const double z3[3] = {0.0, 0.0, 0.0};
        st3<L>(a.x3, r, n, all, z3);
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] += b[d] * b[d];
    }
    if (bad) atomicOr(a.status, ST_NONFINITE);
    sum = group_sum<G, 3>(v, sh, rb);
    // the leader's: sigma, ||b||, r.D^-1 r, r.r that asks for a replacement, of direction dir
    double sigma = 0.0, def0 = 0.0, rho = 0.0, limit2 = 0.0;
    bool on = false, brk = false;
    int m = 0;   // directions still iterating
    if (leader<G>()) {
        def0 = sigma = sqrt(__shfl_sync(FULL, sum, dir));
        const bool fin = isfinite(def0);
        brk = !fin;
        on = fin && !(def0 < 1e-30);
        limit2 = on ? replace_below(a, sigma, def0) : 0.0;
        if (tid < 3) {
            a.iters[3 * g + tid] = fin ? (on ? -1 : 0) : -1;
            a.red[3 * g + tid] = on ? 1.0 : 0.0;
        }
        put3<G>(sigma, dv0);
        put_mask<G>(on, m, mk);
    }
    publish<G>();
    {
        double sig[3];
        get3<G>(sigma, dv0, sig);
        if (G != G_WARP) m = mk[0];
        bool act[3];
        bits(m, act);
        float u[3] = {0.f, 0.f, 0.f};
        for (int k = tid; k < R.n; k += nthr) {
            const int r = R.row(k);
            double b[3];
            ld3<0>(a.b3, r, n, all, b);
            const float dv = a.dinv[r];
            float rr[3], pp[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                rr[d] = act[d] ? float(b[d] / sig[d]) : 0.f;
                pp[d] = dv * rr[d];
                u[d] += rr[d] * pp[d];
            }
            st3<L>(a.r32, r, n, all, rr);
            stp(a.p4, r, pp);
        }
        sum = group_sum<G, 3>(u, sh, rb);
        if (leader<G>()) rho = __shfl_sync(FULL, sum, dir);
        publish<G>();   // the leader has read the partials
    }
    int it = 0;
    while (m && it < maxit) {
        ++it;
        // pass A: q = A32 p, p.q
        {
            float w[3] = {0.f, 0.f, 0.f};
            for (int k = tid; k < R.n; k += nthr) {
                const int r = R.row(k);
                float p[3], q[3];
                ldp(a.p4, r, p);
                row_apply3<L, float>(a.sp, a.col, a.val32, a.p4, n, r, q);
                st3<L>(a.q32, r, n, all, q);
#pragma unroll
                for (int d = 0; d < 3; ++d) w[d] += p[d] * q[d];
            }
            sum = group_sum<G, 3>(w, sh, rb);
        }
        double alpha = 0.0;
        if (leader<G>()) {
            const double c = __shfl_sync(FULL, sum, dir);
            if (on && !(c > 0.0 && finite_bits(c))) {   // non-positive curvature: stop
                on = false;
                brk = true;
            }
            alpha = on ? rho / c : 0.0;
            put3<G>(sigma * alpha, dv0);
            put3<G>(float(alpha), fv0);
            put_mask<G>(on, m, mk);
        }
        publish<G>();
        // pass B: x += sigma alpha p, r -= alpha q; r.D^-1 r, r.r
        double u = 0.0;       // r.D^-1 r (leader)
        bool again = false;   // this direction replaces its residual (leader)
        int mrep = 0;
        float beta = 0.f;
        {
            double sa[3];
            float al[3];
            get3<G>(sigma * alpha, dv0, sa);
            get3<G>(float(alpha), fv0, al);
            if (G != G_WARP) m = mk[0];
            bool act[3];
            bits(m, act);
            float part[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int k = tid; k < R.n; k += nthr) {
                const int r = R.row(k);
                const float dv = a.dinv[r];
                double x[3];
                float p[3], rr[3], q[3];
                ld3<L>(a.x3, r, n, act, x);
                ldp(a.p4, r, p);
                ld3<L>(a.r32, r, n, act, rr);
                ld3<L>(a.q32, r, n, act, q);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (act[d]) {
                        const float rn = rr[d] - al[d] * q[d];
                        x[d] += sa[d] * widen(p[d]);
                        rr[d] = rn;
                        part[d] += rn * (dv * rn);
                        part[3 + d] += rn * rn;
                    }
                st3<L>(a.x3, r, n, act, x);
                st3<L>(a.r32, r, n, act, rr);
            }
            sum = group_sum<G, 6>(part, sh, rb);
            if (leader<G>()) {
                // reliable update: which directions replace their residual
                u = __shfl_sync(FULL, sum, dir);
                const double ratio = u / rho, rr2 = __shfl_sync(FULL, sum, 3 + dir);
                again = on && (rr2 < limit2 || !finite_bits(rr2) || it >= maxit);
                put_mask<G>(again, mrep, mk + 1);
                if (mrep == 0) {
                    if (on && !finite_bits(u)) {
                        on = false;
                        brk = true;
                    }
                    beta = on ? float(ratio) : 0.f;
                    rho = u;
                    put3<G>(beta, fv0);
                    put_mask<G>(on, m, mk);
                }
            }
        }
        publish<G>();
        if (G != G_WARP) mrep = mk[1];
        if (mrep) {
            // pass R: the true residual b - A x (FP64) of the replacing directions
            bool rep[3];
            bits(mrep, rep);
            double t2[3] = {0.0, 0.0, 0.0};
            for (int k = tid; k < R.n; k += nthr) {
                const int r = R.row(k);
                double ax[3], b[3], t[3];
                row_apply3<L, double>(a.sp, a.col, a.val, a.x3, n, r, ax);
                ld3<0>(a.b3, r, n, all, b);
                ld3<L>(a.r64, r, n, rep, t);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (rep[d]) {
                        t[d] = b[d] - ax[d];
                        t2[d] += t[d] * t[d];
                    }
                st3<L>(a.r64, r, n, rep, t);
            }
            sum = group_sum<G, 3>(t2, sh, rb);
            float fac = 1.f;
            bool scaled = false;
            int mres = 0;
            if (leader<G>()) {
                const double dd = sqrt(__shfl_sync(FULL, sum, dir));
                if (again) {
                    if (tid < 3) a.red[3 * g + tid] = dd / def0;
                    if (!isfinite(dd)) {
                        on = false;
                        brk = true;
                    } else if (dd < a.tol * def0 || dd < 1e-30) {
                        on = false;
                        if (tid < 3) a.iters[3 * g + tid] = it;
                    } else if (it >= maxit) {
                        on = false;
                    } else {
                        const double f = sigma / dd;
                        fac = float(f);
                        rho *= f * f;
                        sigma = dd;
                        limit2 = replace_below(a, sigma, def0);
                        scaled = true;
                    }
                }
                put3<G>(sigma, dv0);
                put3<G>(fac, fv1);
                put_mask<G>(scaled, mres, mk + 1);
            }
            publish<G>();
            double sig[3];
            float fc[3];
            get3<G>(sigma, dv0, sig);
            get3<G>(fac, fv1, fc);
            if (G != G_WARP) mres = mk[1];
            if (mres) {
                // pass S: r = r_true / sigma, p in units of the new sigma; r.D^-1 r of the new r
                bool resc[3];
                bits(mres, resc);
                float uu[3] = {0.f, 0.f, 0.f};
                for (int k = tid; k < R.n; k += nthr) {
                    const int r = R.row(k);
                    const float dv = a.dinv[r];
                    double t[3];
                    float p[3], rr[3];
                    ld3<L>(a.r64, r, n, resc, t);
                    ldp(a.p4, r, p);
                    ld3<L>(a.r32, r, n, resc, rr);
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        if (resc[d]) {
                            rr[d] = float(t[d] / sig[d]);
                            p[d] *= fc[d];
                            uu[d] += rr[d] * (dv * rr[d]);
                        }
                    st3<L>(a.r32, r, n, resc, rr);
                    stp(a.p4, r, p);
                }
                sum = group_sum<G, 3>(uu, sh, rb);
                if (leader<G>()) {
                    const double un = __shfl_sync(FULL, sum, dir);
                    if (scaled) u = un;
                }
            }
            if (leader<G>()) {
                if (on && !finite_bits(u)) {
                    on = false;
                    brk = true;
                }
                beta = on ? float(u / rho) : 0.f;
                rho = u;
                put3<G>(beta, fv0);
                put_mask<G>(on, m, mk);
            }
            publish<G>();
        }
        if (G != G_WARP) m = mk[0];
        if (!m) break;
        // pass C: p = D^-1 r + beta p
        float be[3];
        get3<G>(beta, fv0, be);
        bool act[3];
        bits(m, act);
        for (int k = tid; k < R.n; k += nthr) {
            const int r = R.row(k);
            const float dv = a.dinv[r];
            float p[3], rr[3];
            ldp(a.p4, r, p);
            ld3<L>(a.r32, r, n, act, rr);
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if (act[d]) p[d] = dv * rr[d] + be[d] * p[d];
            stp(a.p4, r, p);
        }
        group_sync<G>();
    }
    if (brk && tid < 3) atomicOr(a.status, ST_BREAKDOWN);
}

// The persistent kernel: cluster items while any is left (rank 0 of the cluster takes the next
// one and the other CTAs read it from rank 0's shared memory), then CTA items (each CTA takes the
// next one), then warp items (each warp on its own).  Every loop ends: the counters only grow, and
// each CG is bounded by maxit.  Every cluster barrier is reached by all CTAs of the cluster: the
// item and every sum that steers the CG are the same in all of them.  After its last cluster
// item a CTA passes two more cluster barriers, so no CTA reads another's shared memory once any has
// moved on (or exited).
template <int L, bool CLUSTER>
__global__ void __launch_bounds__(UP_MAX_THREADS, 1) k_upscale_persistent(const UpArgs a)
{
    __shared__ UpShared sh;
    __shared__ int s_item;
    if constexpr (CLUSTER) {
        cg::cluster_group cl = cg::this_cluster();
        const int crank = int(cl.block_rank()), csize = int(cl.num_blocks());
        for (;;) {
            if (crank == 0 && threadIdx.x == 0) s_item = atomicAdd(a.counters, 1);
            cl.sync();
            const int item = *cl.map_shared_rank(&s_item, 0);
            cl.sync();   // every CTA has read rank 0's s_item before it is written again
            if (item >= a.ncl) break;
            solve_one<G_CLUSTER, L>(a, a.order[item], crank * int(blockDim.x) + int(threadIdx.x),
                                    csize * int(blockDim.x), &sh);
        }
    }
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(a.counters + 1, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();   // every thread has read s_item before thread 0 writes it again
        if (item >= a.ntile) break;
        solve_one<G_CTA, L>(a, a.order[a.ncl + item], threadIdx.x, blockDim.x, &sh);
    }
    const int lane = threadIdx.x & 31;
    const int first = a.ncl + a.ntile, nwarp = a.nitems - first;
    for (;;) {
        int item = 0;
        if (lane == 0) item = atomicAdd(a.counters + 2, 1);
        item = __shfl_sync(FULL, item, 0);
        if (item >= nwarp) break;
        solve_one<G_WARP, L>(a, a.order[first + item], lane, 32, nullptr);
    }
}

__global__ void k_put3(int n, const double* __restrict__ v, double* __restrict__ v3, int d)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v3[3 * size_t(i) + d] = v[i];
}

__global__ void k_get3(int n, const double* __restrict__ v3, double* __restrict__ v, int d, int layout)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = layout == 0 ? v3[3 * size_t(i) + d] : v3[size_t(d) * size_t(n) + i];
}

__global__ void k_fill(int n, double value, double* __restrict__ v)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = value;
}

__global__ void k_jump_values(int nhf, const int* __restrict__ side, int d, double* __restrict__ bcv)
{
    const int hf = blockIdx.x * blockDim.x + threadIdx.x;
    if (hf >= nhf) return;
    const int sd = side[hf];
    bcv[hf] = sd == 2 * d + 1 ? 1.0 : (sd == 2 * d + 2 ? -1.0 : 0.0);
}

// Autotuner choices, per batch shape (sub-grid count, log2 of the unknowns, log2 of the largest
// sub-grid's unknowns), for the life of the process.
std::mutex& tune_mutex()
{
    static std::mutex m;
    return m;
}
std::unordered_map<long long, UpscaleSchedule>& tune_cache()
{
    static std::unordered_map<long long, UpscaleSchedule> c;
    return c;
}

int ilog2(long long v)
{
    int l = 0;
    while ((2LL << l) <= v) ++l;
    return l;
}

}  // namespace

void launch_put3(cudaStream_t s, int n, const double* v, double* v3, int d)
{
    if (n <= 0) return;
    PORSOL_LAUNCH(k_put3<<<div_up(n, 256), 256, 0, s>>>(n, v, v3, d));
    PORSOL_CUDA(cudaGetLastError());
}

void launch_get3(cudaStream_t s, int n, const double* v3, double* v, int d, int layout)
{
    if (n <= 0) return;
    PORSOL_LAUNCH(k_get3<<<div_up(n, 256), 256, 0, s>>>(n, v3, v, d, layout));
    PORSOL_CUDA(cudaGetLastError());
}

void launch_fill(cudaStream_t s, int n, double value, double* v)
{
    if (n <= 0) return;
    PORSOL_LAUNCH(k_fill<<<div_up(n, 256), 256, 0, s>>>(n, value, v));
    PORSOL_CUDA(cudaGetLastError());
}

void launch_jump_values(cudaStream_t s, int nhf, const int* side, int d, double* bcv)
{
    if (nhf <= 0) return;
    PORSOL_LAUNCH(k_jump_values<<<div_up(nhf, 256), 256, 0, s>>>(nhf, side, d, bcv));
    PORSOL_CUDA(cudaGetLastError());
}

PersistentUpscale::~PersistentUpscale()
{
    if (exec_) cudaGraphExecDestroy(exec_);
}

void PersistentUpscale::item_classes(const std::vector<int>& rg, const UpscaleSchedule& sc, int& ncl, int& ntile) const
{
    ncl = ntile = 0;
    for (int g : order_h_) {
        const int n = (rg[4 * size_t(g) + 1] - rg[4 * size_t(g)]) + (rg[4 * size_t(g) + 3] - rg[4 * size_t(g) + 2]);
        if (sc.cluster > 1 && n >= sc.cluster_min_unknowns) ++ncl;
        else if (n >= sc.warp_max_unknowns) ++ntile;
    }
}

void PersistentUpscale::launch(cudaStream_t s, const SellPattern& P, const double* val, const float* val32,
                               const int* ranges_d, const double* b3, double* x3, double tol, double delta, int maxit,
                               const UpscaleSchedule& sc, bool graph, int trial)
{
    UpArgs a;
    std::memset(&a, 0, sizeof(a));
    a.nitems = nblk_;
    item_classes(rg_h_, sc, a.ncl, a.ntile);
    a.n = n_;
    a.maxit = maxit;
    a.trial = trial;
    a.tol = tol;
    a.delta = delta;
    a.order = order_.p;
    a.ranges = ranges_d;
    a.sp = P.slice_ptr.p;
    a.col = P.col.p;
    a.val = val;
    a.val32 = val32;
    a.diag = P.diag.p;
    a.b3 = b3;
    a.x3 = x3;
    a.r64 = r64_.p;
    a.r32 = r32_.p;
    a.p4 = reinterpret_cast<float4*>(p32_.p);
    a.q32 = q32_.p;
    a.dinv = dinv_.p;
    a.iters = iters_.p;
    a.red = red_.p;
    a.counters = counters_.p;
    a.status = status_.p;
    const bool cl = sc.cluster > 1;
    void (*kern)(const UpArgs) = sc.layout == 0 ? (cl ? k_upscale_persistent<0, true> : k_upscale_persistent<0, false>)
                                                : (cl ? k_upscale_persistent<1, true> : k_upscale_persistent<1, false>);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(unsigned(sc.cta_threads));
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    int grid = 1;
    if (cl) {
        // as many clusters as can be resident at once (each CTA fills its SM)
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = unsigned(sc.cluster);
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(unsigned(sc.cluster));
        int nclusters = 0;
        PORSOL_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg));
        PORSOL_REQUIRE(nclusters > 0, PORSOL_ERR_BAD_ARG, "persistent upscaling: cluster schedule cannot be resident");
        grid = nclusters * sc.cluster;
    } else {
        int dev = 0, sms = 0, per = 0;
        PORSOL_CUDA(cudaGetDevice(&dev));
        PORSOL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        PORSOL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, sc.cta_threads, 0));
        grid = std::max(1, sms * std::max(per, 1));
        cfg.attrs = nullptr;
        cfg.numAttrs = 0;
    }
    cfg.gridDim = dim3(unsigned(grid));
    auto enqueue = [&] {
        PORSOL_CUDA(cudaMemsetAsync(counters_.p, 0, 3 * sizeof(int), s));
        PORSOL_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
        PORSOL_COUNT_LAUNCH();
        PORSOL_CUDA(cudaGetLastError());
    };
    if (!graph) {
        enqueue();
        return;
    }
    // the launch (with the queue reset) as a captured graph, rebuilt when an argument changes
    std::vector<unsigned char> key(sizeof(a) + 4 * sizeof(int));
    std::memcpy(key.data(), &a, sizeof(a));
    std::memcpy(key.data() + sizeof(a), &grid, sizeof(int));
    std::memcpy(key.data() + sizeof(a) + sizeof(int), &sc.cta_threads, sizeof(int));
    std::memcpy(key.data() + sizeof(a) + 2 * sizeof(int), &sc.layout, sizeof(int));
    std::memcpy(key.data() + sizeof(a) + 3 * sizeof(int), &sc.cluster, sizeof(int));
    if (!exec_ || key != exec_key_) {
        if (exec_) PORSOL_CUDA(cudaGraphExecDestroy(exec_));
        exec_ = nullptr;
        cudaGraph_t gr;
        const long long l0 = g_launches.load();
        PORSOL_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        enqueue();
        PORSOL_CUDA(cudaStreamEndCapture(s, &gr));
        g_launches.fetch_sub(g_launches.load() - l0);
        PORSOL_CUDA(cudaGraphInstantiate(&exec_, gr, 0));
        PORSOL_CUDA(cudaGraphDestroy(gr));
        exec_key_ = key;
    }
    PORSOL_CUDA(cudaGraphLaunch(exec_, s));
    PORSOL_COUNT_LAUNCH();
}

// Candidate schedules: CTAs of 512 or 1024 threads for the CTA items (256-thread CTAs always measured slower on
// the 512-sub-grid batch) and the sub-grids of at least half the largest one's unknowns solved by clusters of 1
// (none), 2 or 4 CTAs; then, with the fastest of these, sub-grids below 4096 unknowns (sides up to about 11 in the
// unit-cube batches) left to single warps, and the other vector layout.  Each runs TUNE_ITERS iterations of the
// largest sub-grid, of the others fewer in proportion to their sides, as whole solves do, after one warm-up launch;
// the fastest is kept for the batch shape.  A cluster shape that cannot be resident on this GPU is skipped.
// Trials of few iterations misjudge: their start and last replacement weigh more than in a solve, most for the
// small sub-grids.  192 sub-grids of 5 to 17 cells a side: 48 weighted iterations take clusters of 4 and 1024
// threads, 44.6 ms, 16 take 512 threads, 49.3, eight of each took clusters of 2, 49.7; 512 of 8 to 32: 48 take
// clusters of 2, 922 ms, or none, 1035 (a tie in the trials), 12 to 32 always none.  All combinations of the four
// choices, 14 to 24 trials, picked none faster, and a batch solved once paid for them: first call on 128
// sub-grids of 8 to 32 cells a side 1.65 s, with these eight 1.13.
UpscaleSchedule PersistentUpscale::tune(cudaStream_t s, const SellPattern& P, const double* val, const float* val32,
                                        const std::vector<int>& rg, const int* ranges_d, const double* b3, double* x3)
{
    long long total = 0, largest = 0;
    for (int g = 0; g < nblk_; ++g) {
        const long long n = (rg[4 * size_t(g) + 1] - rg[4 * size_t(g)]) + (rg[4 * size_t(g) + 3] - rg[4 * size_t(g) + 2]);
        total += n;
        largest = std::max(largest, n);
    }
    const long long key = ((long long)nblk_ << 16) | ((long long)ilog2(std::max(total, 1LL)) << 8) |
                          (long long)ilog2(std::max(largest, 1LL));
    {
        std::lock_guard<std::mutex> lk(tune_mutex());
        auto it = tune_cache().find(key);
        if (it != tune_cache().end()) return it->second;
    }
    static const bool debug = std::getenv("PORSOL_DEBUG_UPSCALE") != nullptr;
    cudaEvent_t e0, e1;
    PORSOL_CUDA(cudaEventCreate(&e0));
    PORSOL_CUDA(cudaEventCreate(&e1));
    UpscaleSchedule best;
    float best_ms = 1e30f;
    bool warmed = false;
    auto trial = [&](const UpscaleSchedule& c) {
        auto run = [&] { launch(s, P, val, val32, ranges_d, b3, x3, 0.0, 0.0, TUNE_ITERS, c, false, int(largest)); };
        try {
            if (!warmed) run();
            warmed = true;
            PORSOL_CUDA(cudaEventRecord(e0, s));
            run();
        } catch (const Error& e) {
            if (e.code != PORSOL_ERR_BAD_ARG) throw;
            return;   // cluster shape not resident here
        }
        PORSOL_CUDA(cudaEventRecord(e1, s));
        PORSOL_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        PORSOL_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (debug)
            std::fprintf(stderr, "[upscale] trial cluster=%d layout=%d cta=%d warp_below=%d: %.3f ms\n", c.cluster, c.layout,
                         c.cta_threads, c.warp_max_unknowns, ms);
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    };
    try {
        for (int cluster : {1, 2, 4})
            for (int threads : {512, 1024}) {
                UpscaleSchedule c;
                c.cta_threads = threads;
                c.cluster = cluster;
                c.cluster_min_unknowns = cluster > 1 ? int(largest / 2) : 0;
                c.tuned = true;
                trial(c);
            }
        UpscaleSchedule c = best;
        c.warp_max_unknowns = 4096;
        trial(c);
        c = best;
        c.layout = 0;
        trial(c);
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    PORSOL_REQUIRE(best_ms < 1e30f, PORSOL_ERR_CUDA, "persistent upscaling: no schedule could be launched");
    std::lock_guard<std::mutex> lk(tune_mutex());
    tune_cache()[key] = best;
    return best;
}

UpscaleResult PersistentUpscale::solve(cudaStream_t s, const SellPattern& P, const double* val, const float* val32,
                                       const std::vector<int>& rg, const int* ranges_d, const double* b3, double* x3,
                                       double tol, double delta, int maxit, const UpscaleSchedule& fixed)
{
    PORSOL_REQUIRE(rg.size() % 4 == 0 && !rg.empty(), PORSOL_ERR_BAD_ARG, "persistent upscaling: no sub-grids");
    PORSOL_REQUIRE(P.n <= INT_MAX / 3, PORSOL_ERR_BAD_ARG, "persistent upscaling: too many unknowns");
    PORSOL_REQUIRE(fixed.layout == 0 || fixed.layout == 1, PORSOL_ERR_BAD_ARG,
                   "persistent upscaling: vector layout must be 0 or 1");
    PORSOL_REQUIRE(fixed.cluster == 1 || fixed.cluster == 2 || fixed.cluster == 4, PORSOL_ERR_BAD_ARG,
                   "persistent upscaling: cluster size must be 1, 2 or 4");
    PORSOL_REQUIRE(fixed.cta_threads == 0 || fixed.cta_threads == 256 || fixed.cta_threads == 512 ||
                       fixed.cta_threads == 1024,
                   PORSOL_ERR_BAD_ARG, "persistent upscaling: CTA threads must be 256, 512 or 1024");
    n_ = P.n;
    nblk_ = int(rg.size() / 4);
    r64_.alloc(3 * size_t(n_));
    r32_.alloc(3 * size_t(n_));
    p32_.alloc(4 * size_t(n_));   // float4 per unknown
    q32_.alloc(3 * size_t(n_));
    dinv_.alloc(size_t(n_));
    red_.alloc(3 * size_t(nblk_));
    iters_.alloc(3 * size_t(nblk_));
    counters_.alloc(3);
    rg_h_ = rg;
    status_.alloc(1);
    // largest sub-grids first (ties by index): the cluster items, the CTA items, then the warp items,
    // each in decreasing size, so the longest solves start first
    std::vector<int> nrow(static_cast<size_t>(nblk_));
    for (int g = 0; g < nblk_; ++g)
        nrow[size_t(g)] = (rg[4 * size_t(g) + 1] - rg[4 * size_t(g)]) + (rg[4 * size_t(g) + 3] - rg[4 * size_t(g) + 2]);
    order_h_.resize(size_t(nblk_));
    std::iota(order_h_.begin(), order_h_.end(), 0);
    std::stable_sort(order_h_.begin(), order_h_.end(),
                     [&](int x, int y) { return nrow[size_t(x)] > nrow[size_t(y)]; });
    order_.upload(order_h_, s);
    status_.zero(s);
    sched_ = fixed.cta_threads ? fixed : tune(s, P, val, val32, rg, ranges_d, b3, x3);
    if (fixed.cta_threads) sched_.tuned = false;
    status_.zero(s);
    launch(s, P, val, val32, ranges_d, b3, x3, tol, delta, maxit, sched_, true, 0);
    std::vector<int> its(3 * size_t(nblk_));
    std::vector<double> red(3 * size_t(nblk_));
    int st = 0;
    iters_.download(its.data(), its.size(), s);
    red_.download(red.data(), red.size(), s);
    PORSOL_CUDA(cudaMemcpyAsync(&st, status_.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    PORSOL_CUDA(cudaStreamSynchronize(s));
    UpscaleResult res;
    res.converged = true;
    res.breakdown = (st & (ST_BREAKDOWN | ST_NONFINITE)) != 0;
    const double avg_entries = n_ > 0 ? double(P.nent) / n_ : 0.0;
    bytes_ = 0.0;
    for (int g = 0; g < nblk_; ++g) {
        int gi = 0;
        for (int d = 0; d < 3; ++d) {
            const int k = its[3 * size_t(g) + d];
            res.reduction = std::max(res.reduction, red[3 * size_t(g) + d]);
            if (k < 0) {
                res.converged = false;
                if (res.worst_block < 0) res.worst_block = g;
                gi = maxit;
            } else {
                gi = std::max(gi, k);
            }
        }
        res.iterations = std::max(res.iterations, gi);
        // start: diagonal and b twice, x, r, p; per iteration: stored entries (column 4 + FP32 value
        // 4), p gathered once, its own value read and q written (3 x 4 each), pass B (D^-1 4; x read
        // and written 16, p 4, r read and written 8, q 4 per direction) and pass C (D^-1 4; r 4, p
        // read and written 8 per direction); p's fourth, unused value and replacements are not counted
        const double n = nrow[size_t(g)];
        bytes_ += n * (12.0 + 48.0 + 3 * (8.0 + 4.0 + 4.0)) +
                  gi * n * (8.0 * avg_entries + 36.0 + 4.0 + 3 * 32.0 + 4.0 + 3 * 12.0);
    }
    return res;
}

}  // namespace porsol
