// rock.cuh -- rock tables (RockJfunc) evaluated on the device and on the host.
//
// Reference: RockJfunc::krw/kro/capPress/capPressDeriv/satFromCapPress
// (common/RockJfunc.hpp:63-141) and the per-cell dispatch of ReservoirPropertyCommon
// (common/ReservoirPropertyCommon_impl.hpp:466-528).  The tables are opm-core
// NonuniformTableLinear objects in the reference (that library is not part of the reference
// tree): here they are piecewise linear with the end value outside the table; the derivative is
// the slope of the interval holding the point (0 outside); the inverse of the J table
// interpolates s in J with the table read in increasing-J order (kept as a second copy, Jx/sy).
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#include "quotient.cuh"
#endif

namespace porsol {

struct RockView {
    int nrock = 0;                 // 0: no tables (kr1 = s^2, kr2 = (1-s)^2, pc = 1e5 (1-s))
    const int* pos = nullptr;      // [nrock + 1] row range of each rock
    const double* s = nullptr;     // saturations, non-decreasing per rock
    const double* krw = nullptr;
    const double* kro = nullptr;
    const double* J = nullptr;
    const double* Jx = nullptr;    // J in increasing order ...
    const double* sy = nullptr;    // ... with the matching saturations
    const int* cell = nullptr;     // rock of each cell
    const double* skp = nullptr;   // per cell sqrt(tr K / (3 phi)) (J scaling)
    int jscale = 1;
    double sct = 1.0;              // sigma cos(theta)
};

// interval [lo, lo + 1] of x (non-decreasing, n >= 2) with x[lo] <= v < x[lo + 1], for
// x[0] < v < x[n - 1]
__host__ __device__ inline int tab_interval(const double* x, int n, double v)
{
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (x[mid] <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

__host__ __device__ inline double tab_value(const double* x, const double* y, int n, double v)
{
    if (v <= x[0]) return y[0];
    if (v >= x[n - 1]) return y[n - 1];
    const int lo = tab_interval(x, n, v);
    const double w = (v - x[lo]) / (x[lo + 1] - x[lo]);
    return (1.0 - w) * y[lo] + w * y[lo + 1];
}

__host__ __device__ inline double tab_slope(const double* x, const double* y, int n, double v)
{
    if (n < 2 || v < x[0] || v > x[n - 1]) return 0.0;
    const int lo = v >= x[n - 1] ? n - 2 : tab_interval(x, n, v);
    return x[lo + 1] > x[lo] ? (y[lo + 1] - y[lo]) / (x[lo + 1] - x[lo]) : 0.0;
}

// relative permeability of phase 0 (krw) or 1 (kro) in cell c
__host__ __device__ inline double rock_kr(const RockView& R, int phase, int c, double s)
{
    const int r = R.cell[c], a = R.pos[r], n = R.pos[r + 1] - a;
    return tab_value(R.s + a, (phase == 0 ? R.krw : R.kro) + a, n, s);
}

// RockJfunc::capPress
__host__ __device__ inline double rock_pc(const RockView& R, int c, double s)
{
    const int r = R.cell[c], a = R.pos[r], n = R.pos[r + 1] - a;
    const double j = tab_value(R.s + a, R.J + a, n, s);
    return R.jscale ? j * R.sct / R.skp[c] : j;
}

// RockJfunc::satFromCapPress: inverse J curve, clamped to [s_min, s_max] of the rock
__host__ __device__ inline double rock_sat(const RockView& R, int c, double pc)
{
    const int r = R.cell[c], a = R.pos[r], n = R.pos[r + 1] - a;
    const double v = R.jscale ? pc * R.skp[c] / R.sct : pc;
    const double s = tab_value(R.Jx + a, R.sy + a, n, v);
    return fmin(R.s[a + n - 1], fmax(R.s[a], s));
}

// ---- the tables as the transport sub-steps read them ----
// GB300 issues two FP64 operations a clock and SM, so these kernels search the rows on the integer pipe
// and keep one subtraction and one FMA per value: saturations as ordered 64-bit keys, and 8 doubles per
// row: s, krw / mu1 and its slope to the next row, kro / mu2 and its slope, J and its slope, unused.
// The mobilities and pressures differ from rock_kr / rock_pc by rounding only.
struct RockTab {
    int nrock = 0;                    // 0: no tables
    const int* pos = nullptr;         // [nrock + 1]
    const long long* key = nullptr;   // tab_key(s) per row
    const double* node = nullptr;     // 8 per row
    const int* cell = nullptr;        // rock of each cell
    const double* pcs = nullptr;      // per cell factor from J to the capillary pressure
};

// 64-bit integers in the order of the doubles (-0 before +0, NaN outside)
__host__ __device__ inline long long tab_key(double v)
{
    long long b;
#ifdef __CUDA_ARCH__
    b = __double_as_longlong(v);
#else
    memcpy(&b, &v, sizeof(b));
#endif
    return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFll);
}

#ifdef __CUDACC__
// Row of rock r whose interval holds v, and v's distance from its start: 0 outside the table, where the
// end value holds (NaN for a NaN, which then reaches every value).
__device__ __forceinline__ const double* tab_row(const RockTab& R, int r, double v, double& dx)
{
    const int a = R.pos[r], e = R.pos[r + 1] - 1;
    const long long k = tab_key(v);
    int lo = a;
    const bool nan = ((unsigned long long)__double_as_longlong(v) << 1) > 0xFFE0000000000000ull;
    dx = nan ? v : 0.0;
    if (k >= R.key[e]) {
        lo = e;
        if (k <= R.key[a]) lo = a;
    } else if (k > R.key[a]) {
        int hi = e;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (R.key[mid] <= k) lo = mid;
            else hi = mid;
        }
        dx = v - R.node[8 * size_t(lo)];
    }
    return R.node + 8 * size_t(lo);
}
#endif

}  // namespace porsol
