// match.cuh -- strengths and their order in the pairwise matching of the AMG setup.
#pragma once

#include "porsol_internal.h"

namespace porsol {

// Symmetric 32-bit hash of an edge {i, j}: equal strengths (common on uniform grids) are
// ordered by this pseudo-random priority, the same from both endpoints, so locally
// dominant edges are unique and mutual-best matching pairs most rows in a few sweeps.
__device__ __forceinline__ unsigned edge_hash(int i, int j)
{
    const unsigned lo = unsigned(min(i, j)), hi = unsigned(max(i, j));
    unsigned x = lo * 0x9E3779B1u + hi * 0x85EBCA77u;
    x ^= x >> 15;
    x *= 0x2C1B3C6Du;
    x ^= x >> 12;
    x *= 0x297A2D39u;
    x ^= x >> 15;
    return x;
}

// (s, hash) lexicographic comparison with the column as the last key
__device__ __forceinline__ bool stronger(float s, unsigned h, int j, float bs, unsigned bh, int bj)
{
    return s > bs || (s == bs && (h > bh || (h == bh && j < bj)));
}

// Entry (j, a) of row i as a candidate: kept when its neighbour has the wanted state, its strength
// s = a' rs_i rs_j (a' = -a for negative couplings, |a| otherwise) passes the floor, and it beats the
// best so far.  stronger() is a total order, so the best is the same whatever the order of the entries.
__device__ __forceinline__ void consider(int i, int j, float a, int stj, float rsj, float ri, int want_state,
                                         bool neg, float floor_s, float& bs, unsigned& bh, int& bj)
{
    if (j == i || stj != want_state) return;
    const float s = (neg ? -a : fabsf(a)) * ri * rsj;
    if (!(s > 0.0f && s >= floor_s)) return;
    const unsigned h = edge_hash(i, j);
    if (bj < 0 || stronger(s, h, j, bs, bh, bj)) {
        bs = s;
        bh = h;
        bj = j;
    }
}

// best candidate of K lanes: (strength, hash, column) is a strict total order over the distinct
// columns of a row, so the reduction gives the one-lane scan's answer in any lane order
template <int K>
__device__ __forceinline__ void best_of_lanes(float& bs, unsigned& bh, int& bj)
{
#pragma unroll
    for (int o = K >> 1; o > 0; o >>= 1) {
        const float s2 = __shfl_xor_sync(0xffffffffu, bs, o);
        const unsigned h2 = __shfl_xor_sync(0xffffffffu, bh, o);
        const int j2 = __shfl_xor_sync(0xffffffffu, bj, o);
        if (j2 >= 0 && (bj < 0 || stronger(s2, h2, j2, bs, bh, bj))) {
            bs = s2;
            bh = h2;
            bj = j2;
        }
    }
}

}  // namespace porsol
