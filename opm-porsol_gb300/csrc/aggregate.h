// aggregate.h -- one pairing round of the AMG setup as one launch of a thread-block cluster.
//
// A round of the launch-per-step path is 25 to 45 launches of a few microseconds (strengths, four or eight
// sweeps of picking and matching, joins, numbering, member lists, candidate offsets) and three reads back by
// the host.  On levels of up to AGG_ROWS rows, where those launches are latency, one cluster runs the
// whole round with cluster barriers between the steps; the arrays stay in L2, each block keeps the
// worklist of its own rows in shared memory, and the host reads three numbers.  From 55 us (300 rows) to
// 230-260 us (44k rows, about what the launches take there: the limit) a round; the whole setup of a 38k-unknown
// FP64 system went from 3.0 to 1.8 ms, of a 255k-unknown mixed one from 4.2 to 3.1 ms, of 3M unknowns from
// 11.5 to 10.7 ms.
#pragma once

#include "porsol_internal.h"

namespace porsol {

constexpr int AGG_CTAS = 16;         // blocks of a cluster at most
constexpr int AGG_THREADS = 1024;
constexpr int AGG_ROWS = 48 * 1024;
constexpr long long AGG_ENTRIES = 1LL << 20;
constexpr int AGG_SCRATCH = 3 + 4 * AGG_CTAS;   // results (aggregates, candidates, longest), block totals

inline bool agg_small(int n, long long nent) { return n <= AGG_ROWS && nent <= AGG_ENTRIES; }

template <class T>
struct AggArgs {
    int n;
    const int *sp, *col, *rowlen, *diag;
    const T* A;
    int neg_first;     // first the strong negative couplings, on all couplings with joins where that stalls
    float theta;
    // scratch of n (cnt, cidx: n + 1) values
    float* rs;
    int *state, *partner, *join, *best, *cidx, *cnt;
    // row -> aggregate, members (ptr n + 1, idx n), candidate offsets (goff n + 1, woff n)
    int *agg, *ptr, *idx, *goff, *woff;
    int* scratch;
};

// Both return false, with nothing launched, where the device holds no cluster of the size (of at most `limit`
// blocks) that the level needs; the caller then takes a launch per step.
template <class T>
bool agg_launch(cudaStream_t s, int lanes, const AggArgs<T>& a, int limit);

// agg1 = agg2 o agg1 (n rows onto nc aggregates) with member lists
bool compose_launch(cudaStream_t s, int n, int nc, int* agg1, const int* agg2, int* cnt, int* ptr, int* idx, int* scratch,
                    int limit);

}  // namespace porsol
