// tail.h -- the smallest AMG levels of a V-cycle as one launch of a thread-block cluster.
//
// The last levels of the hierarchy (a few thousand rows down to the dense coarsest one) hold under a
// megabyte of matrix, and their kernels cost launch latencies and chains of dependent L2 loads, not
// bandwidth: seven launches per level and cycle at 3-6 us each.  Here one cluster of TAIL_CTAS blocks runs
// all of them.  Each block owns a contiguous part of every level's rows, with their matrix entries in its
// shared memory (copied in before the preceding kernel has finished), and every block holds the whole
// vector that the next product gathers: a row's new value is written to all blocks through distributed
// shared memory, and a cluster barrier separates the phases.  The arithmetic of a row is that of the
// per-level kernels, its entries summed in another order.
#pragma once

#include "porsol_internal.h"

namespace porsol {

constexpr int TAIL_CTAS = 8;
constexpr int TAIL_THREADS = 512;
constexpr int TAIL_LEVELS = 4;                     // smoothed levels in the tail at most
constexpr int TAIL_ROWS = 4096;                    // rows of its first level at most
constexpr int TAIL_BLOB = 160 * 1024;              // bytes of one level's part of one block at most
constexpr int TAIL_SMEM = 224 * 1024;
constexpr int TAIL_DENSE = 160;                    // rows of the dense level at most
// Unknowns of the system at most.  The tail adds a row's entries in another order than the per-level kernels,
// and what a solve to the tightest tolerances leaves in single fluxes of a strongly heterogeneous system follows
// every rounding of the cycle: at 3M unknowns in mixed precision by 1e-7 of their mean, for 1 to 3 % of a cycle
// saved (20 us of 800).  Measured on systems of 3M (not taken) and of up to 1.5M unknowns (taken: 5 to 13 % of an
// iteration); the limit lies between the two.
constexpr int TAIL_SYSTEM = 2 << 20;

// Part of one level that one block owns, as k_tail_pack writes it (offsets in bytes from its start; the
// first TailHead bytes are this header).
struct TailHead {
    int bytes;                 // total, a multiple of 16; > TAIL_BLOB: does not fit (nothing else is valid)
    int vals, cols, dinv, diag, agg, mptr, midx;
    int woff[TAIL_THREADS / 32], iters[TAIL_THREADS / 32];   // per warp: first entry and entries per lane
};

template <class T>
struct TailLevel {
    int n, lanes;              // rows, lanes per row
    int blob, f0, f1, bo;      // shared-memory offsets: the part, two whole vectors, own right-hand sides
    T inv_theta, c1[2], c2[2];
};

template <class T>
struct TailArgs {
    int levels;                // smoothed levels
    TailLevel<T> lv[TAIL_LEVELS];
    const unsigned char* blob; // [level][block][TAIL_BLOB]
    int part_bytes[TAIL_LEVELS];   // the largest block's part per level
    // the dense level
    int nd, db, dx, dinv;      // rows; shared-memory offsets: right-hand side, solution, own rows of the inverse
    const double* cinv;
    // restriction into the first level, its result
    const int *rptr, *ridx;
    const T* rfine;
    T* x;
    T wp;
    const int* stop;
};

// Rows of a level that block `rank` owns: [rank * per, min(n, (rank + 1) * per)).
__host__ __device__ inline int tail_per(int n) { return (n + TAIL_CTAS - 1) / TAIL_CTAS; }

// lanes per row: as many as keep the working threads at 256, two warps per scheduler (128, 256 and 512
// measured within 1 % in FP32; in FP64, where a warp instruction occupies the pipe for 64 clocks, 512 costs
// 3 % of an iteration)
constexpr int TAIL_LANE_THREADS = 256;
int tail_lanes(int n);

// One level's parts for all blocks.  h: FP16 D^-1 A (then dv, the diagonal, is used) or null, A: the matrix.
// nn, nptr, nidx: the next level's rows and member lists; all_members: every block gets all of them (dense).
template <class T>
void tail_pack(cudaStream_t s, int n, const int* sp, const int* col, const int* rowlen, const void* h, const T* A,
               const T* dinv, const T* dv, const int* agg, int nn, const int* nptr, const int* nidx, bool all_members,
               unsigned char* blob);

// Shared-memory layout of the levels [0, a.levels) and the dense one; returns the bytes (a's offsets are set).
template <class T>
int tail_layout(TailArgs<T>& a);

template <class T>
void tail_launch(cudaStream_t s, bool half, const TailArgs<T>& a, int shm);

// whether the device holds such a cluster
template <class T>
bool tail_fits(bool half);

}  // namespace porsol
