// batch.h -- preconditioned CG over block-diagonal systems, one independent CG per block.
//
// Batched periodic upscaling solves the disjoint union of many sub-grids as one system.  One
// CG over the union converges at the rate of its whole spectrum: every sub-grid contributes
// its own smallest eigenvalue (its regularised constant mode), so the union needs several times
// the iterations of its hardest sub-grid.  BatchedPcg runs the CG recurrences per block instead
// (per-block alpha, beta, residual norm and stopping test) while every kernel still sweeps the
// whole union: the iteration count is that of the slowest sub-grid.  The preconditioner must be
// block diagonal too (an AMG hierarchy of the union is: aggregates never cross sub-grids).
#pragma once

#include "amg.h"
#include "krylov.h"
#include "vec3.cuh"

namespace porsol {

// Block g owns the unknowns [r[4g], r[4g+1]) and [r[4g+2], r[4g+3]) (the internal and the
// boundary face unknowns of a sub-grid are each numbered contiguously).
struct BatchRanges {
    int nblk = 0, n = 0;
    std::vector<int> h;
    DBuf<int> ranges, blk;
    // the unknowns in chunks of at most CHUNK of one block, block by block: (first unknown, unknowns,
    // block, -), and each block's range of chunks
    static constexpr int CHUNK = 2048;
    int nchunks = 0;
    DBuf<int4> chunks;
    DBuf<int> cptr;
    void build(const std::vector<int>& four_per_block, int n_unknowns, cudaStream_t s);
};

// Global state of a batched solve (device), mirrored for the host in mapped memory.
struct BatchDev {
    int iter, maxit, stop, active, breakdown, pad;
};
struct BatchHostView {
    volatile int iter, stop, active, breakdown;
};

template <class TV, class T>
class BatchedPcg {
public:
    // x holds the initial guess.  tol[g] (device, per block): stop block g when
    // ||r_g|| < tol[g] ||r_g^0|| or ||r_g|| < 1e-30.  On return def0/def (device, per block)
    // hold the initial and final residual norms.
    CgResult solve(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, const BatchRanges& B,
                   const T* b, T* x, const double* tol, int maxit);
    const double* def0() const { return def0_.p; }
    const double* def() const { return def_.p; }
    ~BatchedPcg();

private:
    int n_ = 0, nblk_ = 0;
    DBuf<T> r_, z_, p_, q_;
    DBuf<double> rho_, rholast_, lambda_, beta_, def0_, def_;
    DBuf<int> conv_;   // per block: 0 active, 1 converged, 2 breakdown
    DBuf<BatchDev> st_;
    DBuf<unsigned int> counter_;
    BatchHostView* hview_ = nullptr;
    BatchHostView* dview_ = nullptr;
    std::vector<cudaEvent_t> ev_;
    cudaGraphExec_t exec_ = nullptr;
    const void* key_[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    long long key_gen_ = -1;
    long long nodes_ = 0;
    void setup(int n, int nblk, cudaStream_t s);
    void iteration(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, const BatchRanges& B, T* x,
                   const double* tol);
};

// State of BatchedCg3 (device), mirrored for the host in mapped memory: blocks left and iterations run
// per direction.
struct Batch3Dev {
    int iter, maxit, stop, left[3], iters[3], pad;
};
struct Batch3HostView {
    volatile int stop, active, breakdown, iters[3];
};

// The three right-hand sides of an upscaling batch, one CG recurrence per block and direction (the
// recurrences and tests of BatchedPcg), run together: the matrix and the AMG hierarchy are read once per
// iteration for three products and three cycles.  The CG is FP64; with an FP32 hierarchy the residual of
// each block and direction enters scaled by 1 / ||r0|| and the correction is scaled back (the hierarchy is
// linear and block diagonal, so the scaling only keeps the FP32 vectors in range).
class BatchedCg3 {
public:
    // b3, x3 (initial guess and result): three values per unknown, side by side.  Every block and
    // direction stops when ||r|| < tol ||r0|| or ||r|| < 1e-30.  iterations of the result: the sum over the
    // directions of the iterations until their last block stopped.
    template <class T>
    CgResult solve(cudaStream_t s, const SellPattern& P, const double* val, Amg<T>& M, const BatchRanges& B,
                   const double* b3, double* x3, double tol, int maxit);
    ~BatchedCg3();

private:
    void setup(const BatchRanges& B, bool fp32, cudaStream_t s);
    template <class T>
    void precondition(cudaStream_t s, Amg<T>& M);
    template <class T>
    void direction(cudaStream_t s, const BatchRanges& B, int first);
    template <class T>
    void iteration(cudaStream_t s, const SellPattern& P, const double* val, Amg<T>& M, const BatchRanges& B,
                   V3<double>* x, double tol);
    DBuf<V3<double>> r_, p_, q_, z64_, part_, part2_, scale_, iscale_;
    DBuf<V3<float>> r32_, z32_;
    DBuf<double> rho_, def0_, def_;
    DBuf<int> done_, broken_, conv_;   // per block and direction: 0 active, 1 converged, 2 breakdown; per block
    DBuf<Batch3Dev> st_;
    DBuf<unsigned int> counter_;
    Batch3HostView* hview_ = nullptr;
    Batch3HostView* dview_ = nullptr;
    std::vector<cudaEvent_t> ev_;
    cudaGraphExec_t exec_ = nullptr;
    const void* key_[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    long long key_gen_ = -1, nodes_ = 0;
    int key_n_[2] = {0, 0};
    double key_tol_ = 0.0;
};

}  // namespace porsol
