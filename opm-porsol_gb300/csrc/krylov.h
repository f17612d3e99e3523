// krylov.h -- SELL SpMV, preconditioned CG with device-side scalars, ILU(0).
#pragma once

#include "porsol_internal.h"

namespace porsol {

// Device-resident CG scalars, written by one thread of a kernel and read by the next ones in stream order,
// so no host round trip is needed per iteration.  rho alternates between two slots (iter & 1): the blocks of
// the kernel that writes the new one still read the last.
struct CgDev {
    double rho[2], def0, def, tol;
    int iter, maxit, converged, stop, breakdown, pad;
};

// Mirror of the stopping state in mapped pinned host memory; the host reads it after an event behind the
// kernel that wrote it.
struct CgHostView {
    volatile double def0, def;
    volatile int iter, converged, stop, breakdown;
};

// Reduction scratch: partial sums per block + arrival counter (reset by the last block).
struct RedScratch {
    DBuf<double> partial;
    DBuf<unsigned int> counter;
    int max_blocks = 0;
    void ensure(int blocks, cudaStream_t s);
};

template <class T>
struct Precond {
    virtual ~Precond() = default;
    // z = M^{-1} r; kernels must do nothing when *stop != 0.  apply() must not synchronise
    // or allocate: it is captured into a CUDA graph.
    virtual void apply(cudaStream_t s, const T* r, T* z, const int* stop) = 0;
    // A preconditioner whose first kernel only forms r0 = dinv r and d = inv_theta r0 names them here; the
    // CG's last update of r then writes them and calls apply_started() (one launch and one pass less).
    struct Start {
        const T* dinv = nullptr;
        T *r0 = nullptr, *d = nullptr;
        T inv_theta = T(0);
    };
    virtual Start start() { return {}; }
    virtual void apply_started(cudaStream_t s, const T* r, T* z, const int* stop) { apply(s, r, z, stop); }
    // Batched solves: the per-block convergence flags (device, 0: block still iterating), so a
    // block-diagonal preconditioner may skip the rows of converged blocks; null for one system.
    virtual void set_block_state(const int*) {}
    // Changes whenever the kernels apply() launches change (new setup/factorisation).
    long long generation() const { return gen_; }
    void bump_generation() { ++gen_; }

private:
    long long gen_ = 0;
};

template <class TV, class TX>
void spmv(cudaStream_t s, const SellPattern& P, const TV* val, const TX* x, TX* y);

// y = b - A x  (residual)
template <class TV, class TX>
void residual(cudaStream_t s, const SellPattern& P, const TV* val, const TX* x, const TX* b, TX* y);

struct CgResult {
    int iterations = 0;
    double reduction = 0.0, def0 = 0.0, def = 0.0;
    bool converged = false, breakdown = false;
};

// Preconditioned CG, the algorithm of dune-istl's CGSolver::apply: stop when
// ||b - A x||_2 < tol ||b - A x0||_2 (or < 1e-30) or after maxit iterations.
// x holds the initial guess on entry.  TV = matrix value type, T = vector type.
template <class TV, class T>
class PcgSolver {
public:
    void setup(int n, cudaStream_t s);
    CgResult solve(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, const T* b, T* x,
                   double tol, int maxit, Profiler* prof = nullptr, int prof_kernel = -1);
    // Replay one CG iteration (SpMV, updates, preconditioner) as a CUDA graph.
    void set_graphs(bool on) { use_graphs_ = on; }
    ~PcgSolver();

private:
    int n_ = 0;
    DBuf<T> r_, z_, p_, q_;
    DBuf<CgDev> st_;
    RedScratch red_;       // residual norms
    DBuf<double> pq_, zr_;   // partial sums of p.q and z.r
    CgHostView* hview_ = nullptr;
    CgHostView* dview_ = nullptr;
    std::vector<cudaEvent_t> ev_;
    bool use_graphs_ = true;
    cudaGraphExec_t exec_ = nullptr;
    const void* key_[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    long long key_gen_ = -1;
    long long nodes_ = 0;   // kernels in one captured iteration
    void iteration(cudaStream_t s, const SellPattern& P, const TV* val, Precond<T>& M, T* x, Profiler* prof,
                   int prof_kernel);
};

// Mixed-precision CG with reliable updates (residual replacement; Sleijpen and van der Vorst,
// "Reliable updated residuals in hybrid Bi-CG methods", Computing 56, 1996): one FP32 CG
// recurrence (FP32 matrix copy, FP32 preconditioner) on the system scaled by sigma, the
// solution accumulated in FP64 (x += sigma alpha p), and the iterated residual replaced by the
// true FP64 residual b - A x whenever it has dropped by `delta` since the last replacement or
// the estimate reaches the tolerance.  Unlike restarted iterative refinement the search
// direction is kept across replacements (rescaled), so no Krylov information and no extra
// preconditioner application is lost.  Stops when the true residual satisfies
// ||b - A x|| < tol ||b - A x0|| (or < 1e-30).
//
// The recurrence's alpha and beta hold while r stays orthogonal to the last direction and z to the last
// residual.  Rounding and replacements take that away in some large, strongly heterogeneous systems: the
// residual then hardly drops (1M cells with log-normal layers: 3 of 48 realisations took 150 iterations to
// thousands or broke down, the others 40 to 80).  A stage between replacements that lasts RC_STAGE iterations
// (10 to 15 are usual), or a curvature that is not positive, switches to the guarded form, alpha = p.r / p.q
// and beta = -z.q / p.q, which minimise along the direction at hand whatever came before: a solve of 5874
// iterations then takes 180.  A curvature that is not positive in the guarded form ends the solve.
struct RcDev {
    double rho[2], pq, sigma, isig, def0, tol, delta, true_def;
    float factor;
    int iter, last, maxit, stop, converged, breakdown, replaced, nrep;
    int guard, restart, fresh;   // fresh: p = z; restart: make it so
};

class ReliableCg {
public:
    // prof (may be null): when per-kernel event timing is on, iterations run uncaptured
    CgResult solve(cudaStream_t s, const SellPattern& P, const double* val64, const float* val32,
                   Precond<float>& M, const double* b, double* x, double tol, int maxit, double delta,
                   Profiler* prof = nullptr);
    int replacements() const { return nrep_; }
    bool guarded() const { return guarded_; }   // the last solve ended in the guarded form
    ~ReliableCg();

private:
    int n_ = 0, nrep_ = 0;
    bool guarded_ = false;
    DBuf<float> r_, z_, p_, q_;
    DBuf<double> r64_;       // the true residual at a replacement
    DBuf<RcDev> st_;
    RedScratch red_;         // FP64 residual norms
    DBuf<double> pq_, pr_, rr_, zr_;   // partial sums of p.q, p.r, r.r and z.r (guarded: z.q)
    CgHostView* hview_ = nullptr;
    CgHostView* dview_ = nullptr;
    std::vector<cudaEvent_t> ev_;
    cudaGraphExec_t exec_ = nullptr;
    const void* key_[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    long long key_gen_ = -1;
    long long nodes_ = 0;
    void setup(int n, cudaStream_t s);
    void iteration(cudaStream_t s, const SellPattern& P, const double* val64, const float* val32, Precond<float>& M,
                   const double* b, double* x, Profiler* prof);
};

// Mixed CG from x = 0 on a symmetric CSR matrix (host arrays) with a Jacobi preconditioner whose applications
// [skip, skip + skips) return zero (a direction of zero curvature); throws what a solve does.
int mixed_cg_selftest(int n, const int* ptr, const int* col, const double* val, const double* b, double* x, double tol,
                      int maxit, double delta, int skip, int skips, int* iterations, int* guarded);

// ILU(0) with the pivots stored inverted, factor and triangular solves level-scheduled
// (rows of one level are independent).  The algorithm of dune-istl's SeqILU0 with
// relaxation 1 (IncompFlowSolverHybrid.hpp:1404).
//
// The levels of a mid-size grid hold tens of rows and a sweep has a hundred levels, so a launch per
// level costs a launch latency per handful of rows.  Runs of levels of at most FUSE_ROWS rows are swept
// by one block in one launch (k_ilu_steps), from records of the two triangles in sweep order;
// wider levels, which would wait for one SM's FP64 pipe, keep a launch of their own.  Per CG iteration, with
// levels fused up to 0 / 384 / 512 / 768 / 1024 rows: 30^3 cells 1653 / 1184 / 1186 / 1195 / 1195 us, 40^3 2304 / 1883 /
// 1876 / 2029 / 2682, 100 x 100 x 10 3539 / 2929 / 3012 / 3234 / 3855, 60^3 5216 / 4571 / 4511 / 4492 / 4638.  Small
// systems without a level of more than SHARED_ROWS rows are swept in one launch, the vector in shared memory.
class Ilu0 : public Precond<double> {
public:
    // structure only; shared: the sweep's vector may live in shared memory
    void build_levels(const SellPattern& P, cudaStream_t s, bool shared = true);
    void factor(cudaStream_t s, const SellPattern& P, const double* val);
    void apply(cudaStream_t s, const double* r, double* z, const int* stop) override;
    // error bits set by apply() (ST_TIMEOUT: a bounded wait for a bulk copy gave up); synchronises the stream
    int solve_status(cudaStream_t s) const;
    int num_levels_lower() const { return int(h_lptr_.size()) - 1; }
    int num_levels_upper() const { return int(h_uptr_.size()) - 1; }

private:
    static constexpr int FUSE_ROWS = 512, SHARED_ROWS = 1024;
    const SellPattern* P_ = nullptr;
    DBuf<double> lu_;
    std::vector<int> h_lptr_, h_uptr_;
    DBuf<int> lrows_, urows_;
    DBuf<int> status_;
    // a launch of apply(): steps [a, b) of the fused sweep, or (fused false) level a of the lower (b = 0)
    // or upper (b = 1) triangle
    struct Run {
        bool fused;
        int a, b;
    };
    std::vector<Run> runs_;
    DBuf<int2> steps_;             // the fused sweep's steps and their records (k_ilu_steps)
    DBuf<unsigned char> blob_;
    DBuf<int> pos_, from_;         // value pos_[e] of the records is the factor's slot from_[e]
    bool shared_z_ = false;        // the sweep's vector lives in shared memory
    int stages_ = 2;
    size_t steps_shm() const;      // dynamic shared memory of k_ilu_steps
    friend int ilu_sweep_selftest(int thread, bool shared, double* z);
};

// The fused sweeps on a fixed 48-row system (thread >= 0: that thread's wait for a step record runs out); returns
// the kernel's status bits and the 48 values of z.
int ilu_sweep_selftest(int thread, bool shared, double* z);

// Helpers used by the solver front end.
void device_copy(cudaStream_t s, void* dst, const void* src, size_t bytes);
template <class TA, class TB>
void convert(cudaStream_t s, long long n, const TA* a, TB* b);
// x += y (FP64)
void axpy_add(cudaStream_t s, int n, const double* y, double* x);
// Dirichlet-row initial guess (IncompFlowSolverHybrid.hpp:1521-1532): x_i = b_i / a_ii
// where all off-diagonal entries of row i are zero, else 0.
void dirichlet_guess(cudaStream_t s, const SellPattern& P, const double* val, const double* b, double* x);
// 2-norm of a vector (synchronous, FP64 accumulation)
template <class T>
double norm2(cudaStream_t s, int n, const T* x, RedScratch& red);

}  // namespace porsol
