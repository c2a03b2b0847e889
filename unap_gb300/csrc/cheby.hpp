// Chebyshev smoothing (chebySmoother.cpp:44-148) and its largest-eigenvalue
// estimate (eigenDiagPCG.cpp:11-361) on the device, shared by the
// reference MGSolver (mg.cu) and the AMG V-cycle (amg.cu).
//
// A Chebyshev step is SpMV-shaped: every row reads the previous iterate of
// its neighbours and nothing else of the step, so a level is one launch per
// step (no wavefronts), with the iterate double-buffered.  Per row, in the
// reference's arithmetic order (A x as lduMatrix::spMV sums it, rD = 1/diag):
//   first step from x = 0:  w = rD b Rtheta;              x = w
//   first step from x:      w = rD (b - A x) Rtheta;      x = x + w
//   step j >= 1:            w = d1_j w + d2_j rD (b - A x); x = x + w
#pragma once

#include "kernels.hpp"

namespace unapgpu {

constexpr int kChebyMaxDegree = 16;

// Eigenvalue estimate state of one smoother (eigenDiagPCG.cpp:48-238:
// diagonal-PCG iterations recording alpha and beta).
struct EigState {
    double wArA, wArAold, wApA, alpha, beta;
    int broken, pad;
    double alphas[16], betas[16];
    double maxEig;
};

// A level whose largest eigenvalue is estimated.  x: start, updated in place.
// es must hold wArA = GREAT and zeros on entry.  rA, wA, pA: n-vector scratch;
// wr and al: two reduction sites of its own.
struct EigLevel {
    Rows<double> A;
    const double* rD;
    double *x, *rA, *wA, *pA;
    EigState* es;
    RSpec wr, al;
    int block0 = 0, nBlocks = 0;  // set by eig_diag_pcg
};
constexpr int kEigSet = 16;

// eigenDiagPCG::diagPCGLoops on each of `count` (<= kEigSet) levels: nIt
// (<= 16) diagonal-PCG iterations on (x, b).  A breakdown (|wArA| < VSMALL)
// sets es->broken and leaves the remaining alphas 0.
void eig_diag_pcg(const Exec& ex, EigLevel* lv, int count, const double* const* b, int nIt);

// eigenDiagPCG::computeMaxEig (eigenDiagPCG.cpp:242-361) on one device
// thread: es->maxEig = the largest eigenvalue of the Lanczos tridiagonal of
// the iterations done (nonzero alphas, at most nMax <= 16) by Sturm-sequence
// bisection to a band of 1e-5; 1 / alpha_0 after one iteration, 1 after none.
void k_eig_sturm(const Exec& ex, EigState* es, int nMax, int count = 1);

// Start vector of the AMG levels' eigenvalue estimate: cell c (reference
// numbering of its level) gets a uniform value in [-1, 1) from splitmix64.
void k_eig_start(const Exec& ex, int n, const int* perm, double* b);

// r[i] = 1 / d[i] (lduDiagPrecond.cpp:13-41)
void k_reciprocal(const Exec& ex, int n, const double* d, double* r);

// chebySmoother.cpp:62-108 for the interval [lam / ratio, 1.1 lam]:
// Rtheta of the first step and (d1[j], d2[j]) of steps j = 1 .. deg - 1.
void cheby_coeffs(double lam, double ratio, int deg, double* Rtheta, double* d1, double* d2);

// One Chebyshev step on every row of A: first != 0 is the first step from a
// nonzero x (c1 = Rtheta), else a later step (c1 = d1, c2 = d2).  xin and
// xout are distinct.  Launched with programmatic dependent launch when
// wave_pdl() is on: the kernel loads its rows' matrix data and b before it
// waits for the previous kernel.
template <class T>
void k_cheb_step(const Exec& ex, const Rows<T>& A, const T* xin, T* xout, const T* b, T* w, T c1,
                 T c2, int first, Gate g);
// First step from x = 0: w = x = rD b Rtheta.  With r64 != null (FP32
// levels entered from FP64) b is first set to (float)r64.
template <class T>
void k_cheb_zero(const Exec& ex, int n, const T* diag, T* b, const double* r64, T* x, T* w, T Rth,
                 Gate g);
// Restriction into a Chebyshev level fused with that level's first step:
// coarse[C] = sum of the children (ascending), then w = x = rD coarse Rtheta.
template <class T>
void k_restrict_cheb_zero(const Exec& ex, int nC, const int* childStart, const int* child,
                          const T* fine, T* coarse, const T* diagC, T* xC, T* wC, T Rth, Gate g);
// Out-of-place prolongation: xout[i] = xin[i] + coarse[cmap[i]].
template <class T>
void k_prolong_add_to(const Exec& ex, int n, const int* cmap, const T* coarse, const T* xin,
                      T* xout, Gate g);

// ---- the coarse end of a Chebyshev V-cycle in one launch (cheb_flow.cu) --
constexpr int kChebTailRows = 60000;   // default of set_cheby_tail_rows
// By default a tail level's rows also hold up to this many entries on average,
// what a task loads before any wait: longer rows take another dependent load per
// 32 entries, past L1, where the per-step kernels' gathers hit it.  What one more
// level in the tail changes of a V-cycle, us: FP32, 4 to 25 entries, -6 to -18 at
// 100 to 30,000 rows; 50 to 100 entries, +5 to +40; 150 to 900, +15 to +165 (a
// hierarchy of a random graph of 30,000 cells and 20 entries: 512 without a tail,
// 736 with all levels in it).  FP64, where the sums are longer than the loads:
// 32 to 900 entries, -35 to +57 up to 2,048 rows, -30 to +424 at 2,500 to 8,000.
constexpr int kChebTailEntries = 32;
constexpr int kChebTailLongRows64 = 2048;  // FP64 levels of any row length
constexpr int kChebTailMaxStages = 600;
constexpr int kChebTailCtas = 8;       // CTAs of 128 threads an SM at most

// one tail level: its matrix, the restriction into it (children of each
// cell, ascending), the prolongation from it (finer row -> cell) and its
// Chebyshev coefficients
template <class T>
struct ChebFlowLevel {
    Rows<T> A;
    const int* childStart;
    const int* child;
    const int* cmap;
    double Rth;
    const double* d1;
    const double* d2;
};

// stages of a tail of `levels` levels above the coarsest
inline int cheb_flow_stages(int levels, int deg) { return levels * (2 * deg + 2) + 3; }

template <class T>
struct ChebFlow {
    DevArray<unsigned char> arena;   // task counters, then every stage's vectors
    DevArray<unsigned char> stages;
    int nStages = 0, nTasks = 0, nc = 0, grid = 0;
    const double* M = nullptr;
    double* part = nullptr;
    int* err = nullptr;              // pinned: set when a wait ran out
    int spent = 0;                   // of its waits' polls (WaitBound)
    ChebFlow() = default;
    ChebFlow(const ChebFlow&) = delete;
    ChebFlow& operator=(const ChebFlow&) = delete;
    ~ChebFlow();
    // levels in order, finest first; rIn: the residual of the level above
    // the first; result: where the first level's iterate goes
    void build(const std::vector<ChebFlowLevel<T>>& lev, int deg, const T* rIn, int nc,
               const int* cChildStart, const int* cChild, const int* cCmap, const double* Minv,
               T* result, cudaStream_t s);
    void launch(const Exec& ex, Gate g) const;
    bool ranOut() const { return wait_ran_out(err); }  // a wait (after synchronizing)
    size_t bytes() const { return arena.bytes() + stages.bytes(); }
};

// Chebyshev V-cycles run their levels of at most `rows` rows (and every
// level below them) in the tail launch; 0 turns it off.  The default also
// looks at the rows' length (above), other values do not.  Returns the
// previous value; applies to hierarchies built afterwards.
int set_cheby_tail_rows(int rows);
int cheby_tail_rows();

// Rows per level below which Chebyshev-step launches use one-warp CTAs
// (spread over more SMs); returns the previous value.
int set_cheby_small_rows(int rows);
// Entries of a row loaded per dependent round trip by the Chebyshev step: 0
// (default) 16 on levels averaging more than 8 entries per row, except FP32
// levels of a million rows or more (8: more CTAs per SM), else 8; 8 or 16
// on every level.  Returns the previous value.
int set_cheby_chunk(int entries);

}  // namespace unapgpu
