// Wavefront sweeps as one launch (implemented in flow.cu): Gauss-Seidel
// sweeps, the DIC/DILU factorisation and the DIC/DILU forward and backward
// sweeps of a level, with its rows as warp tasks taken in dependency order.
#pragma once

#include "kernels.hpp"
#include "small_solve.hpp"

namespace unapgpu {

// Most sweeps of one flow_gs launch.
constexpr int kFlowMaxSweeps = 16;
// Task counters at the head of a half: four, this far apart.
constexpr int kFlowCounterBytes = 4096;
constexpr int kFlowHeader = 4 * kFlowCounterBytes;

// Storage of one level's sweeps: one or two halves of `sweeps` vectors of n
// elements, each half headed by the task counters of the launch that writes
// it.  A launch reads its input from one half (or from elsewhere) and writes
// the other; the written half is filled with 0xff bytes first.
struct FlowRing {
    DevArray<unsigned char> mem;
    size_t stride = 0;   // bytes of one vector
    size_t half = 0;     // bytes of one half
    int sweeps = 0;      // vectors of one half
    int halves = 0;
    int* err = nullptr;  // pinned: set by a launch whose wait ran out
    int spent = 0;       // of its waits' polls (WaitBound)
    FlowRing() = default;
    FlowRing(const FlowRing&) = delete;
    FlowRing& operator=(const FlowRing&) = delete;
    FlowRing(FlowRing&& o) noexcept;
    FlowRing& operator=(FlowRing&& o) noexcept;
    ~FlowRing();
    void init(size_t n, size_t elemBytes, int sweepsPerHalf, int nHalves = 2);
    // grows to what nSweeps sweeps from an input outside the ring need, with up
    // to `most` of them in a launch: one half, or two if a launch follows that
    // reads the one before
    void ensure(size_t n, size_t elemBytes, int nSweeps, int most);
    size_t bytes() const { return mem.bytes(); }
    WaitBound bound() const { return {err, spent}; }
    // the half (0 or 1) that does not hold p; throws if the ring has one and
    // p is in it
    int other(const void* p) const;
    unsigned* counter(int h) const { return reinterpret_cast<unsigned*>(mem.p + h * half); }
    unsigned char* vec(int h, int i) const { return mem.p + h * half + kFlowHeader + i * stride; }
    // whether a wait of one of this ring's launches ran out since the last call
    // (after synchronizing with them); check() throws if so
    bool ranOut() const { return wait_ran_out(err); }
    void check() const;
};

[[noreturn]] void throw_ran_out();

// nSweeps Gauss-Seidel sweeps (forward, or backward in reverse cell order)
// from `in`; xIsZero: in is zero (forward, the first sweep then reads only
// its lower side, in may be null).  Returns the result's address: `last`
// where it is given (n elements, not `in`), else one of the ring's vectors.
// copy (optional, may be `in`: an entry is overwritten only by a row whose value
// depends, over its neighbours' values, on every row that read the old entry; a
// plain store cannot pass the loads that its value is made of): the result is
// written there too, row r at copyAt[r] if that is given (a launch that put the result into the caller's
// order took 16 of 278 us for two sweeps at 128^3).
template <class T>
T* flow_gs(const Exec& ex, const Level& L, const Rows<T>& A, const FlowRing& ring, const T* in,
           const T* b, int nSweeps, bool backward, bool xIsZero, T* last, T* copy, Gate g,
           const int* copyAt = nullptr);

// DIC / DILU.  rD: the factored diagonal's reciprocal; f: every entry times
// its row's reciprocal (rD coef on the lower side, rD upper on the upper
// side); part: partial sums of w.r, one per task; ring: the factored diagonal,
// then the forward sweep's vector.
struct DicFlow {
    DevArray<double> rD, f, part;
    FlowRing ring;
    void init(const Level& L);
    // after the factorisation, where only whole-solve launches use it (their
    // sweeps' vectors are in the solve's workspace): drops what they do not read
    void keepFactor();
    void check() const { ring.check(); }
};
// factors the level's matrix (DIC, or DILU); check() once it is done
void flow_dic_factor(const Exec& ex, const Level& L, bool dilu, DicFlow& D);
// w = M^-1 r; with a pool, w.r is reduced into `site` and finalized with fin
void flow_dic_apply(const Exec& ex, const Level& L, const DicFlow& D, const double* r, double* w,
                    const RedPool* pool, int site, KState* st, int fin, Gate g);

// the DIC/DILU fields of a whole-solve system (the level's and D's arrays)
void small_sweeps(SmallSystem& S, const Level& L, const DicFlow& D);
// the level's task table, built with the level (build_level)
void flow_tasks(Level& L, cudaStream_t s);

}  // namespace unapgpu
