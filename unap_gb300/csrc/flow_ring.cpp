// The storage of wavefront sweeps (see flow.hpp).
#include <algorithm>

#include "flow.hpp"

namespace unapgpu {

FlowRing::FlowRing(FlowRing&& o) noexcept
    : mem(std::move(o.mem)), stride(o.stride), half(o.half), sweeps(o.sweeps), halves(o.halves),
      err(o.err), spent(o.spent)
{
    o.err = nullptr;
}

FlowRing& FlowRing::operator=(FlowRing&& o) noexcept
{
    mem = std::move(o.mem);
    stride = o.stride;
    half = o.half;
    sweeps = o.sweeps;
    halves = o.halves;
    std::swap(err, o.err);
    spent = o.spent;
    return *this;
}

FlowRing::~FlowRing() { pinned_block_free(err); }

void FlowRing::init(size_t n, size_t elemBytes, int sweepsPerHalf, int nHalves)
{
    // set last: an allocation that throws leaves the ring without vectors
    sweeps = halves = 0;
    const int per = std::max(1, std::min(sweepsPerHalf, kFlowMaxSweeps));
    stride = (n * elemBytes + 255) / 256 * 256;
    half = kFlowHeader + stride * (size_t)per;
    if (!err) {
        // not cleared when the ring grows: a launch on it may have set it
        err = static_cast<int*>(pinned_block_alloc(64));
        *err = 0;
    }
    mem.alloc((size_t)nHalves * half);
    sweeps = per;
    halves = nHalves;
}

void FlowRing::ensure(size_t n, size_t elemBytes, int nSweeps, int most)
{
    if (nSweeps <= 0) return;
    const int per = std::min(nSweeps, most), h = nSweeps > per ? 2 : 1;
    if (sweeps < per || halves < h)
        init(n, elemBytes, std::max(per, sweeps), std::max(h, halves));
}

int FlowRing::other(const void* p) const
{
    const unsigned char* q = static_cast<const unsigned char*>(p);
    if (!(q >= mem.p && q < mem.p + half)) return 0;
    if (halves < 2) throw std::logic_error("sweeps in place on a ring of one half");
    return 1;
}

void DicFlow::init(const Level& L)
{
    rD.alloc((size_t)L.n);
    f.alloc((size_t)L.nEntries);
    part.alloc((size_t)std::max(L.tasks[0].n, 1));
    ring.init((size_t)L.n, sizeof(double), 1, 1);
}

void DicFlow::keepFactor()
{
    ring.mem.release();
    ring.sweeps = ring.halves = 0;
    part.release();
}

void throw_ran_out()
{
    throw CudaError("a wait for another row of a sweep ran out");
}

void FlowRing::check() const
{
    if (ranOut()) throw_ran_out();
}

}  // namespace unapgpu
