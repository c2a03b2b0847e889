// FlowRing: the vectors of wavefront sweeps (see flow.hpp).
#include <algorithm>

#include "flow.hpp"

namespace unapgpu {

FlowRing::FlowRing(FlowRing&& o) noexcept
    : mem(std::move(o.mem)), stride(o.stride), half(o.half), sweeps(o.sweeps), err(o.err), polls(o.polls)
{
    o.err = nullptr;
}

FlowRing& FlowRing::operator=(FlowRing&& o) noexcept
{
    mem = std::move(o.mem);
    stride = o.stride;
    half = o.half;
    sweeps = o.sweeps;
    std::swap(err, o.err);
    polls = o.polls;
    return *this;
}

FlowRing::~FlowRing() { pinned_block_free(err); }

void FlowRing::init(size_t n, size_t elemBytes, int sweepsPerHalf, int halves)
{
    // set last: an allocation that throws leaves the ring without vectors
    sweeps = 0;
    const int per = std::max(1, std::min(sweepsPerHalf, kFlowMaxSweeps));
    stride = (n * elemBytes + 255) / 256 * 256;
    half = kFlowHeader + stride * (size_t)per;
    if (!err) {
        // not cleared when the ring grows: a launch on it may have set it
        err = static_cast<int*>(pinned_block_alloc(64));
        *err = 0;
    }
    mem.alloc((size_t)halves * half);
    sweeps = per;
}

int FlowRing::other(const void* p) const
{
    const unsigned char* q = static_cast<const unsigned char*>(p);
    return q >= mem.p && q < mem.p + half ? 1 : 0;
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
