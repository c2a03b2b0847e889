// An array or a sweep's vectors whose allocation failed hold nothing: their
// sizes, by which a later call decides whether to allocate, say so.
#include "fake_runtime.hpp"
#include "flow.hpp"

using namespace unapgpu;

int main()
{
    DevArray<double> a(5);
    fake::fail_next = 2;
    bool threw = false;
    try {
        a.alloc(10);
    } catch (const CudaError&) {
        threw = true;
    }
    EXPECT(threw && !a.p && a.n == 0);
    a.alloc(10);
    EXPECT(a.p && a.n == 10);
    {
        FlowRing r;
        r.init(100, 8, 2);
        EXPECT(r.sweeps == 2 && r.mem.p);
        fake::fail_next = 2;
        threw = false;
        try {
            r.init(100, 8, 4);
        } catch (const CudaError&) {
            threw = true;
        }
        EXPECT(threw && r.sweeps == 0 && !r.mem.p);
        r.init(100, 8, 4);
        EXPECT(r.sweeps == 4 && r.mem.p);
    }
    a.release();
    EXPECT(fake::live == 0);
    std::puts("ok");
    return 0;
}
