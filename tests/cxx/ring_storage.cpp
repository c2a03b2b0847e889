// The vectors that sweeps keep: as many as their launches write, and a second
// half only where a launch reads what the one before wrote.
#include "fake_runtime.hpp"
#include "flow.hpp"

using namespace unapgpu;

int main()
{
    const size_t n = 1 << 15, vec = n * sizeof(double);
    {
        FlowRing r;
        r.ensure(n, sizeof(double), 0, 4);
        EXPECT(r.bytes() == 0);
        r.ensure(n, sizeof(double), 2, 4);
        EXPECT(r.bytes() == kFlowHeader + 2 * vec && r.other(nullptr) == 0);
        bool threw = false;
        try {
            r.other(r.vec(0, 1));
        } catch (const std::logic_error&) {
            threw = true;
        }
        EXPECT(threw);
        r.ensure(n, sizeof(double), 4, 4);
        EXPECT(r.bytes() == kFlowHeader + 4 * vec);
        const void* p = r.mem.p;
        r.ensure(n, sizeof(double), 1, 4);
        EXPECT(r.mem.p == p && r.sweeps == 4);
        r.ensure(n, sizeof(double), 5, 4);
        EXPECT(r.bytes() == 2 * (kFlowHeader + 4 * vec));
        EXPECT(r.other(r.vec(0, 3)) == 1 && r.other(r.vec(1, 0)) == 0);
    }
    {
        FlowRing r;  // 16 sweeps in one launch
        r.ensure(n, sizeof(double), 16, kFlowMaxSweeps);
        EXPECT(r.bytes() == kFlowHeader + 16 * vec);
    }
    {
        Level L;
        L.n = (int)n;
        L.nEntries = 7 * (long long)n;
        L.tasks[0].n = 100;
        DicFlow D;
        D.init(L);
        EXPECT(D.ring.bytes() == kFlowHeader + vec);
        D.keepFactor();
        EXPECT(D.rD.p && D.f.p && D.ring.bytes() == 0 && D.part.bytes() == 0);
        EXPECT(D.ring.err && !D.ring.ranOut());
    }
    EXPECT(fake::live == 0);
    std::puts("ok");
    return 0;
}
