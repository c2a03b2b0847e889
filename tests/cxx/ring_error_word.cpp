// A ring that grows keeps the error word of a launch on its former vectors;
// the word is read once.
#include "fake_runtime.hpp"
#include "flow.hpp"

using namespace unapgpu;

int main()
{
    FlowRing r;
    r.init(100, 8, 2);
    EXPECT(!r.ranOut());
    *r.err = 1;  // a launch's wait ran out
    r.init(100, 8, 4);
    EXPECT(r.ranOut() && !r.ranOut());
    *r.err = 1;
    bool threw = false;
    try {
        r.check();
    } catch (const CudaError&) {
        threw = true;
    }
    EXPECT(threw && !r.ranOut());
    std::puts("ok");
    return 0;
}
