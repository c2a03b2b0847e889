// An allocation that fails while the workspace pool holds unused blocks
// succeeds once they are given back: cudaMalloc, either pool of a
// stream-ordered array, and setup scratch.
#include "fake_runtime.hpp"

using namespace unapgpu;

int main()
{
    cudaStream_t s = reinterpret_cast<cudaStream_t>(0x10);
    cudaMemPool_t pool = reinterpret_cast<cudaMemPool_t>(0x20);
    int want = 0;
    try {
        {
            fake::pool_holds = true;
            DevArray<double> a(10);
            EXPECT(a.p && fake::trims == ++want);
        }
        {
            StreamAllocScope scope(s);
            fake::pool_holds = true;
            DevArray<double> a(10);
            EXPECT(a.p && fake::trims == ++want);
        }
        {
            StreamAllocScope scope(s, pool);
            fake::pool_holds = true;
            DevArray<double> a(10);
            EXPECT(a.p && fake::trims == ++want);
        }
        {
            fake::pool_holds = true;
            StreamScratch<int> a(10, s);
            EXPECT(a.p && fake::trims == ++want);
        }
        // memory that is really gone is an error after one more try
        fake::fail_next = 2;
        fake::calls = 0;
        bool threw = false;
        try {
            StreamScratch<int> a(10, s);
        } catch (const CudaError&) {
            threw = true;
        }
        EXPECT(threw && fake::calls == 2);
    } catch (const std::exception& e) {
        std::printf("%s\n", e.what());
        return 1;
    }
    EXPECT(fake::live == 0);
    std::puts("ok");
    return 0;
}
