// Where setup runs by kernels: matrices, levels of a hierarchy, COO/CSR input.
#include "fake_runtime.hpp"

using namespace unapgpu;

int main()
{
    const long long m = kDeviceSetupCells;
    EXPECT(m == 32768);
    // a level above the limit always, a smaller one where its chain is short
    EXPECT(setup_level_on_device(m, m, -1, kCellsPerRound));
    EXPECT(!setup_level_on_device(m, m - 1, -1, kCellsPerRound));
    EXPECT(setup_level_on_device(m, m / 4, 0, kCellsPerWavefront));
    EXPECT(!setup_level_on_device(m, m / 4 - 1, 0, kCellsPerWavefront));
    EXPECT(setup_level_on_device(m, 20480, 80, 256) && !setup_level_on_device(m, 20479, 80, 256));
    EXPECT(setup_level_on_device(m, m, 1 << 30, 512));
    EXPECT(!setup_level_on_device(-1, 1 << 30, 0, 256));
    EXPECT(setup_level_on_device(1, 1, -1, 256) && setup_level_on_device(0, 0, -1, 256));
    // input: by cells, or by entries from a quarter of the cells on
    EXPECT(setup_input_on_device(m, m, 0) && !setup_input_on_device(m, m - 1, 2 * m - 1));
    EXPECT(setup_input_on_device(m, m / 4, 2 * m) && !setup_input_on_device(m, m / 4 - 1, 2 * m));
    EXPECT(!setup_input_on_device(-1, m, 2 * m));
    std::puts("ok");
    return 0;
}
