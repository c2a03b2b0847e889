// Entry counts of a row in one word: every split of rows of up to 65,535
// faces comes back as it went in.
#include <cstdio>

#include "unap_internal.hpp"

int main()
{
    using namespace unapgpu;
    const int lens[] = {0, 1, 32767, 32768, 40000, 65534, 65535};
    for (int len : lens)
        for (int low : lens) {
            if (low > len) continue;
            const int info = row_info(len, low);
            if (row_len(info) != len || row_low(info) != low) {
                std::printf("len %d low %d: read back %d %d\n", len, low, row_len(info),
                            row_low(info));
                return 1;
            }
        }
    std::puts("ok");
    return 0;
}
