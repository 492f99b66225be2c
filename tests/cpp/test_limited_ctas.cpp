// The CTAs per SM of a ragged pass under a tuning's limit, whose unit is 8
// warps whatever the CTA size is.
#include <cuda_runtime.h>

#include "sbf_internal.h"

using sbf::limited_ctas;

int main() {
    bool ok = limited_ctas(0, 6, 128) == 6 && limited_ctas(0, 2, 256) == 2;
    for (uint32_t threads = 64; threads <= 256; threads *= 2) {
        const uint32_t occupancy = 24 * 32 / threads;  // 24 warps fit
        ok = ok && limited_ctas(1, occupancy, threads) * threads == 256;
        ok = ok && limited_ctas(2, occupancy, threads) * threads == 512;
        ok = ok && limited_ctas(3, occupancy, threads) * threads == 768;
        ok = ok && limited_ctas(4, occupancy, threads) == occupancy;
        ok = ok && limited_ctas(0xFFFFFFFFu, occupancy, threads) == occupancy;
    }
    ok = ok && limited_ctas(1, 3, 512) == 1;  // never none
    return ok ? 0 : 1;
}
