// Host entry over the decision that the scans make on a total, for the CPU
// test (tests/test_offset_totals.py).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "../pdf-raster_b200/csrc/rrb_device.cuh"
#include "../pdf-raster_b200/csrc/rrb_kernels.cuh"

extern "C" int ot_fits(const uint32_t* counts, uint64_t n, uint32_t cap) {
    unsigned long long total = 0;
    for (uint64_t i = 0; i < n; ++i) total += counts[i];
    return rrb::scan_fits(total, std::min(cap, rrb::MAX_OFFSET)) ? 1 : 0;
}
