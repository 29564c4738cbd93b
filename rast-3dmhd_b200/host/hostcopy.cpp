// hostcopy.cpp - host memory copies by several threads (device transfers of pageable arrays).
#include <algorithm>
#include <cstring>

#include "r3d_host.hpp"

namespace r3db {

// One thread copies into freshly allocated pages at a few GB/s (it takes their page faults on the
// way), far below the link to the device; eight run at several times that.
void parallel_copy(void* dst, const void* src, size_t bytes) {
    constexpr size_t kBlock = size_t(1) << 19;
    const long blocks = (long)((bytes + kBlock - 1) / kBlock);
#pragma omp parallel for schedule(static) num_threads(8) if (blocks > 1)
    for (long b = 0; b < blocks; ++b) {
        const size_t off = (size_t)b * kBlock;
        std::memcpy((char*)dst + off, (const char*)src + off, std::min(kBlock, bytes - off));
    }
}

}  // namespace r3db
