// Chunk boundaries of a host-buffer trace's pipeline (host code, no CUDA).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace rg {

// 0, the boundaries and n, ascending, for n rays in chunks of `chunk` (at
// least 1024 when below n): with three or more full chunks, the first two and
// the last two ramp (a quarter, a half of a chunk) so that the first trace
// starts early and the last download is short. The ramps take 6 quarters, and
// a quarter is at least 1024 rays: small chunks go without them where that is
// not less than n.
inline std::vector<uint64_t> trace_cuts(uint64_t n, uint64_t chunk) {
    std::vector<uint64_t> cut{0};
    const uint64_t q = std::max<uint64_t>(1024, (chunk / 4) & ~uint64_t(1023));
    if (chunk < n && n + 4096 > 4 * chunk && n > 6 * q) { // (host_chunk rounds a quarter up)
        const uint64_t mid = n - 6 * q, parts = (mid + chunk - 1) / chunk, step = ((mid + parts - 1) / parts + 1023) & ~uint64_t(1023);
        cut.push_back(q);
        cut.push_back(3 * q);
        for (uint64_t b = 3 * q + step; b < n - 3 * q; b += step) cut.push_back(b);
        cut.push_back(n - 3 * q);
        cut.push_back(n - q);
    } else {
        for (uint64_t b = chunk; b < n; b += chunk) cut.push_back(b);
    }
    cut.push_back(n);
    return cut;
}

} // namespace rg
