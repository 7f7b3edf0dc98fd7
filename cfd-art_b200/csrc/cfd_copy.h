// A copy of `bytes` bytes cut into `parts` parts that start on 4096-byte steps.
#pragma once

#include <algorithm>
#include <cstddef>

namespace cfd {

struct CopyPart {
    size_t lo, n;
};
// Part k of 0 .. parts - 1; the last one takes whatever the others leave.
inline CopyPart copy_part(size_t bytes, size_t parts, size_t k) {
    const size_t step = (bytes / parts + 4095) / 4096 * 4096;
    const size_t lo = std::min(k * step, bytes);
    return {lo, k + 1 == parts ? bytes - lo : std::min(step, bytes - lo)};
}

}  // namespace cfd
