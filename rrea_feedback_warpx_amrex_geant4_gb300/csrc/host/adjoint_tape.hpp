// How much of the adjoint's tape is kept between the forward and the reverse
// pass.
#pragma once

#include <cstdint>

namespace rrea_host {

// Segments of the tape, of `segment_bytes` each, that a problem of `segments`
// keeps where the device has `free_bytes` left after all other arrays: within
// `limit_bytes` and half of what is free, since anything beyond the one
// segment every reverse pass needs only saves time.  At least that one.
inline int kept_segments(int64_t segments, int64_t segment_bytes, int64_t limit_bytes, int64_t free_bytes)
{
    int64_t const budget = limit_bytes < free_bytes / 2 ? limit_bytes : free_bytes / 2;
    int64_t const fit = segment_bytes > 0 ? budget / segment_bytes : segments;
    return static_cast<int>(fit < 1 ? 1 : fit < segments ? fit : segments);
}

}  // namespace rrea_host
