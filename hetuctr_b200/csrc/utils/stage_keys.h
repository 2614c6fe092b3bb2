// Copies a host key batch into the table's pinned staging area and checks its range on the way.
#pragma once
#include <cstddef>
#include <cstdint>

namespace hetuCTR {

// dst[i] = src[i] for n keys at any address; true when every key lies in [0, length).  The 32-bit form (length <= 2^31) halves what
// crosses the host link.  Out-of-range keys leave meaningless values in dst.
bool stage_keys(const int64_t *src, int32_t *dst, size_t n, size_t length);
bool stage_keys(const int64_t *src, int64_t *dst, size_t n, size_t length);

}  // namespace hetuCTR
