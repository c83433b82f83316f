// host_range.hpp — whether a kernel may read or write all of a host buffer.  Plain C++, so that it is tested without a GPU.
#pragma once

#include <cstddef>
#include <cstdint>

namespace hc {

// `mapped(address)`: whether the device reaches the byte there under the same address.  Memory is pinned by the page, and a
// buffer may be pinned in part: its first byte, a byte of every page it reaches into and its last byte are asked for (a page
// is 4 KB or a multiple of it).
template <typename Mapped>
bool host_range_mapped(Mapped mapped, const void* buffer, size_t bytes) {
    if (bytes == 0) return false;
    constexpr uintptr_t kPage = 4096;
    const uintptr_t first = reinterpret_cast<uintptr_t>(buffer), last = first + (bytes - 1);
    if (last < first || !mapped(reinterpret_cast<const void*>(first)) || !mapped(reinterpret_cast<const void*>(last))) return false;
    for (uintptr_t page = first / kPage + 1; page < last / kPage; ++page) {
        if (!mapped(reinterpret_cast<const void*>(page * kPage))) return false;
    }
    return true;
}

}  // namespace hc
