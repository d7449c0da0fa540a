// host_view.h — which host memory of a caller a kernel may address itself.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace ft {

// one allocation or registration of pinned memory, as the driver knows it
struct HostBlock {
    const uint8_t *start;
    size_t bytes;
    uint8_t *device; // where the device addresses the byte that was asked for
};

// Where the device addresses the `bytes` bytes at p: all of them in one block
// of pinned memory, 16-byte aligned; else nullptr.  (Pages between two blocks
// need not be the device's, whatever the bytes at both ends are.)  query(b, p)
// fills in the block that holds p; false: none.
template <class Query>
uint8_t *device_view(const uint8_t *p, size_t bytes, Query query)
{
    HostBlock b;
    if (!query(b, p) || !b.device || (uintptr_t)b.device % 16 || p < b.start) return nullptr;
    const size_t at = (size_t)(p - b.start);
    if (at > b.bytes || bytes > b.bytes - at) return nullptr;
    return b.device;
}

} // namespace ft
