// host_view_host.cpp — host build of host_view.h over a made-up map of pinned
// memory, for tests/test_host_view.py.  Nothing is dereferenced.  TEST HARNESS
// ONLY.
#include "../../libftcrypto_gb300/csrc/host_view.h"

// the device address of p[0, bytes) where the blocks i are [start[i], start[i]
// + size[i]), each `shift` away for the device
extern "C" uint64_t hv_device_view(const uint64_t *start, const uint64_t *size, int n, uint64_t shift, uint64_t p,
                                   uint64_t bytes)
{
    return (uint64_t)ft::device_view((const uint8_t *)p, bytes, [&](ft::HostBlock &b, const uint8_t *q) {
        for (int i = 0; i < n; ++i)
            if ((uint64_t)q >= start[i] && (uint64_t)q - start[i] < size[i]) {
                b.start = (const uint8_t *)start[i];
                b.bytes = size[i];
                b.device = (uint8_t *)((uint64_t)q + shift);
                return true;
            }
        return false;
    });
}
