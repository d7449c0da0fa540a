// fe_inv_host.cpp — host build of the division-step inversion (fe_inv.cuh)
// over the C stand-ins of ptx_emul.h, for tests/test_fe_inv_host.py.  TEST
// HARNESS ONLY.
#include <string.h>
#include "../../libftcrypto_gb300/csrc/fe_inv.cuh"

extern "C" void hi_fe_inv(uint32_t *out, const uint32_t *z, size_t n)
{
    for (size_t i = 0; i < n; ++i) {
        fe a, h;
        memcpy(a.v, z + 8 * i, 32);
        fe_inv(h, a);
        memcpy(out + 8 * i, h.v, 32);
    }
}
