// Buffers an entry point keeps between calls and only ever grows (engine.cu).
#pragma once

#include <stdint.h>

namespace fcw {

// Makes p hold at least `need` entries: 0, or the error of alloc(&p, need). The capacity follows the
// buffer at every step, so after an allocation that failed the next call, whatever its size, allocates
// again instead of using a buffer that is gone.
template <class T, class Alloc, class Free>
int grow_staging(T*& p, int64_t& cap, int64_t need, Alloc&& alloc, Free&& free) {
    if (p && cap >= need) return 0;
    if (p) free(p);
    p = nullptr;
    cap = 0;
    const int rc = alloc(&p, need);
    if (rc) {
        p = nullptr;
        return rc;
    }
    cap = need;
    return 0;
}

}  // namespace fcw
