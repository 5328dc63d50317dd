// Window search of a sorted list of adjacency entries: the index arithmetic, for host and device.
// A reader r(i) gives entry i of the list, for i < size only.  Positions and sizes are below 2^32,
// windows powers of two up to 2^31 (a list has fewer than 2^31 entries, one per vertex), so that a
// cursor and a window never wrap when added.
#pragma once

#include <stdint.h>

#include "common.h"

namespace csm {

constexpr uint32_t kWindowMin = 64u, kWindowMax = 1u << 31;

// First window of a search: about twice what 32 consecutive entries of a list of `short_size` span in one
// of `size`, a power of two of at least 64.  Where a list is 2^25 or more times as long as the other the
// window stays at 2^30 entries, and the search widens it where it has to.
CSM_HD uint32_t first_window(uint32_t size, uint32_t short_size) {
    uint32_t w = kWindowMin;
    const uint32_t per = short_size ? size / short_size : 0u;
    if (per == 0u) return w;
#ifdef __CUDA_ARCH__
    const uint32_t shift = 31u - (uint32_t)__clz(per);
#else
    const uint32_t shift = 31u - (uint32_t)__builtin_clz(per);
#endif
    return w << (shift < 24u ? shift : 24u);
}

// Window from position c0 on that holds the lower bound of `top`: w doubled until its last entry is at
// least `top` or past the end of the list.
template <typename R>
CSM_HD uint32_t window_for(const R &r, uint32_t size, uint32_t c0, uint32_t w, uint32_t top) {
    while (w < kWindowMax && c0 + w < size && r(c0 + w - 1u) < top) w <<= 1;
    return w;
}

// Lower bound of `key` in the window of w entries from c0 on (a lower bound past the window gives its last
// position).  Reads past the end count as large, so there is no data-dependent branch.
template <typename R>
CSM_HD uint32_t window_lower_bound(const R &r, uint32_t size, uint32_t c0, uint32_t w, uint32_t key) {
    uint32_t pos = c0;
    for (uint32_t s = w >> 1; s; s >>= 1) {
        const uint32_t p = pos + s - 1u;
        const uint32_t v = p < size ? r(p) : 0xFFFFFFFFu;
        if (v < key) pos += s;
    }
    return pos;
}

}  // namespace csm
