// Donation ring: what its two counters say (EnumControl.q_head, q_tail), for the kernel and the CPU test.
#pragma once

#include "common.h"

namespace csm {

// Positions taken by waiting warps that no item has been reserved for.
CSM_HD uint32_t ring_unserved(uint32_t head, uint32_t tail) {
    const int32_t n = (int32_t)(tail - (head & ~CSM_QUEUE_CLOSED));
    return n > 0 ? (uint32_t)n : 0u;
}

// Warps that an item may be handed to.
CSM_HD uint32_t ring_wanted(uint32_t head, uint32_t tail) {
    return head & CSM_QUEUE_CLOSED ? 0u : ring_unserved(head, tail);
}

// Whether a warp that waits at `pos` may leave without an item, having closed the ring when its head was
// `head`: nobody has reserved its position, and nobody will.  Otherwise its item is on the way.
CSM_HD bool ring_may_leave(uint32_t head, uint32_t pos) {
    return (int32_t)(pos - (head & ~CSM_QUEUE_CLOSED)) >= 0;
}

}  // namespace csm
