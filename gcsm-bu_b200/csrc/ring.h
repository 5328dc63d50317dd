// Donation ring: what its two counters say (EnumControl.q_head, q_tail), for the kernel and the CPU test.
#pragma once

#include "common.h"

namespace csm {

// Warps that an item may be handed to, as a signed number: not above zero when none waits.  The closing bit
// of the head takes 2^31 off, so a closed ring needs no test of its own.
CSM_HD int32_t ring_wanted(uint32_t head, uint32_t tail) { return (int32_t)(tail - head); }

// Positions taken by waiting warps that no item has been reserved for, in a closed ring too.
CSM_HD uint32_t ring_unserved(uint32_t head, uint32_t tail) {
    const int32_t n = ring_wanted(head & ~CSM_QUEUE_CLOSED, tail);
    return n > 0 ? (uint32_t)n : 0u;
}

// Whether a warp that waits at `pos` may leave without an item, having closed the ring when its head was
// `head`: nobody has reserved its position, and nobody will.  Otherwise its item is on the way.
CSM_HD bool ring_may_leave(uint32_t head, uint32_t pos) {
    return (int32_t)(pos - (head & ~CSM_QUEUE_CLOSED)) >= 0;
}

}  // namespace csm
