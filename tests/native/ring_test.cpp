// CPU model of the donation ring's waiting and closing (gcsm-bu_b200/csrc/ring.h): threads stand in for
// warps, with the counters, the slot words and the steps of reserve_slots, publish_items and await_item
// (enumerate.cu).  The patience of a waiting thread is a few polls, so the ring is closed at every point of
// a launch.  Every item handed out is run exactly once, and a thread whose
// patience ends leaves without one.
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <thread>
#include <vector>

#include "ring.h"

namespace {

constexpr uint32_t kSlots = 32;

struct Launch {
    std::atomic<uint32_t> head{0}, tail{0}, active{0}, ticket{0}, closed{0}, handed{0}, run{0};
    std::atomic<uint64_t> seq[kSlots];
    uint32_t item[kSlots];  // pieces the item may still be split into
    uint32_t limit;
    explicit Launch(uint32_t l) : limit(l) {
        for (auto &s : seq) s = ~0ull;  // another launch's words
    }
};

bool hand_out(Launch &L, uint32_t pieces) {
    const uint32_t pos = L.head.load(), tail = L.tail.load();
    if (csm::ring_wanted(pos, tail) <= 0) return false;
    if (pos >= kSlots && L.seq[pos % kSlots].load() != pos) return false;
    uint32_t expect = pos;
    if (!L.head.compare_exchange_strong(expect, pos + 1)) return false;
    L.active.fetch_add(1);
    L.item[pos % kSlots] = pieces;
    L.seq[pos % kSlots].store(pos + 1);
    L.handed.fetch_add(1);
    return true;
}

void run(Launch &L, uint32_t pieces, uint32_t work) {
    for (; pieces; pieces--) {
        if (pieces > 1 && hand_out(L, pieces / 2)) pieces -= pieces / 2;
        for (volatile uint32_t i = 0; i < work; i = i + 1) {
        }
        L.run.fetch_add(1);
    }
}

// 1 = an item, 0 = over for this thread.
int await(Launch &L, uint32_t &pieces) {
    const uint32_t pos = L.tail.fetch_add(1);
    if (L.active.fetch_sub(1) == 1) {
        const uint32_t h = L.head.load() & ~CSM_QUEUE_CLOSED, n = csm::ring_unserved(h, L.tail.load());
        for (uint32_t i = 0; i < n && i < kSlots; i++) L.seq[(h + i) % kSlots].store(~1ull);
        return 0;
    }
    for (uint32_t polls = 0;;) {
        const uint64_t w = L.seq[pos % kSlots].load();
        if (w == pos + 1) break;
        if (w == ~1ull) return 0;
        if (++polls >= L.limit) {
            if (csm::ring_may_leave(L.head.fetch_or(CSM_QUEUE_CLOSED), pos)) {
                L.closed++;
                return 0;
            }
            polls = 0;  // its item is on the way
        }
        if (L.active.load() == 0 && L.seq[pos % kSlots].load() != pos + 1) return 0;
        std::this_thread::yield();
    }
    pieces = L.item[pos % kSlots];
    L.seq[pos % kSlots].store(pos + kSlots);
    return 1;
}

}  // namespace

int main() {
    uint64_t closed = 0, handed = 0;
    for (uint32_t limit : {1u, 2u, 5u, 40u, 1000000u})
        for (uint32_t rep = 0; rep < 150; rep++) {
            Launch L(limit);
            const uint32_t threads = 2 + rep % 7, pieces = 1 + 37 * (rep % 11), work = 1u << (rep % 13);
            std::vector<std::thread> th;
            for (uint32_t t = 0; t < threads; t++)
                th.emplace_back([&L, pieces, work] {
                    L.active.fetch_add(1);
                    uint32_t mine = L.ticket.fetch_add(1) == 0 ? pieces : 0;  // one ticket holds the launch's work
                    do run(L, mine, work);
                    while (await(L, mine));
                });
            for (auto &t : th) t.join();
            if (L.run != pieces) {
                std::printf("FAIL limit %u, run %u: %u of %u pieces run, %u handed out\n", limit, rep, L.run.load(), pieces,
                            L.handed.load());
                return 1;
            }
            closed += L.closed;
            handed += L.handed;
        }
    // The arithmetic at the ends: a closed ring hands out nothing, whatever the counters say.
    for (uint32_t h : {0u, 1u, 1000u, 0x7FFFFFFFu})
        for (uint32_t n : {0u, 1u, 5000u}) {
            const uint32_t t = h + n;
            if (csm::ring_wanted(h, t) != (int32_t)n || csm::ring_wanted(h | CSM_QUEUE_CLOSED, t) > 0 ||
                csm::ring_unserved(h | CSM_QUEUE_CLOSED, t) != n || !csm::ring_may_leave(h, h) ||
                csm::ring_may_leave(h | CSM_QUEUE_CLOSED, h - 1)) {
                std::printf("FAIL counters %u %u\n", h, n);
                return 1;
            }
        }
    if (closed < 20 || handed < 20) return std::printf("too little: %llu closed, %llu handed out\n", (unsigned long long)closed,
                                                         (unsigned long long)handed), 1;
    std::printf("ok, %llu left a closed ring, %llu items handed out\n", (unsigned long long)closed, (unsigned long long)handed);
    return 0;
}
