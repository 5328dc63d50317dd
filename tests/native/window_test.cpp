// Host check of the window search (gcsm-bu_b200/csrc/window.h) over the sizes a list can have, with a
// stand-in for the list: entry i is a function of i, reads outside the list or without end are caught.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "window.h"

namespace {

struct List {
    uint32_t size;
    uint32_t step;  // vertex of entry i: i * step + step - 1
    mutable int reads = 0;
    uint32_t operator()(uint32_t i) const {
        if (i >= size || ++reads > 200) {
            std::printf("FAIL entry %u of a list of %u, read %d\n", i, size, reads);
            std::exit(1);
        }
        return (i * step + step - 1) << 1 | (i & 1u);
    }
    uint32_t lower_bound(uint32_t key) const {  // first entry >= key (an even number: a vertex without flag)
        const uint64_t v = key >> 1, i = v < step - 1 ? 0 : (v - (step - 1) + step - 1) / step;
        return i < size ? (uint32_t)i : size;
    }
};

int checks = 0;

void check(const List &l, uint32_t short_size, uint32_t c0, uint32_t key, uint32_t top) {
    const uint32_t w0 = csm::first_window(l.size, short_size);
    l.reads = 0;
    const uint32_t w = csm::window_for(l, l.size, c0, w0, top);
    const uint32_t pos = csm::window_lower_bound(l, l.size, c0, w, key);
    const uint32_t want = l.lower_bound(key);
    // A key that is there is found; the position of any other is no later than its lower bound, which
    // keeps it good as the cursor of the next search.
    const bool there = want < l.size && want * l.step + l.step - 1 == key >> 1;
    if (w0 < 64 || (w & (w - 1)) != 0 || pos > want || (there && pos != want)) {
        std::printf("FAIL list of %u (step %u), other list of %u, from %u: key %u at %u, found at %u (windows %u, %u)\n",
                    l.size, l.step, short_size, c0, key >> 1, want, pos, w0, w);
        std::exit(1);
    }
    checks++;
}

}  // namespace

int main() {
    const uint32_t sizes[] = {1, 2, 31, 32, 63, 64, 65, 127, 4096, 100003, (1u << 26) - 1, 1u << 26, (1u << 26) + 1,
                              (1u << 30) - 1, 1u << 30, (1u << 30) + 7, (1u << 31) - 2, (1u << 31) - 1};
    const uint32_t shorts[] = {0, 1, 2, 31, 33, 1000, 1u << 20, 1u << 30};
    for (uint32_t size : sizes)
        for (uint32_t step = 1; (uint64_t)size * step < (1ull << 31) && step <= 3; step++)
            for (uint32_t short_size : shorts) {
                const List l{size, step};
                // A chunk's keys ascend from the cursor's entry on to `top`, which may lie past the list.
                for (uint64_t at : {0ull, 1ull, (unsigned long long)size / 3, (unsigned long long)size - 1})
                    for (uint64_t span : {0ull, 1ull, 31ull, 70ull, 5000ull, (unsigned long long)size / 2, (unsigned long long)size}) {
                        if (at >= size) continue;
                        const uint32_t c0 = (uint32_t)at;
                        const uint64_t lo = (uint64_t)c0 * step, hi = lo + span * step;
                        const uint32_t last = hi < (1ull << 31) - 1 ? (uint32_t)hi : (1u << 31) - 1;
                        for (uint64_t v : {lo, lo + 1, (lo + last) / 2, (uint64_t)last - 1, (uint64_t)last})
                            if (v >= lo && v <= last) check(l, short_size, c0, (uint32_t)v << 1, last << 1);
                    }
            }
    std::printf("ok %d searches\n", checks);
    return 0;
}
