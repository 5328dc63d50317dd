// Persistent warp-DFS enumeration of incremental matches.
//
// Replaces the reference's enumeration kernels: write_initial_partial_results
// (kernels/enumeration.cu:24-79), extendBFSDFSRegTwo (enumeration.cu:407-781),
// gamma_enumerate with its work stealing (kernels/gamma_enumeration.cu:209-880) and the
// Cartesian-product flattening GetNumTree / enumerateCartesianProductTree
// (kernels/cartesian_product.cu:193-284).
//
// One launch covers every (query, updated query edge) plan of a batch.  A warp owns one work
// item at a time and walks its subtree depth first: at each level the candidates are the
// entries of the smallest backward-neighbour list (the pivot), filtered 32 at a time by the
// lanes (flag rule, NLF bitmap, injectivity, membership in the other backward lists by binary
// search) and compacted with ballot/popc into a per-level shared-memory buffer.
//
// Counting rule of the per-query-edge decomposition (technique_permutation.h:125-212): for the
// plan of query edge i the starting edge is a batch edge; an edge matched to a query edge with
// index > i must not be a batch edge; edges of query edges < i may be either.  Every new
// embedding is counted exactly once, at the largest query-edge index it maps to a batch edge.
//
// Load balance: warps first take seed chunks from a ticket counter.  A warp that runs out of
// work takes the next position of a global ring and waits there; a busy warp that sees waiting
// positions hands out pending work of its shallowest level that has some: the candidate range in as
// many parts as warps wait (at most 31), or the buffered sibling candidates, one item each.  Every
// wait is bounded: a warp whose bound runs out closes the ring and leaves (ring.h).  A warp never
// waits on another warp's progress to finish its own items.
//
// Tail vertices (the last of the order, pairwise non-adjacent, all their neighbours matched before
// them) are not enumerated: the number of their injective assignments is computed by
// inclusion-exclusion from the sizes of their lists and of the lists' intersections.
#include <cuda_runtime.h>

#include "kernels.cuh"
#include "ring.h"
#include "window.h"

namespace csm {

namespace {

struct __align__(16) WarpState {
    uint32_t f[CSM_MAXQV];
    uint32_t buf[CSM_MAXQV][CSM_WARP];
    uint32_t lo[CSM_MAXQV];
    uint32_t hi[CSM_MAXQV];
    uint32_t base[CSM_MAXQV];
    // Backward-neighbour lists of every level, in one flat array: level d uses slots
    // [lv[d].bn_base, lv[d].bn_base + nbn) (all levels together hold at most CSM_MAXQE lists).
    uint32_t poff[CSM_MAXQE];
    uint32_t psz[CSM_MAXQE];
    uint32_t cur[CSM_MAXQE];   // per probe list: entries before it are below the next chunk
    uint8_t bnb[CSM_MAXQV];
    uint32_t nlf[CSM_MAXQV];
    uint16_t oldm[CSM_MAXQV];
    uint16_t exm[CSM_MAXQV];   // per level: prefix depths the candidate may coincide with
    uint8_t nbuf[CSM_MAXQV];
    uint8_t pos[CSM_MAXQV];
    uint8_t piv[CSM_MAXQV];
    uint8_t nbn[CSM_MAXQV];
    uint32_t t_off[CSM_TAIL_MAXKEYS];
    uint32_t t_size[CSM_TAIL_MAXKEYS];
    uint32_t t_flag[CSM_TAIL_MAXKEYS];
    uint32_t t_excl[CSM_TAIL_MAXKEYS];
    uint32_t t_cur[CSM_TAIL_MAXKEYS];  // cursor of a probed list while an intersection is counted
    unsigned long long msize[CSM_TAIL_MAXMASKS];
    // Lane-parallel tail: per key whose parent is matched before the counting level, its
    // list and the list size left after the flag rule and the shared prefix.
    uint32_t ts_off[CSM_TAIL_MAXKEYS];
    uint32_t ts_size[CSM_TAIL_MAXKEYS];
    uint32_t ts_base[CSM_TAIL_MAXKEYS];
    uint32_t ts_cur[CSM_TAIL_MAXKEYS];  // cursor of the shared list over ascending candidates
    uint32_t item_plan;
    uint32_t item_depth;
    uint32_t item_lo;
    uint32_t item_hi;
    // Shared last level (DevPlan.shared_last): its candidate count for the current prefix
    // f[0..n-3], and whether it is being counted (1) or known (2).
    unsigned long long sl_count;
    uint32_t sl_state;
    // Kept intersections of the counting level (DevTail.mask_set): entries held, or kSetOpen while
    // there is none for the current prefix.
    uint32_t set_n[CSM_SETS];
};

constexpr uint32_t kSetOpen = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t warp_min_index(uint32_t v, uint32_t lane) {
    // Returns the lane holding the smallest v (smallest lane on ties).
    unsigned long long key = ((unsigned long long)v << 5) | lane;
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
        key = other < key ? other : key;
    }
    return (uint32_t)(key & 31u);
}

__device__ __forceinline__ const uint32_t *bitmap(const EnumParams &P, uint32_t id) {
    return P.bits + (size_t)id * P.words;
}

// Records the launch's first failed consistency check (the caller skips what failed it).
__device__ void record_bad(const EnumParams &P, uint32_t where, uint32_t a, uint32_t b, uint32_t c) {
    if (atomicCAS(&P.ctrl->bad_where, 0u, where) == 0u) {
        P.ctrl->bad_a = a;
        P.ctrl->bad_b = b;
        P.ctrl->bad_c = c;
    }
    atomicOr(&P.ctrl->error, CSM_ERRBIT_CORRUPT);
}

// {offset, size} of list (rel, v), checked against the vertex range and the pool; a list that
// fails is recorded and read as empty.
__device__ __forceinline__ uint2 list_of(const EnumParams &P, uint32_t rel, uint32_t v, uint32_t level) {
    if (v >= P.g.V || rel >= P.g.R) {
        record_bad(P, CSM_BAD_LIST, v, rel, 0x80000000u | level);
        return make_uint2(0u, 0u);
    }
    const uint2 ms = __ldg(P.g.meta + (size_t)rel * P.g.V + v);
    if ((unsigned long long)ms.x + ms.y > P.g.pool_cap) {
        record_bad(P, CSM_BAD_LIST, ms.x, ms.y, level);
        return make_uint2(0u, 0u);
    }
    return ms;
}

// First index in [lo, hi) of the sorted list L whose entry is >= key2, found by the whole warp
// with 32-ary search: each round reads 32 evenly spaced entries and keeps the bracket that
// holds the answer, so a list of n entries costs about log32(n) dependent reads.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t *L, uint32_t lo, uint32_t hi, uint32_t key2,
                                                     uint32_t lane) {
    while (hi - lo > 32) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t p = lo + (lane + 1) * step - 1;
        const uint32_t v = p < hi ? __ldg(L + p) : 0xFFFFFFFFu;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, v < key2));
        const uint32_t nhi = lo + (c + 1) * step - 1;
        lo = lo + c * step;
        if (nhi < hi) hi = nhi;
    }
    const uint32_t p = lo + lane;
    const uint32_t v = p < hi ? __ldg(L + p) : 0xFFFFFFFFu;
    return lo + __popc(__ballot_sync(0xffffffffu, v < key2));
}

// Entries of a list in device memory (window.h).
struct ListReader {
    const uint32_t *L;
    __device__ __forceinline__ uint32_t operator()(uint32_t i) const { return __ldg(L + i); }
};

// Entry of the sorted list L that names this lane's vertex (key = vertex << 1), or 0xFFFFFFFF.  The
// lanes' keys ascend, `top` is the one of lane `last` and the largest; c0 is a position no lane's
// entry lies before, and moves on to where the next keys start.  All lanes search a window from c0 on,
// w0 entries wide and doubled until it holds `top`.  The window is a power of two and reads past the
// end count as large, so the search has no data-dependent branch: log2(window) dependent reads, most
// of them from a few cache lines.  In the level scan it took the place of a register window, shuffles
// and a warp search (four queries at 16,411 updates 39.6 -> 34.1 ms, 1M on 43M edges 55.8 -> 52.1 ms).
__device__ __forceinline__ uint32_t window_find(const uint32_t *L, uint32_t size, uint32_t &c0, uint32_t w0, uint32_t key,
                                                uint32_t top, uint32_t last) {
    const ListReader r{L};
    const uint32_t pos = window_lower_bound(r, size, c0, window_for(r, size, c0, w0, top), key);
    const uint32_t e = pos < size ? __ldg(L + pos) : 0xFFFFFFFFu;
    c0 = __shfl_sync(0xffffffffu, pos, last);
    return (e & ~1u) == key ? e : 0xFFFFFFFFu;
}

// Lower bound of key2 among the 32 register-held window entries (sorted, padded with ~0).
__device__ __forceinline__ uint32_t shfl_lower_bound(uint32_t win, uint32_t key2) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, win, pos + step - 1) < key2) pos += step;
    return pos;
}

// Flagged entries of list (rel, x) in this phase (batch edges of that list), 0 if none.
__device__ __forceinline__ uint32_t flagged_in_list(const EnumParams &P, uint32_t rel, uint32_t x) {
    // Lists of vertices no batch key starts from hold no batch entry: skip the key search.
    if (P.touched != nullptr && !((__ldg(P.touched + (x >> 5)) >> (x & 31)) & 1u)) return 0u;
    const unsigned long long lk = P.kl.list_key(rel, x);
    const uint32_t h = find_list_head(P.keys, P.m, P.kl, lk);
    return (h < P.m && P.kl.list_of(__ldg(P.keys + h)) == lk) ? __ldg(P.seg_flagged + h) : 0u;
}

// Whether entry e of a tail key's list counts under the key's rule (CSM_KEY_*).
__device__ __forceinline__ bool key_counts(uint32_t rule, uint32_t e) {
    return rule == CSM_KEY_ANY || (e & 1u) == (rule >> 1);
}

// Entries of list (rel, x), of `size` entries, that count under a tail key's rule.
__device__ __forceinline__ uint32_t key_entries(const EnumParams &P, uint32_t rel, uint32_t x, uint32_t size,
                                                uint32_t rule) {
    if (rule == CSM_KEY_ANY) return size;
    const uint32_t batch = flagged_in_list(P, rel, x);
    return rule == CSM_KEY_OLD ? size - batch : batch;
}

// Lane-parallel tail, shared part: for the counting level d = tail_start - 1 and the current
// prefix f[0..d-1], every tail key whose parent is matched before depth d gets its list and
// the number of its entries the leaves may still use given that prefix.
__device__ void prep_tail_shared(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d) {
    const uint32_t lane = lane_id();
    const DevTail *T = &pl->tail;
    const uint32_t nkeys = __ldg(&T->nkeys);
    if (lane < nkeys && ((__ldg(&T->single) >> lane) & 1u)) {
        const uint32_t pd = __ldg(&T->key_parent[lane]);
        if (pd < d) {
            const uint32_t rel = __ldg(&T->key_rel[lane]);
            const uint32_t rule = __ldg(&T->key_old[lane]);
            const uint32_t x = S.f[pd];
            const uint2 ms = list_of(P, rel, x, 100 + d);
            uint32_t left = key_entries(P, rel, x, ms.y, rule);
            const uint32_t excl = __ldg(&T->key_excl[lane]);
            for (uint32_t j = 0; j < d; j++) {
                if (j == pd || !((excl >> j) & 1u)) continue;
                const uint32_t e = find_entry(P.g.pool + ms.x, ms.y, S.f[j]);
                if (e != 0xFFFFFFFFu && key_counts(rule, e)) left--;
            }
            S.ts_off[lane] = ms.x;
            S.ts_size[lane] = ms.y;
            S.ts_base[lane] = left;
            S.ts_cur[lane] = 0;
        }
    }
    __syncwarp();
}

// Lane-parallel tail, per lane: what is left of tail key k's list for the prefix f[0..d-1] + v, where
// v is this lane's candidate at depth d (for d == 1 the prefix is the seed (x0, v)).
__device__ __forceinline__ uint32_t tail_key_left(const uint32_t *ts_base, const uint32_t *f, const EnumParams &P,
                                                  const DevTail *T, uint32_t k, uint32_t d, uint32_t x0, uint32_t v,
                                                  uint32_t shared_hit, uint32_t &probes) {
    const uint32_t pd = __ldg(&T->key_parent[k]);
    // Shared list: only this lane's candidate may still sit in it (looked up by the warp beforehand,
    // bit k of shared_hit).
    if (pd < d && d >= 2) return ts_base[k] - ((shared_hit >> k) & 1u);
    const uint32_t rel = __ldg(&T->key_rel[k]);
    const uint32_t rule = __ldg(&T->key_old[k]);
    const uint32_t x = (pd == d) ? v : x0;  // d >= 2: pd == d; d == 1: parent 0 or 1
    const uint2 ms = list_of(P, rel, x, 200 + d);
    uint32_t left = key_entries(P, rel, x, ms.y, rule);
    const uint32_t excl = __ldg(&T->key_excl[k]);
    for (uint32_t j = 0; j <= d; j++) {
        if (j == pd || !((excl >> j) & 1u)) continue;
        const uint32_t z = (j == d) ? v : (d == 1 ? x0 : f[j]);
        const uint32_t e = find_entry(P.g.pool + ms.x, ms.y, z);
        probes++;
        if (e != 0xFFFFFFFFu && key_counts(rule, e)) left--;
    }
    return left;
}

// Value of a tail polynomial whose masks are single keys (mask mi stands for key ffs(mask) - 1), over
// the tail classes in `classes`.
__device__ __forceinline__ unsigned long long tail_product(const EnumParams &P, const DevPlan *pl,
                                                           const uint32_t (&ksize)[CSM_TAIL_MAXKEYS], uint32_t classes) {
    const DevTail *T = &pl->tail;
    unsigned long long total = 1;
    if (classes == 0xFFu && __ldg(&T->product)) {
        const uint32_t nkeys = __ldg(&T->nkeys);
#pragma unroll 1
        for (uint32_t k = 0; k < nkeys; k++) total *= ksize[k];
        return total;
    }
    const DevTailTerm *terms = P.terms + pl->term_begin;
    const uint32_t nclasses = __ldg(&T->nclasses);
    for (uint32_t c = 0; c < nclasses; c++) {
        if (!((classes >> c) & 1u)) continue;
        unsigned long long s = 0;
        const uint32_t tb = __ldg(&T->class_term_begin[c]), te = __ldg(&T->class_term_begin[c + 1]);
        for (uint32_t t = tb; t < te; t++) {
            unsigned long long prod = (unsigned long long)__ldg(&terms[t].coef);
            const uint32_t nf = __ldg(&terms[t].nf);
            for (uint32_t j = 0; j < nf; j++) {
                prod *= ksize[__ffs(__ldg(&T->mask[__ldg(&terms[t].f[j])])) - 1];
            }
            s += prod;
        }
        total *= s;
    }
    return total;
}

// Lane-parallel tail, per lane: the tail count of the prefix f[0..d-1] + v.  Only for plans whose
// masks are single keys (no list intersections).
__device__ unsigned long long tail_count_lane(const uint32_t *ts_base, const uint32_t *f, const EnumParams &P,
                                              const DevPlan *pl,
                                              uint32_t d, uint32_t x0, uint32_t v, uint32_t shared_hit,
                                              uint32_t &probes) {
    const DevTail *T = &pl->tail;
    const uint32_t nkeys = __ldg(&T->nkeys);
    uint32_t ksize[CSM_TAIL_MAXKEYS];
#pragma unroll 1
    for (uint32_t k = 0; k < nkeys; k++) {
        ksize[k] = tail_key_left(ts_base, f, P, T, k, d, x0, v, shared_hit, probes);
    }
    return tail_product(P, pl, ksize, 0xFFu);
}

// Entries that two sorted lists share, each under its rule (CSM_KEY_*).  The warp scans the shorter
// list 32 entries at a time; every lane searches its entry in the longer one (window_find).
// KEEP: the vertices found, without the prefix vertices f[j] with bit j of `excl`, go to `out`, and
// the scan starts at entry `from` of the shorter list and stops (returning where in `from`) before a
// chunk that might not fit in CSM_SET_CAP entries.
template <bool KEEP>
__device__ uint32_t intersect_lists(const EnumParams &P, uint2 a, uint32_t rule_a, uint2 b, uint32_t rule_b,
                                    const uint32_t *f, uint32_t excl, uint32_t *out, uint32_t &from) {
    const uint32_t lane = lane_id();
    if (b.y < a.y) {
        const uint2 t = a;
        a = b;
        b = t;
        const uint32_t r = rule_a;
        rule_a = rule_b;
        rule_b = r;
    }
    const uint32_t *A = P.g.pool + a.x, *B = P.g.pool + b.x;
    const uint32_t w0 = first_window(b.y, a.y);
    uint32_t cnt = 0, c0 = 0, base = KEEP ? from : 0u;
    for (; base < a.y && c0 < b.y; base += 32) {
        if (KEEP && cnt > CSM_SET_CAP - 32u) break;
        const uint32_t i = base + lane;
        const uint32_t e = i < a.y ? __ldg(A + i) : 0xFFFFFFFFu;
        const uint32_t last = a.y - base < 32u ? a.y - base - 1u : 31u;
        const uint32_t g = window_find(B, b.y, c0, w0, e & ~1u, __shfl_sync(0xffffffffu, e & ~1u, last), last);
        bool hit = i < a.y && g != 0xFFFFFFFFu && key_counts(rule_a, e) && key_counts(rule_b, g);
        if (KEEP)
            for (uint32_t em = excl; hit && em; em &= em - 1) hit = f[__ffs(em) - 1] != (e >> 1);
        const uint32_t hits = __ballot_sync(0xffffffffu, hit);
        if (KEEP && hit) out[cnt + __popc(hits & ((1u << lane) - 1u))] = e >> 1;
        cnt += __popc(hits);
    }
    if (KEEP) {
        from = c0 < b.y ? base : a.y;
        __syncwarp();
    }
    return cnt;
}

// Slot of the pair table for (a, b) under `tag`.
__device__ __forceinline__ uint4 *pair_slot(const EnumParams &P, uint32_t a, uint32_t b, uint32_t tag) {
    uint32_t h = a * 0x9E3779B1u ^ (b * 0x85EBCA77u + tag * 0xC2B2AE3Du);
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 13;
    return P.pairs + (h & (P.pair_slots - 1u));
}

// A table entry is read and written as one 128-bit access, so a reader sees an entry of one writer.
__device__ __forceinline__ uint4 load_pair(const uint4 *slot) {
    unsigned long long lo, hi;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(lo), "=l"(hi)
                 : "l"(slot)
                 : "memory");
    return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

__device__ __forceinline__ void store_pair(uint4 *slot, uint32_t a, uint32_t b, uint32_t tag, uint32_t count) {
    const unsigned long long lo = (unsigned long long)b << 32 | a, hi = (unsigned long long)count << 32 | tag;
    asm volatile("{ .reg .b128 t; mov.b128 t, {%0, %1}; st.relaxed.gpu.global.b128 [%2], t; }" ::"l"(lo), "l"(hi), "l"(slot)
                 : "memory");
}

// Size of the intersection of lists (ra, a) and (rb, b) under their rules, for every lane with ok set:
// from the pair table under signature `sig`, or counted by the warp and put there.  `uniform`: a and b
// are the same for all lanes.
__device__ uint32_t pair_lookup(const EnumParams &P, uint32_t sig, uint32_t ra, uint32_t rule_a, uint32_t a, uint32_t rb,
                                uint32_t rule_b, uint32_t b, bool ok, bool uniform, uint32_t where) {
    const uint32_t lane = lane_id();
    const uint32_t tag = P.ctrl->pair_phase << 12 | (sig & 0xFFFu);
    uint32_t ta = a, tb = b;  // lists of one relation and rule: either order is the same pair
    if (ra == rb && rule_a == rule_b && b < a) {
        ta = b;
        tb = a;
    }
    uint4 *slot = pair_slot(P, ta, tb, tag);
    uint32_t count = 0;
    bool miss = false;
    if (ok) {
        const uint4 e = load_pair(slot);
        miss = e.x != ta || e.y != tb || e.z != tag;
        count = e.w;
    }
    uint32_t need = __ballot_sync(0xffffffffu, miss);
    if (need) {
        uint2 la = make_uint2(0u, 0u), lb = la;
        if (miss) {
            la = list_of(P, ra, a, where);
            lb = list_of(P, rb, b, where);
        }
        // The shorter list of every missing pair; all of them end to end where they are short (64
        // entries on average), so that pairs over short lists share the warp's lanes instead of taking
        // a pass each.  Pairs that do not depend on the candidate are one pair for all lanes.
        const bool swap = lb.y < la.y;
        const uint2 sh = swap ? lb : la, lg = swap ? la : lb;
        uint32_t incl = sh.y;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        if (!uniform && total <= 64u * __popc(need)) {
            const uint32_t start = incl - sh.y;
            uint32_t mine = 0;
            for (uint32_t g0 = 0; g0 < total; g0 += 32) {
                const uint32_t g = g0 + lane;
                // The pair of position g: the first lane whose inclusive prefix exceeds g.
                uint32_t j = 0;
#pragma unroll
                for (uint32_t step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, j + step - 1) <= g) j += step;
                const uint32_t first = __shfl_sync(0xffffffffu, start, j), off = __shfl_sync(0xffffffffu, sh.x, j);
                const uint32_t loff = __shfl_sync(0xffffffffu, lg.x, j), size = __shfl_sync(0xffffffffu, lg.y, j);
                const bool sw = __shfl_sync(0xffffffffu, swap, j);
                bool hit = false;
                if (g < total) {
                    const uint32_t e = __ldg(P.g.pool + off + (g - first));
                    if (key_counts(sw ? rule_b : rule_a, e)) {
                        const uint32_t x = find_entry(P.g.pool + loff, size, e >> 1);
                        hit = x != 0xFFFFFFFFu && key_counts(sw ? rule_a : rule_b, x);
                    }
                }
                const uint32_t hits = __ballot_sync(0xffffffffu, hit);
                const uint32_t lo = start > g0 ? start - g0 : 0u, hi = incl > g0 ? incl - g0 : 0u;
                if (lo < 32u && hi > lo)
                    mine += __popc(hits & (0xFFFFFFFFu << lo) & (hi >= 32u ? 0xFFFFFFFFu : (1u << hi) - 1u));
            }
            if (miss) {
                count = mine;
                store_pair(slot, ta, tb, tag, mine);
            }
            need = 0;
        }
        while (need) {
            const uint32_t l = __ffs(need) - 1;
            const uint32_t va = __shfl_sync(0xffffffffu, a, l), vb = __shfl_sync(0xffffffffu, b, l);
            const uint2 xa = make_uint2(__shfl_sync(0xffffffffu, la.x, l), __shfl_sync(0xffffffffu, la.y, l));
            const uint2 xb = make_uint2(__shfl_sync(0xffffffffu, lb.x, l), __shfl_sync(0xffffffffu, lb.y, l));
            uint32_t from = 0;
            const uint32_t c = intersect_lists<false>(P, xa, rule_a, xb, rule_b, nullptr, 0u, nullptr, from);
            const bool same = miss && a == va && b == vb;
            if (same) count = c;
            if (lane == l) store_pair(slot, ta, tb, tag, c);
            need &= ~__ballot_sync(0xffffffffu, same);
        }
    }
    return count;
}

// Size of the pair mask mi for this lane's prefix f[0..d-1] + cand (where ok).  The table holds the
// intersection of the two lists under their rules; the prefix vertices of the mask's label that sit in
// both are taken off here.
__device__ uint32_t pair_size(const WarpState &S, const EnumParams &P, const DevTail *T, uint32_t mi, uint32_t d, bool ok,
                              uint32_t cand) {
    const uint32_t mask = __ldg(&T->mask[mi]), sig = __ldg(&T->mask_pair[mi]);
    uint32_t ka = __ffs(mask) - 1, kb = 31 - __clz(mask);
    if (sig & CSM_PAIR_SWAP) {
        const uint32_t t = ka;
        ka = kb;
        kb = t;
    }
    const uint32_t pa = __ldg(&T->key_parent[ka]), pb = __ldg(&T->key_parent[kb]);
    const uint32_t ra = __ldg(&T->key_rel[ka]), rb = __ldg(&T->key_rel[kb]);
    const uint32_t rule_a = __ldg(&T->key_old[ka]), rule_b = __ldg(&T->key_old[kb]);
    const uint32_t a = pa == d ? cand : S.f[pa], b = pb == d ? cand : S.f[pb];
    uint32_t count = pair_lookup(P, sig, ra, rule_a, a, rb, rule_b, b, ok, pa != d && pb != d, 1000 + d);
    uint32_t excl = __ldg(&T->key_excl[ka]) & ((2u << d) - 1u) & ~(1u << pa) & ~(1u << pb);
    if (excl && ok) {
        const uint2 la = list_of(P, ra, a, 1100 + d), lb = list_of(P, rb, b, 1100 + d);
        for (; excl; excl &= excl - 1) {
            const uint32_t j = __ffs(excl) - 1, z = j == d ? cand : S.f[j];
            const uint32_t ea = find_entry(P.g.pool + la.x, la.y, z);
            if (ea == 0xFFFFFFFFu || !key_counts(rule_a, ea)) continue;
            const uint32_t eb = find_entry(P.g.pool + lb.x, lb.y, z);
            if (eb != 0xFFFFFFFFu && key_counts(rule_b, eb)) count--;
        }
    }
    return count;
}

// Size of the three-key mask mi for this lane's prefix f[0..d-1] + cand (where ok).  The intersection
// of the two keys above the counting level is the same for all of the level's candidates: it is made
// once and kept (a few dozen vertices as a rule), and the warp then looks up all (candidate, kept
// vertex) pairs of the chunk, 32 at a time, in the candidates' lists of the third key.  Before, a tail
// count scanned all three lists for every candidate (65,536 updates, dense query: 51 -> 26 ms).
__device__ uint32_t set_size(WarpState &S, const EnumParams &P, const DevTail *T, uint32_t mi, uint32_t d, bool ok,
                             uint32_t cand) {
    const uint32_t lane = lane_id();
    const uint32_t set = __ldg(&T->mask_set[mi]);
    const uint32_t slot = set & 7u, ka = (set >> 3) & 7u, kb = (set >> 6) & 7u, kc = (set >> 9) & 7u;
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint32_t *kept = P.sets + ((size_t)slot * gridDim.x * (blockDim.x >> 5) + warp) * CSM_SET_CAP;
    const uint32_t pc = __ldg(&T->key_parent[kc]), rule_c = __ldg(&T->key_old[kc]);
    uint2 list = make_uint2(0u, 0u);
    if (ok) list = list_of(P, __ldg(&T->key_rel[kc]), pc == d ? cand : S.f[pc], 1200 + d);
    const uint32_t excl = __ldg(&T->key_excl[kc]);
    const uint32_t oks = __ballot_sync(0xffffffffu, ok);
    const uint32_t nok = __popc(oks), rank = __popc(oks & ((1u << lane) - 1u));
    __syncwarp();
    if (ok) S.buf[d][rank] = lane;  // the level's buffer is not in use: its candidates are counted here
    __syncwarp();
    uint32_t count = 0, from = 0, n = S.set_n[slot];
    bool more = true;
    while (more) {
        if (n == kSetOpen) {
            const uint2 a = list_of(P, __ldg(&T->key_rel[ka]), S.f[__ldg(&T->key_parent[ka])], 1200 + d);
            const uint2 b = list_of(P, __ldg(&T->key_rel[kb]), S.f[__ldg(&T->key_parent[kb])], 1200 + d);
            const uint32_t start = from;
            n = intersect_lists<true>(P, a, __ldg(&T->key_old[ka]), b, __ldg(&T->key_old[kb]), S.f,
                                      excl & ((1u << d) - 1u), kept, from);
            more = from < (a.y < b.y ? a.y : b.y);
            if (lane == 0 && start == 0 && !more) S.set_n[slot] = n;  // all of it
        } else {
            more = false;
        }
        const uint32_t total = n * nok;
        for (uint32_t g0 = 0; g0 < total; g0 += 32) {
            const uint32_t g = g0 + lane, r = n ? g / n : 0u;
            const bool in = g < total;
            const uint32_t src = in ? S.buf[d][r] : 0u;
            const uint32_t off = __shfl_sync(0xffffffffu, list.x, src), size = __shfl_sync(0xffffffffu, list.y, src);
            const uint32_t c = __shfl_sync(0xffffffffu, cand, src);
            bool hit = false;
            if (in) {
                const uint32_t w = kept[g - r * n];
                const uint32_t e = find_entry(P.g.pool + off, size, w);
                hit = e != 0xFFFFFFFFu && key_counts(rule_c, e) && !(((excl >> d) & 1u) && w == c);
            }
            const uint32_t hits = __ballot_sync(0xffffffffu, hit);
            // This lane's candidate has positions [rank * n, rank * n + n) of the pairs.
            const uint32_t s0 = rank * n, s1 = s0 + n;
            const uint32_t lo = s0 > g0 ? s0 - g0 : 0u, hi = s1 > g0 ? s1 - g0 : 0u;
            if (ok && lo < 32u && hi > lo)
                count += __popc(hits & (0xFFFFFFFFu << lo) & (hi >= 32u ? 0xFFFFFFFFu : (1u << hi) - 1u));
        }
        if (more) n = kSetOpen;
    }
    __syncwarp();
    return count;
}

// Lane-parallel tail with pair masks (DevTail.pair_par), counting level d >= 2: the tail count of the
// prefix f[0..d-1] + cand for every lane with ok set (0 for the others).  A pair of data vertices
// recurs under many prefixes — the lists of two vertices intersect the same whatever was matched
// between them — so most sizes are one table read instead of a scan of two lists (98% on the dense
// queries of the 43M-edge graph, whose 1M-update batch and inverse went from 356 to 104 ms).
__device__ unsigned long long tail_count_pairs(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d,
                                               bool ok, uint32_t cand, uint32_t shared_hit, uint32_t &probes) {
    const DevTail *T = &pl->tail;
    const uint32_t nmasks = __ldg(&T->nmasks);
    uint32_t msize[CSM_PAIR_MAXMASKS];
    unsigned long long total = ok ? 1 : 0;
    // A loop, like those over tail keys, although the sizes then live in local memory: unrolled, this
    // function held eight copies of the three cases, and the kernel waited for instructions more than
    // half of the time (no_instruction 16.5 of 31 cycles per issue, 65,536 updates with a dense query):
    // 22.3 -> 16.3 ms there, 1M on 43M edges 52.2 -> 38.9 ms.
#pragma unroll 1
    for (uint32_t mi = 0; mi < nmasks; mi++) {
        uint32_t size = 0;
        if (__ldg(&T->mask_pair[mi]) != CSM_NO_PAIR) {
            size = pair_size(S, P, T, mi, d, ok, cand);
        } else if (__ldg(&T->mask_set[mi]) != CSM_NO_SET) {
            size = set_size(S, P, T, mi, d, ok, cand);
        } else if (ok) {
            size = tail_key_left(S.ts_base, S.f, P, T, __ffs(__ldg(&T->mask[mi])) - 1, d, 0, cand, shared_hit, probes);
        }
        msize[mi] = size;
        total *= size;
    }
    if (__ldg(&T->product)) return total;
    total = ok ? 1 : 0;
    const DevTailTerm *terms = P.terms + pl->term_begin;
    const uint32_t nclasses = __ldg(&T->nclasses);
    for (uint32_t c = 0; c < nclasses; c++) {
        unsigned long long s = 0;
        const uint32_t tb = __ldg(&T->class_term_begin[c]), te = __ldg(&T->class_term_begin[c + 1]);
        for (uint32_t t = tb; t < te; t++) {
            unsigned long long prod = (unsigned long long)__ldg(&terms[t].coef);
            const uint32_t nf = __ldg(&terms[t].nf);
            for (uint32_t j = 0; j < nf; j++) {
                prod *= msize[__ldg(&terms[t].f[j])];
            }
            s += prod;
        }
        total *= s;
    }
    return total;
}

// Sets up level d for the current prefix: the backward-neighbour lists and the pivot.
__device__ void enter_level(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d, uint32_t rlo,
                            uint32_t rhi) {
    const uint32_t lane = lane_id();
    const DevLevel *lv = &pl->lv[d];
    const uint32_t nbn = __ldg(&lv->nbn);
    uint32_t sz = 0xFFFFFFFFu;
    if (lane < nbn) {
        const uint32_t rel = __ldg(&lv->bn_rel[lane]);
        const uint32_t dep = __ldg(&lv->bn_depth[lane]);
        const uint32_t v = S.f[dep];
        const uint2 ms = list_of(P, rel, v, d);
        const uint32_t slot = __ldg(&lv->bn_base) + lane;
        S.poff[slot] = ms.x;
        S.psz[slot] = ms.y;
        S.cur[slot] = 0;
        sz = ms.y;
    }
    const uint32_t piv = warp_min_index(sz, lane);
    __syncwarp();
    if (lane == 0) {
        S.piv[d] = (uint8_t)piv;
        S.nbn[d] = (uint8_t)nbn;
        const uint32_t bb = __ldg(&lv->bn_base);
        S.bnb[d] = (uint8_t)bb;
        S.base[d] = S.poff[bb + piv];
        const uint32_t psize = S.psz[bb + piv];
        S.lo[d] = rlo;
        S.hi[d] = rhi < psize ? rhi : psize;
        S.nbuf[d] = 0;
        S.pos[d] = 0;
        S.oldm[d] = __ldg(&lv->old_mask);
        S.nlf[d] = __ldg(&lv->nlf_bitmap);
        S.exm[d] = __ldg(&lv->excl_mask);
    }
    if (lane < CSM_SETS && d + 1 == pl->tail_start) S.set_n[lane] = kSetOpen;
    __syncwarp();
    if (d + 1 == pl->tail_start && pl->tail_start < pl->n && (pl->tail.lane_par || pl->tail.pair_par))
        prep_tail_shared(S, P, pl, d);
}

// Size of the intersection of the tail lists in `mask` (at least two), each under its flag rule,
// without the prefix vertices f[0..E-1]: the warp scans the smallest list 32 entries at a time.
// A chunk's entries ascend, so every other list keeps a cursor: the 32 entries at the cursor
// are read with one coalesced load and shuffles find each candidate; when the chunk reaches past
// them, a 32-ary warp search brackets the window and lanes search inside it.
__device__ uint32_t tail_intersection(WarpState &S, const EnumParams &P, const DevTail *T, uint32_t nkeys,
                                      uint32_t mask, uint32_t E, uint32_t &probes) {
    const uint32_t lane = lane_id();
    uint32_t k0 = 0, best = 0xFFFFFFFFu;
    for (uint32_t k = 0; k < nkeys; k++)
        if (((mask >> k) & 1u) && S.t_size[k] < best) {
            best = S.t_size[k];
            k0 = k;
        }
    if (lane < nkeys) S.t_cur[lane] = 0;
    __syncwarp();
    const uint32_t rule0 = __ldg(&T->key_old[k0]);
    const uint32_t excl = __ldg(&T->key_excl[k0]) & ((1u << E) - 1u);  // the keys of a mask share their label
    uint32_t cnt = 0;
    for (uint32_t base = 0; base < best; base += 32) {
        const uint32_t idx = base + lane;
        bool ok = idx < best;
        uint32_t w = 0;
        if (ok) {
            const uint32_t e = __ldg(P.g.pool + S.t_off[k0] + idx);
            w = e >> 1;
            ok = key_counts(rule0, e);
            if (w >= P.g.V) {
                record_bad(P, CSM_BAD_ENTRY, e, S.t_off[k0] + idx, 700 + E);
                ok = false;
            }
        }
        for (uint32_t em = excl; ok && em; em &= em - 1) ok = S.f[__ffs(em) - 1] != w;
        const uint32_t vmask = __ballot_sync(0xffffffffu, idx < best);
        const uint32_t target = __shfl_sync(0xffffffffu, w, 31 - __clz(vmask));
        const uint32_t key_hi = (target + 1) << 1;
        for (uint32_t k = 0; k < nkeys; k++) {
            if (k == k0 || !((mask >> k) & 1u)) continue;
            if (!__any_sync(0xffffffffu, ok)) break;
            const uint32_t *L = P.g.pool + S.t_off[k];
            const uint32_t size = S.t_size[k], c0 = S.t_cur[k];
            const uint32_t win = c0 + lane < size ? __ldg(L + c0 + lane) : 0xFFFFFFFFu;
            const uint32_t below = __ballot_sync(0xffffffffu, win < key_hi);
            uint32_t e = 0xFFFFFFFFu, hi;
            if (below != 0xffffffffu) {
                hi = c0 + __popc(below);
                const uint32_t pos = shfl_lower_bound(win, w << 1);
                const uint32_t got = __shfl_sync(0xffffffffu, win, pos);
                if ((got >> 1) == w && got != 0xFFFFFFFFu) e = got;
            } else {
                hi = warp_lower_bound(L, c0 + 32, size, key_hi, lane);
                if (ok) e = find_entry(L + c0, hi - c0, w);
            }
            if (ok) {
                probes++;
                ok = e != 0xFFFFFFFFu && key_counts(__ldg(&T->key_old[k]), e);
            }
            __syncwarp();
            if (lane == 0) S.t_cur[k] = hi;
            __syncwarp();
        }
        cnt += __popc(__ballot_sync(0xffffffffu, ok));
    }
    return cnt;
}

// Number of injective assignments of the tail vertices for the full prefix f[0..E-1].
__device__ unsigned long long tail_count(WarpState &S, const EnumParams &P, const DevPlan *pl,
                                         uint32_t &probes) {
    const uint32_t lane = lane_id();
    const DevTail *T = &pl->tail;
    const uint32_t nkeys = __ldg(&T->nkeys);
    const uint32_t nmasks = __ldg(&T->nmasks);
    const uint32_t E = pl->tail_start;
    // Lists whose size is used alone need their batch entries and the prefix vertices they
    // hold; intersections check both entry by entry.
    uint32_t single = 0;
    for (uint32_t mi = 0; mi < nmasks; mi++) {
        const uint32_t m = __ldg(&T->mask[mi]);
        if (__popc(m) == 1) single |= m;
    }
    if (lane < nkeys) {
        const uint32_t rel = __ldg(&T->key_rel[lane]);
        const uint32_t x = S.f[__ldg(&T->key_parent[lane])];
        const uint2 ms = list_of(P, rel, x, 300 + E);
        S.t_off[lane] = ms.x;
        S.t_size[lane] = ms.y;
        // Entries of this list that do not count under its rule.
        S.t_flag[lane] = ((single >> lane) & 1u) ? ms.y - key_entries(P, rel, x, ms.y, __ldg(&T->key_old[lane])) : 0u;
        S.t_excl[lane] = 0;
    }
    __syncwarp();
    // Prefix vertices that sit in a list sized alone are not available to its vertex.
    uint32_t nprobe = 0;
    for (uint32_t pi = lane; pi < nkeys * E; pi += 32) {
        const uint32_t k = pi / E;
        if (!((single >> k) & 1u)) continue;
        if (!((__ldg(&T->key_excl[k]) >> (pi % E)) & 1u)) continue;  // other labels are never in the list
        const uint32_t z = S.f[pi % E];
        const uint32_t e = find_entry(P.g.pool + S.t_off[k], S.t_size[k], z);
        nprobe++;
        if (e != 0xFFFFFFFFu && key_counts(__ldg(&T->key_old[k]), e)) atomicAdd(&S.t_excl[k], 1u);
    }
    probes += nprobe;
    __syncwarp();
    for (uint32_t mi = 0; mi < nmasks; mi++) {
        const uint32_t mask = __ldg(&T->mask[mi]);
        unsigned long long size;
        if (__popc(mask) == 1) {
            const uint32_t k = __ffs(mask) - 1;
            size = (unsigned long long)S.t_size[k] - S.t_flag[k] - S.t_excl[k];
        } else {
            size = tail_intersection(S, P, T, nkeys, mask, E, probes);
        }
        if (lane == 0) S.msize[mi] = size;
    }
    __syncwarp();
    unsigned long long total = 0;
    if (lane == 0) {
        total = 1;
        const DevTailTerm *terms = P.terms + pl->term_begin;
        const uint32_t nclasses = __ldg(&T->nclasses);
        for (uint32_t c = 0; c < nclasses; c++) {
            unsigned long long s = 0;
            const uint32_t tb = __ldg(&T->class_term_begin[c]), te = __ldg(&T->class_term_begin[c + 1]);
            for (uint32_t t = tb; t < te; t++) {
                unsigned long long prod = (unsigned long long)__ldg(&terms[t].coef);
                const uint32_t nf = __ldg(&terms[t].nf);
                for (uint32_t j = 0; j < nf; j++) prod *= S.msize[__ldg(&terms[t].f[j])];
                s += prod;
            }
            total *= s;
        }
    }
    __syncwarp();
    return total;
}

__device__ __forceinline__ unsigned long long slot_stamp(uint32_t epoch, uint32_t pos) {
    return ((unsigned long long)epoch << 32) | pos;
}

__device__ __forceinline__ unsigned long long device_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Checks the work item copied into S: plan, depth, candidate range and prefix vertex ids.  A
// failing item is recorded (`where`, `tag`) and must be skipped.  Warp-uniform.
__device__ bool item_ok(const WarpState &S, const EnumParams &P, uint32_t where, uint32_t tag) {
    const uint32_t lane = lane_id();
    const uint32_t plan = S.item_plan, depth = S.item_depth;
    bool ok = plan < P.nplans;
    if (ok) {
        if (depth == 0) ok = S.item_lo < S.item_hi && S.item_hi <= P.m;
        else ok = depth >= 2 && depth < P.plans[plan].n && S.item_lo <= S.item_hi;
    }
    const bool fok = !ok || lane >= depth || S.f[lane] < P.g.V;
    ok = __all_sync(0xffffffffu, ok && fok);
    if (!ok && lane == 0) record_bad(P, where, plan, depth, tag);
    __syncwarp();
    return ok;
}

// Warps that wait at the ring for an item (for every lane).  One 8-byte read of both ring counters.
__device__ __forceinline__ uint32_t items_wanted(const EnumParams &P) {
    int32_t n = 0;
    if (lane_id() == 0) {
        const unsigned long long w = *(volatile unsigned long long *)&P.ctrl->q_head;
        n = ring_wanted((uint32_t)w, (uint32_t)(w >> 32));
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    return n > 0 ? (uint32_t)n : 0u;
}

// Reserves `cnt` (1..32) consecutive ring positions while a warp waits for one; returns the first,
// or 0xFFFFFFFF when none waits (any more) or the ring has no room (either only costs balance: the
// donor keeps its work).  A position p of a later lap is free once the consumer of p - qcap has
// released its slot with stamp (epoch, p); first-lap positions are free as soon as nobody has
// reserved them.
__device__ uint32_t reserve_slots(const EnumParams &P, uint32_t cnt) {
    const uint32_t lane = lane_id();
    const uint32_t ep = P.ctrl->epoch;
    unsigned long long w = 0;
    if (lane == 0) w = *(volatile unsigned long long *)&P.ctrl->q_head;
    w = __shfl_sync(0xffffffffu, w, 0);
    const uint32_t pos = (uint32_t)w;
    if (ring_wanted(pos, (uint32_t)(w >> 32)) <= 0) return 0xFFFFFFFFu;
    const uint32_t p = pos + lane;
    bool free_slot = pos <= CSM_QUEUE_POS_LIMIT - cnt;
    if (free_slot && lane < cnt && p > P.qmask)
        free_slot = *(volatile unsigned long long *)(P.seq + (p & P.qmask)) == slot_stamp(ep, p);
    if (!__all_sync(0xffffffffu, free_slot)) {
        if (lane == 0) atomicAdd(&P.ctrl->queue_full, 1ull);
        return 0xFFFFFFFFu;
    }
    uint32_t won = 0;
    if (lane == 0) {
        won = atomicCAS(&P.ctrl->q_head, pos, pos + cnt) == pos;
        // Items count as active from here until the warp that receives them has run them.
        if (won) atomicAdd(&P.ctrl->active, cnt);
    }
    // Lost: another warp served the waiting one.  One attempt only, or every busy warp would queue
    // on the counter whenever a single warp waits.
    return __shfl_sync(0xffffffffu, won, 0) ? pos : 0xFFFFFFFFu;
}

// f[0] and f[1] of the seed at sorted batch key c: the edge's endpoints, or, where the plan's seeds
// are the inner endpoint's data vertices, that vertex and its number of batch edges (c is then the
// first key of the vertex's list).
__device__ __forceinline__ uint2 seed_pair(const EnumParams &P, const DevPlan *pl, uint32_t c) {
    const unsigned long long key = __ldg(P.keys + c);
    return make_uint2(P.kl.src(key), pl->seed_group == CSM_SEED_EDGE ? P.kl.dst(key) : __ldg(P.seg_flagged + c));
}

// Writes and publishes `cnt` (at most 32) items from ring position `pos` on, one per lane: lane i's
// item has the range [lo, hi) and the prefix f[0..nf-1], followed by `next` where the depth is nf + 1,
// or the seed `next`, `next2` where nf is 0 and the depth 2.
__device__ void publish_items(const EnumParams &P, uint32_t pos, uint32_t cnt, uint32_t plan, uint32_t depth,
                              const uint32_t *f, uint32_t nf, uint32_t lo, uint32_t hi, uint32_t next, uint32_t next2) {
    const uint32_t lane = lane_id();
    const uint32_t slot = (pos + lane) & P.qmask;
    if (lane < cnt) {
        WorkItem *it = P.queue + slot;
        it->plan = plan;
        it->depth = depth;
        it->lo = lo;
        it->hi = hi;
        for (uint32_t k = 0; k < nf; k++) it->f[k] = f[k];
        if (depth > nf) it->f[nf] = next;
        if (depth > nf + 1) it->f[nf + 1] = next2;
    }
    __threadfence();
    if (lane < cnt) atomicExch(P.seq + slot, slot_stamp(P.ctrl->epoch, pos + lane + 1));
    __syncwarp();
}

// Splits pending work of the current item into the queue, as many pieces as warps wait for (at most
// 31 at a time), from the shallowest level that has some.  Halving ranges, a launch of few heavy items
// took many rounds to spread (eight queries at 4,099 updates 7.0 -> 3.4 ms).
__device__ void try_donate(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t L0, uint32_t d,
                           uint32_t waiting) {
    const uint32_t lane = lane_id();
    const uint32_t E = pl->tail_start;
    // A shared last level is counted once per prefix at depth n - 3: the two deepest levels of
    // a prefix stay with the warp that holds it (so neither is counted twice).
    const uint32_t top = pl->shared_last ? pl->n - 3u : d;
    // Above a pendant counting level, buffered candidates are settled from the table, never
    // entered: they are not handed out as items of the counting level either.
    // The candidates above a tail that is counted one prefix at a time are handed out as items of
    // depth E, a tail count each: those counts are long (20-100 us over hub lists).
    const bool long_tail = E >= 3 && E < pl->n && !pl->tail.lane_par && !pl->tail.pair_par;
    const uint32_t sib_end = pl->memo_slot != CSM_NO_MEMO ? E - 1u : long_tail ? E + 1u : E;
    for (uint32_t l = L0; l <= d && l <= top; l++) {
        const uint32_t lo = S.lo[l], hi = S.hi[l];
        const uint32_t minr = (l == 1) ? 64u : P.steal_min;
        if (hi > lo && hi - lo >= minr) {
            // Equal parts of at least minr / 2 candidates (whole chunks of seeds); the first stays.
            uint32_t cnt = 2u * (hi - lo) / minr - 1u;
            cnt = cnt < waiting ? cnt : waiting;
            cnt = cnt < 31u ? cnt : 31u;
            uint32_t part = (hi - lo + cnt) / (cnt + 1u);
            if (l == 1) part = (part + 31u) & ~31u;
            cnt = (hi - lo - 1u) / part;
            if (cnt == 0) continue;
            const uint32_t slot = reserve_slots(P, cnt);
            if (slot == 0xFFFFFFFFu) return;
            const uint32_t a = lo + (lane + 1u) * part, b = hi - a < part ? hi : a + part;
            publish_items(P, slot, cnt, S.item_plan, l == 1 ? 0u : l, S.f, l == 1 ? 0u : l, a, b, 0, 0);
            if (lane == 0) {
                S.hi[l] = lo + part;
                atomicAdd(&P.ctrl->donations, (unsigned long long)cnt);
            }
            __syncwarp();
            return;
        }
        // Buffered siblings; of the current level's own buffer the next one stays.
        const uint32_t nb = S.nbuf[l], ps = S.pos[l] + (l == d ? 1u : 0u);
        if (l + 1 < sib_end && nb > ps) {
            const uint32_t cnt = nb - ps;
            const uint32_t slot = reserve_slots(P, cnt);
            if (slot == 0xFFFFFFFFu) return;
            uint2 next = make_uint2(0u, 0u);
            if (lane < cnt) next.x = S.buf[l][ps + lane];
            if (lane < cnt && l == 1) next = seed_pair(P, pl, next.x);
            publish_items(P, slot, cnt, S.item_plan, l + 1, S.f, l == 1 ? 0u : l, 0, 0xFFFFFFFFu, next.x, next.y);
            if (lane == 0) {
                S.nbuf[l] = (uint8_t)ps;
                atomicAdd(&P.ctrl->donations, (unsigned long long)cnt);
            }
            __syncwarp();
            return;
        }
    }
}

// Ends the launch for every waiting warp (the caller found that nothing holds work any more): the
// slots of all waiting positions get the stamp that says so.
__device__ void release_waiting(const EnumParams &P) {
    const unsigned long long w = *(volatile unsigned long long *)&P.ctrl->q_head;
    const uint32_t head = (uint32_t)w & ~CSM_QUEUE_CLOSED, waiting = ring_unserved(head, (uint32_t)(w >> 32));
    const uint32_t n = waiting < P.qmask + 1u ? waiting : P.qmask + 1u;
    const unsigned long long over = slot_stamp(P.ctrl->epoch, CSM_QUEUE_OVER);
    for (uint32_t i = lane_id(); i < n; i += 32) *(volatile unsigned long long *)(P.seq + ((head + i) & P.qmask)) = over;
}

// What a warp does whose bound has run out (its sleep time is `ns`): nothing was handed out all that time,
// since some warp has a long piece of work that cannot be split.  With the ring closed no position gets an
// item any more, so the warp leaves (2); unless its own position has been reserved already: it waits for
// the item for another bound (0), and gives up after that (4).  Out of line: inlined into the waiting loop
// it cost the launches that hand out most 2% (eight queries at 4,099 updates 3.15 -> 3.21 ms).
constexpr uint32_t kClosedSleep = 2048;
__device__ __noinline__ uint32_t close_ring(EnumControl *ctrl, uint32_t pos, uint32_t ns) {
    if (ring_may_leave(atomicOr(&ctrl->q_head, CSM_QUEUE_CLOSED), pos)) return 2u;
    return ns == kClosedSleep ? 4u : 0u;
}

// An idle warp takes the next ring position as its own and waits for that position's item: 1 = item
// copied into S, 0 = the launch is over for this warp (or its time limit has passed, err), -1 = an item
// that failed its check.  Every waiting warp polls a word of its own slot, so thousands of waiting warps
// do not crowd the counters the working ones need.  With all of them polling the shared counters, and
// taking back a shared request count by compare-and-swap on leaving, a launch over a handful of items
// took 270 us (4,736 warps queueing on one address); it takes 13-22 us now, and the launches where
// few warps hold work gained most from donors that no longer wait behind the polls (1024 updates on
// 10,000 vertices 10.2 -> 0.86 ms, 65,536 with a tree query 554 -> 306 ms).
__device__ int await_item(WarpState &S, const EnumParams &P, unsigned int &err, unsigned long long deadline) {
    const uint32_t lane = lane_id();
    const uint32_t ep = P.ctrl->epoch;
    uint32_t pos = 0, got = 0;
    if (lane == 0) {
        pos = atomicAdd(&P.ctrl->q_tail, 1u);
        __threadfence();  // the position is taken before this warp stops counting as active
        if (atomicSub(&P.ctrl->active, 1u) == 1u) got = 2;
    }
    pos = __shfl_sync(0xffffffffu, pos, 0);
    if (__shfl_sync(0xffffffffu, got, 0)) {
        release_waiting(P);
        return 0;
    }
    if (lane == 0) {
        volatile unsigned long long *seq = P.seq + (pos & P.qmask);
        uint32_t ns = 64, polls = 0, head = 0;
        while (got == 0) {
            const unsigned long long w = *seq;
            if (w == slot_stamp(ep, pos + 1)) got = 1;
            else if (w == slot_stamp(ep, CSM_QUEUE_OVER)) got = 2;
            else if (deadline && device_ns() > deadline) got = 3;
            else if (++polls >= P.idle_limit) {
                got = close_ring(P.ctrl, pos, ns);
                ns = kClosedSleep;
                polls = 0;
            } else __nanosleep(ns);
            if (ns < 1024) ns <<= 1;
            if (got == 0 && (polls & 255u) == 0) {
                // Seldom: whether anything holds work, and whether it is still being handed out (the
                // bound is on waiting without a sign of progress).
                const uint32_t h = *(volatile unsigned int *)&P.ctrl->q_head & ~CSM_QUEUE_CLOSED;
                if (*(volatile unsigned int *)&P.ctrl->active == 0) got = 2;
                if (h != head) polls = 0;
                head = h;
            }
        }
        __threadfence();
    }
    got = __shfl_sync(0xffffffffu, got, 0);
    if (got == 3) err |= CSM_ERRBIT_TIMEOUT;
    if (got == 4) err |= CSM_ERRBIT_TIMEOUT | CSM_ERRBIT_IDLE;
    if (got != 1) return 0;
    volatile const WorkItem *it = P.queue + (pos & P.qmask);
    if (lane == 0) {
        S.item_plan = it->plan;
        S.item_depth = it->depth;
        S.item_lo = it->lo;
        S.item_hi = it->hi;
    }
    if (lane < CSM_MAXQV) S.f[lane] = it->f[lane];
    __syncwarp();
    if (lane == 0) {
        __threadfence();
        atomicExch(P.seq + (pos & P.qmask), slot_stamp(ep, pos + P.qmask + 1));
    }
    __syncwarp();
    return item_ok(S, P, CSM_BAD_ITEM, pos) ? 1 : -1;
}

// Takes the next seed chunk or frontier item into S: 1 = taken, 0 = none left, -1 = a frontier
// item that failed its check (skipped).
__device__ int take_ticket(WarpState &S, const EnumParams &P, const WorkItem *frontier) {
    const uint32_t lane = lane_id();
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(&P.ctrl->ticket, 1ull);
    t = __shfl_sync(0xffffffffu, t, 0);
    const unsigned long long nt = *(volatile unsigned long long *)&P.ctrl->nticket;
    if (t >= nt) return 0;
    if (frontier != nullptr) {
        const WorkItem *it = frontier + t;
        if (lane == 0) {
            S.item_plan = it->plan;
            S.item_depth = it->depth;
            S.item_lo = it->lo;
            S.item_hi = it->hi;
        }
        if (lane < CSM_MAXQV) S.f[lane] = it->f[lane];
        __syncwarp();
        if (!item_ok(S, P, CSM_BAD_FRONTIER, (uint32_t)t)) return -1;
    } else {
        // Seed chunk t: plan p with ticket_prefix[p] <= t < ticket_prefix[p+1].
        uint32_t lo = 0, hi = P.nplans;
        while (lo + 1 < hi) {
            uint32_t mid = (lo + hi) >> 1;
            if (__ldg(P.ticket_prefix + mid) <= t) lo = mid;
            else hi = mid;
        }
        const uint32_t p = lo;
        const uint32_t chunk = (uint32_t)(t - __ldg(P.ticket_prefix + p));
        const uint32_t s0 = __ldg(P.seed_lo + p) + chunk * 32u;
        const uint32_t s_end = __ldg(P.seed_lo + P.nplans + p);
        if (lane == 0) {
            S.item_plan = p;
            S.item_depth = 0;
            S.item_lo = s0;
            S.item_hi = s0 + 32u < s_end ? s0 + 32u : s_end;
        }
    }
    __syncwarp();
    return 1;
}

__device__ void write_row(const EnumParams &P, const DevPlan *pl, const WarpState &S, uint32_t d, uint32_t w,
                          unsigned long long r) {
    uint32_t *row = P.rows + r * P.row_words;
    row[0] = pl->query;
    for (uint32_t k = 0; k < d; k++) row[1 + pl->order[k]] = S.f[k];
    row[1 + pl->order[d]] = w;
}

// Last counting level with packed siblings.  The buffered candidates s_0..s_{k-1} of level
// d = n - 2 each open a last level whose candidate lists are usually short, so instead of one
// pass per sibling the warp scans all their pivot lists at once, one (sibling, position) pair
// per lane.  A lane finds its sibling by a shuffle search over the inclusive prefix of list
// lengths and checks its candidate like the per-sibling scan (flag rule, injectivity, NLF
// bitmap, membership in the other backward lists by binary search).  Returns false (nothing
// counted) when the lists are long enough for the per-sibling scan to fill the warp.
__device__ bool count_last_packed(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d,
                                  unsigned long long &cnt, uint32_t &scans, uint32_t &probes) {
    const uint32_t lane = lane_id();
    const uint32_t L = d + 1;
    const DevLevel *lv = &pl->lv[L];
    const uint32_t nbn = __ldg(&lv->nbn);
    const uint32_t oldm = __ldg(&lv->old_mask);
    const uint32_t nlf_id = __ldg(&lv->nlf_bitmap);
    const uint32_t *nlf = nlf_id == CSM_NO_BITMAP ? nullptr : bitmap(P, nlf_id);
    const uint32_t exm = __ldg(&lv->excl_mask) & ((1u << d) - 1u);  // depth d is the sibling itself
    const uint32_t ps = S.pos[d], k = S.nbuf[d] - ps;
    // Shared lists: backward neighbours matched before depth d (same for every sibling).
    // sib_b = the backward neighbour at depth d (at most one), whose list is the sibling's own.
    const uint32_t bb = __ldg(&lv->bn_base);
    uint32_t sib_b = 0xFFu, sh_min = 0xFFFFFFFFu, sh_piv = 0;
    for (uint32_t b = 0; b < nbn; b++) {
        const uint32_t dep = __ldg(&lv->bn_depth[b]);
        if (dep == d) {
            sib_b = b;
            continue;
        }
        const uint2 ms = list_of(P, __ldg(&lv->bn_rel[b]), S.f[dep], 400 + L);
        if (lane == 0) {
            S.poff[bb + b] = ms.x;  // level L's own slots: it is counted, never entered
            S.psz[bb + b] = ms.y;
        }
        if (ms.y < sh_min) {
            sh_min = ms.y;
            sh_piv = b;
        }
    }
    __syncwarp();
    // Per sibling (lane j < k): its own list, its pivot and the pivot's list.
    uint32_t sv = 0, s_off = 0, s_sz = 0, pv = sh_piv, p_off = 0, p_len = 0;
    if (lane < k) {
        sv = S.buf[d][ps + lane];
        if (sib_b != 0xFFu) {
            const uint2 ms = list_of(P, __ldg(&lv->bn_rel[sib_b]), sv, 500 + L);
            s_off = ms.x;
            s_sz = ms.y;
        }
        // The smallest list is the pivot, the lowest backward-neighbour index on ties (the
        // choice enter_level makes), so the work counters do not depend on packing.
        if (sib_b != 0xFFu && (s_sz < sh_min || (s_sz == sh_min && sib_b < sh_piv))) {
            pv = sib_b;
            p_off = s_off;
            p_len = s_sz;
        } else {
            p_off = S.poff[bb + sh_piv];
            p_len = sh_min;
        }
    }
    // Inclusive prefix of pivot lengths.
    uint32_t incl = p_len;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if (total > 4u * k) return false;  // longer lists: the per-sibling scan fills the warp better
    for (uint32_t g0 = 0; g0 < total; g0 += 32) {
        const uint32_t g = g0 + lane;
        // Sibling of position g: the first lane whose inclusive prefix exceeds g.
        uint32_t j = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xffffffffu, incl, j + step - 1) <= g) j += step;
        const uint32_t jc = j < 31 ? j : 31;
        const uint32_t excl_j = __shfl_sync(0xffffffffu, incl, jc) - __shfl_sync(0xffffffffu, p_len, jc);
        const uint32_t c_sv = __shfl_sync(0xffffffffu, sv, jc);
        const uint32_t c_soff = __shfl_sync(0xffffffffu, s_off, jc);
        const uint32_t c_ssz = __shfl_sync(0xffffffffu, s_sz, jc);
        const uint32_t c_pv = __shfl_sync(0xffffffffu, pv, jc);
        const uint32_t c_poff = __shfl_sync(0xffffffffu, p_off, jc);
        bool ok = g < total;
        uint32_t w = 0;
        if (ok) {
            const uint32_t e = __ldg(P.g.pool + c_poff + (g - excl_j));
            w = e >> 1;
            scans++;
            ok = !(((oldm >> c_pv) & 1u) && (e & 1u)) && w != c_sv;
            if (w >= P.g.V) {
                record_bad(P, CSM_BAD_ENTRY, e, c_poff + (g - excl_j), 600 + L);
                ok = false;
            }
        }
        for (uint32_t em = exm; ok && em; em &= em - 1) ok = S.f[__ffs(em) - 1] != w;
        const uint32_t nlf_word = !ok ? 0u : (nlf ? __ldg(nlf + (w >> 5)) : 0xFFFFFFFFu);
        for (uint32_t b = 0; ok && b < nbn; b++) {
            if (b == c_pv) continue;
            const uint32_t *list = b == sib_b ? P.g.pool + c_soff : P.g.pool + S.poff[bb + b];
            const uint32_t sz = b == sib_b ? c_ssz : S.psz[bb + b];
            const uint32_t e = find_entry(list, sz, w);
            probes++;
            ok = e != 0xFFFFFFFFu && !(((oldm >> b) & 1u) && (e & 1u));
        }
        if (ok) ok = (nlf_word >> (w & 31)) & 1u;
        cnt += __popc(__ballot_sync(0xffffffffu, ok));
    }
    __syncwarp();
    if (lane == 0) S.pos[d] = S.nbuf[d];
    __syncwarp();
    return true;
}

// Last level of a counting plan without a tail: the matches are the pivot-list candidates that
// pass the flag rule, injectivity and membership in the one other backward list, i.e. a
// filtered count of a sorted-list intersection (the shape of the last level of every dense plan
// measured: two backward neighbours).  The other list's offset, size, cursor and flag rule stay
// in registers for the whole scan instead of being re-read from the warp's shared state for
// every 32 candidates.  Every 8 chunks the warp looks for waiting warps (donating parts
// of the remaining range) and checks the time limit.  Returns the count; the level is left
// exhausted (S.lo[d] >= S.hi[d]).
constexpr uint32_t kLastLists = 1;
constexpr uint32_t kWindows = 3;

__device__ unsigned long long count_last_level(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t L0,
                                               uint32_t d, uint32_t &scans, uint32_t &probes, unsigned int &err,
                                               unsigned long long deadline) {
    const uint32_t lane = lane_id();
    const uint32_t nbn = S.nbn[d], piv = S.piv[d], bb = S.bnb[d];
    const uint32_t oldm = S.oldm[d], exm = S.exm[d], nlf_id = S.nlf[d];
    const bool piv_old = (oldm >> piv) & 1u;
    const uint32_t *nlf = nlf_id == CSM_NO_BITMAP ? nullptr : bitmap(P, nlf_id);
    const uint32_t *base = P.g.pool + S.base[d];
    uint32_t l_off[kLastLists], l_size[kLastLists], l_cur[kLastLists];
    uint32_t l_old = 0;  // bit j: list j's batch entries do not count
    uint32_t nl = 0;
#pragma unroll
    for (uint32_t j = 0; j < kLastLists; j++) l_off[j] = l_size[j] = l_cur[j] = 0;
    for (uint32_t k = 0; k < nbn; k++) {
        if (k == piv) continue;
#pragma unroll
        for (uint32_t j = 0; j < kLastLists; j++)
            if (j == nl) {
                l_off[j] = S.poff[bb + k];
                l_size[j] = S.psz[bb + k];
                l_old |= ((oldm >> k) & 1u) << j;
            }
        nl++;
    }
    uint32_t lo = S.lo[d], hi = S.hi[d];
    unsigned long long cnt = 0;
    for (uint32_t chunk = 1; lo < hi; lo += 32, chunk++) {
        const uint32_t idx = lo + lane;
        const bool in = idx < hi;
        bool ok = in;
        uint32_t cand = 0;
        if (ok) {
            const uint32_t e = __ldg(base + idx);
            cand = e >> 1;
            scans++;
            ok = !(piv_old && (e & 1u));
            if (cand >= P.g.V) {
                record_bad(P, CSM_BAD_ENTRY, e, S.base[d] + idx, d);
                ok = false;
            }
        }
        for (uint32_t em = exm; ok && em; em &= em - 1) ok = S.f[__ffs(em) - 1] != cand;
        const uint32_t nlf_word = !ok ? 0u : (nlf ? __ldg(nlf + (cand >> 5)) : 0xFFFFFFFFu);
        const uint32_t vmask = __ballot_sync(0xffffffffu, in);
        const uint32_t target = __shfl_sync(0xffffffffu, cand, 31 - __clz(vmask));
        const uint32_t key_hi = (target + 1) << 1;
        uint32_t win[kLastLists];
#pragma unroll
        for (uint32_t j = 0; j < kLastLists; j++)
            win[j] = (j < nl && l_cur[j] + lane < l_size[j]) ? __ldg(P.g.pool + l_off[j] + l_cur[j] + lane) : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t j = 0; j < kLastLists; j++) {
            if (j >= nl) break;
            uint32_t e = 0xFFFFFFFFu, nhi = 0;
            // The chunk's candidates span ~40-55 entries of the other list on the measured
            // queries: walk up to kWindows consecutive 32-entry windows (one coalesced load each)
            // before bracketing the rest of the list with the warp search.
            const uint32_t *L = P.g.pool + l_off[j];
            uint32_t c0 = l_cur[j], w = win[j];
            bool done = false;
#pragma unroll 1
            for (uint32_t k = 0; k < kWindows; k++) {
                const uint32_t below = __ballot_sync(0xffffffffu, w < key_hi);
                const uint32_t pos = shfl_lower_bound(w, cand << 1);
                const uint32_t got = __shfl_sync(0xffffffffu, w, pos);
                if ((got >> 1) == cand && got != 0xFFFFFFFFu) e = got;
                if (below != 0xffffffffu) {
                    nhi = c0 + __popc(below);
                    done = true;
                    break;
                }
                c0 += 32;
                w = c0 + lane < l_size[j] ? __ldg(L + c0 + lane) : 0xFFFFFFFFu;
            }
            if (!done) {
                nhi = warp_lower_bound(L, c0, l_size[j], key_hi, lane);
                if (ok && e == 0xFFFFFFFFu) e = find_entry(L + c0, nhi - c0, cand);
            }
            if (ok) {
                probes++;
                ok = e != 0xFFFFFFFFu && !(((l_old >> j) & 1u) && (e & 1u));
            }
            l_cur[j] = nhi;
        }
        if (ok) ok = (nlf_word >> (cand & 31)) & 1u;
        cnt += __popc(__ballot_sync(0xffffffffu, ok));
        if ((chunk & 7u) == 0 && lo + 32 < hi) {
            if (deadline) {
                unsigned int late = 0;
                if (lane == 0) late = device_ns() > deadline;
                if (__shfl_sync(0xffffffffu, late, 0)) {
                    err |= CSM_ERRBIT_TIMEOUT;
                    break;
                }
            }
            if (P.donate) {
                const uint32_t waiting = items_wanted(P);
                if (waiting) {
                    // The remaining range [lo + 32, hi) is this level's pending work.
                    if (lane == 0) {
                        S.lo[d] = lo + 32;
                        S.hi[d] = hi;
                    }
                    __syncwarp();
                    try_donate(S, P, pl, L0, d, waiting);
                    hi = S.hi[d];
                    __syncwarp();
                }
            }
        }
    }
    __syncwarp();
    if (lane == 0) {
        S.lo[d] = hi;
        S.hi[d] = hi;
    }
    __syncwarp();
    return cnt;
}

// Shared last level (DevPlan.shared_last), level d = n - 2 with candidates buffered: the count
// of the last level for the prefix f[0..n-3] was taken once (S.sl_count, with f[n-2] left out of
// its exclusions), so each buffered candidate v contributes that count, minus one when v is
// itself a candidate of the last level — in every backward list of level n - 1 under the flag
// rule and in its NLF bitmap.  v differs from every prefix vertex of its own label already, so
// nothing else changes.  Consumes the buffer.
__device__ unsigned long long count_shared_last(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d,
                                                uint32_t &probes) {
    const uint32_t lane = lane_id();
    const uint32_t L = d + 1;
    const uint32_t ps = S.pos[d], k = S.nbuf[d] - ps;
    unsigned long long total = (unsigned long long)k * S.sl_count;
    if ((__ldg(&pl->lv[L].excl_mask) >> d) & 1u) {
        bool in = lane < k;
        if (in) {
            const uint32_t v = S.buf[d][ps + lane];
            const uint32_t nbn = S.nbn[L], bb = S.bnb[L], oldm = S.oldm[L], nlf_id = S.nlf[L];
            for (uint32_t b = 0; in && b < nbn; b++) {
                const uint32_t e = find_entry(P.g.pool + S.poff[bb + b], S.psz[bb + b], v);
                probes++;
                in = e != 0xFFFFFFFFu && !(((oldm >> b) & 1u) && (e & 1u));
            }
            if (in && nlf_id != CSM_NO_BITMAP) in = test_bit(bitmap(P, nlf_id), v);
        }
        total -= __popc(__ballot_sync(0xffffffffu, in));
    }
    __syncwarp();
    if (lane == 0) S.pos[d] = S.nbuf[d];
    __syncwarp();
    return total;
}

// Pendant counting level c = d + 1 (DevPlan.memo_slot): every buffered candidate of level d
// contributes the table entry of the data vertex y at memo_depth (the candidate itself when that
// depth is d), less the tail values of the prefix vertices of c's label that are candidates of c below
// y, times the tail classes that hang off the prefix.  Where prefix vertices share the label of the one
// tail vertex below c (memo_cut), each is taken off once per candidate of c next to it: a pair
// intersection.  Consumes the buffer.  Walking the level instead was 90% of the tree query's time
// (65,536 updates: 113 -> 4.2 ms; four queries at 16,411, with the cut vertices, 173 -> 56 ms).
template <bool PAIRS>
__device__ unsigned long long settle_pendant(WarpState &S, const EnumParams &P, const DevPlan *pl, uint32_t d,
                                             uint32_t &tails) {
    const uint32_t lane = lane_id();
    const uint32_t ps = S.pos[d], k = S.nbuf[d] - ps;
    const uint32_t md = pl->memo_depth;
    const DevTail *T = &pl->tail;
    const DevLevel *lv = &pl->lv[d + 1];
    unsigned long long v = 0;
    const uint32_t cut = PAIRS ? __ldg(&pl->memo_cut) : 0u;
    const uint32_t x = lane < k ? S.buf[d][ps + lane] : 0u;
    const uint32_t y = md == d ? x : S.f[md];
    unsigned long long cuts = 0;
    if (PAIRS && cut) {
        const uint32_t sig = __ldg(&pl->cut_pair);
        const uint32_t rc = __ldg(&lv->bn_rel[0]), rule_c = (__ldg(&lv->old_mask) & 1u) ? CSM_KEY_OLD : CSM_KEY_ANY;
        const uint32_t rl = __ldg(&pl->cut_rel), rule_l = __ldg(&T->key_old[__ldg(&pl->cut_key)]);
        for (uint32_t em = cut; em; em &= em - 1) {
            const uint32_t j = __ffs(em) - 1, z = j == d ? x : S.f[j];
            const bool uniform = md != d && j != d;
            const bool sw = (sig & CSM_PAIR_SWAP) != 0;  // the signature names the other list first
            cuts += pair_lookup(P, sig, sw ? rl : rc, sw ? rule_l : rule_c, sw ? z : y, sw ? rc : rl, sw ? rule_c : rule_l,
                                sw ? y : z, lane < k, uniform, 970 + d);
        }
    }
    if (lane < k) {
        v = __ldg(P.memo + (size_t)pl->memo_slot * P.g.V + y) - cuts;
        uint32_t excl = __ldg(&lv->excl_mask) & ~(1u << md);
        if (excl) {
            const uint2 ms = list_of(P, __ldg(&lv->bn_rel[0]), y, 950 + d);
            const bool old = (__ldg(&lv->old_mask) & 1u) != 0;
            const uint32_t nlf_id = __ldg(&lv->nlf_bitmap);
            for (; excl; excl &= excl - 1) {
                const uint32_t j = __ffs(excl) - 1, z = j == d ? x : S.f[j];
                const uint32_t e = find_entry(P.g.pool + ms.x, ms.y, z);
                if (e == 0xFFFFFFFFu || (old && (e & 1u))) continue;
                if (nlf_id != CSM_NO_BITMAP && !test_bit(bitmap(P, nlf_id), z)) continue;
                v -= __ldg(P.memo + (size_t)pl->memo_tail * P.g.V + z);
                if (!PAIRS || !cut) continue;
                // z is no candidate: what the cut vertices took off for it comes back.
                const uint32_t key = __ldg(&pl->cut_key), rule = __ldg(&T->key_old[key]);
                const uint2 zs = list_of(P, __ldg(&T->key_rel[key]), z, 980 + d);
                for (uint32_t cm = cut; cm; cm &= cm - 1) {
                    const uint32_t i = __ffs(cm) - 1;
                    const uint32_t en = find_entry(P.g.pool + zs.x, zs.y, i == d ? x : S.f[i]);
                    v += en != 0xFFFFFFFFu && key_counts(rule, en);
                }
            }
        }
        const uint32_t rest = ((1u << __ldg(&T->nclasses)) - 1u) & ~__ldg(&T->deep);
        if (rest && v) {
            const uint32_t nkeys = __ldg(&T->nkeys);
            uint32_t ksize[CSM_TAIL_MAXKEYS];
#pragma unroll 1
            for (uint32_t q = 0; q < nkeys; q++) {
                const uint32_t pd = __ldg(&T->key_parent[q]);
                ksize[q] = 0;
                if (pd > d) continue;
                const uint32_t rel = __ldg(&T->key_rel[q]), rule = __ldg(&T->key_old[q]);
                const uint32_t p = pd == d ? x : S.f[pd];
                const uint2 ms = list_of(P, rel, p, 960 + d);
                uint32_t left = key_entries(P, rel, p, ms.y, rule);
                uint32_t em = __ldg(&T->key_excl[q]) & ((2u << d) - 1u) & ~(1u << pd);
                for (; em; em &= em - 1) {
                    const uint32_t j = __ffs(em) - 1;
                    const uint32_t e = find_entry(P.g.pool + ms.x, ms.y, j == d ? x : S.f[j]);
                    if (e != 0xFFFFFFFFu && key_counts(rule, e)) left--;
                }
                ksize[q] = left;
            }
            v *= tail_product(P, pl, ksize, rest);
        }
    }
    tails += k;  // warp-uniform, like every other use of the tail counter
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncwarp();
    if (lane == 0) S.pos[d] = S.nbuf[d];
    __syncwarp();
    return v;
}

// Runs one work item to completion (or until the device clock passes `deadline`, when that is
// nonzero: the rest of the item is then dropped and CSM_ERRBIT_TIMEOUT set).  Returns the number
// of matches counted.
template <bool LASTLOOP, bool PAIRS, int MODE>
__device__ unsigned long long run_item(WarpState &S, const EnumParams &P, uint32_t &scans,
                                       uint32_t &probes, uint32_t &tails, uint32_t &shared, unsigned int &err,
                                       unsigned long long deadline, WorkItem *expand_out) {
    const uint32_t lane = lane_id();
    const DevPlan *pl = P.plans + S.item_plan;
    const uint32_t n = pl->n;
    const uint32_t E = pl->tail_start;
    uint32_t L0 = S.item_depth == 0 ? 1u : S.item_depth;
    unsigned long long cnt = 0;

    if (MODE == CSM_ENUM_MODE_EXPAND && L0 >= pl->expand_stop) {
        // Nothing left to expand before the counting level: pass the item through.
        unsigned long long r = 0;
        if (lane == 0) r = atomicAdd(&P.ctrl->out_rows, 1ull);
        r = __shfl_sync(0xffffffffu, r, 0);
        if (r < P.frontier_cap) {
            WorkItem *o = expand_out + r;
            if (lane == 0) {
                o->plan = S.item_plan;
                o->depth = S.item_depth;
                o->lo = S.item_lo;
                o->hi = S.item_hi;
            }
            if (lane < CSM_MAXQV) o->f[lane] = S.f[lane];
        } else if (lane == 0) {
            err |= CSM_ERRBIT_FRONTIER;
        }
        __syncwarp();
        return 0;
    }

    if (MODE == CSM_ENUM_MODE_COUNT && L0 == E && E < n) {
        // A single prefix above a tail (see try_donate): the only buffered candidate of its level.
        L0 = E - 1;
        if (lane == 0) {
            S.buf[L0][0] = S.f[L0];
            S.nbuf[L0] = 1;
            S.pos[L0] = 0;
            S.lo[L0] = S.hi[L0] = 0;
        }
        __syncwarp();
    } else if (L0 == 1) {
        if (lane == 0) {
            S.lo[1] = S.item_lo;
            S.hi[1] = S.item_hi;
            S.nbuf[1] = 0;
            S.pos[1] = 0;
        }
        __syncwarp();
    } else {
        enter_level(S, P, pl, L0, S.item_lo, S.item_hi);
    }
    uint32_t d = L0;
    uint32_t iter = 0;
    unsigned long long sl_before = 0;
    // Matches of the seeds already done, and what each match of the current seed counts.
    unsigned long long total = 0;
    uint32_t weight = S.item_depth >= 2 && pl->seed_group == CSM_SEED_WEIGHT ? S.f[1] : 1u;
    if (lane == 0) S.sl_state = 0;
    const uint32_t *nlf0 = bitmap(P, pl->nlf0);
    const uint32_t *nlf1 = bitmap(P, pl->nlf1);

    while (true) {
        ++iter;
        if (deadline && (iter & 63u) == 0) {
            unsigned int late = 0;
            if (lane == 0) late = device_ns() > deadline;
            if (__shfl_sync(0xffffffffu, late, 0)) {
                err |= CSM_ERRBIT_TIMEOUT;
                break;
            }
        }
        if (P.donate && (iter & 7u) == 0) {
            // While a warp waits for work, split off one piece of this warp's pending work.
            const uint32_t waiting = items_wanted(P);
            if (waiting) try_donate(S, P, pl, L0, d, waiting);
        }
        if (S.pos[d] < S.nbuf[d]) {
            if (MODE == CSM_ENUM_MODE_COUNT && d + 2 == E && P.memo != nullptr && pl->memo_slot < CSM_MEMO_PENDING &&
                (PAIRS || !pl->memo_cut)) {
                // Pendant counting level below: each buffered candidate's count is a table entry.
                cnt += settle_pendant<PAIRS>(S, P, pl, d, tails);
                continue;
            }
            if (MODE == CSM_ENUM_MODE_COUNT && d + 2 == n && pl->shared_last) {
                // The last level does not depend on these candidates: count it once for the
                // prefix (first time here), then settle every buffered candidate at once.
                if (S.sl_state == 2) {
                    cnt += count_shared_last(S, P, pl, d, probes);
                    continue;
                }
                sl_before = cnt;
                shared++;
                d++;
                enter_level(S, P, pl, d, 0, 0xFFFFFFFFu);
                if (lane == 0) {
                    S.sl_state = 1;
                    S.exm[d] &= (uint16_t)~(1u << (d - 1));  // f[n-2] is settled per candidate
                }
                __syncwarp();
                continue;
            }
            // Siblings whose subtree is only the last level: count them together.  Tried once per
            // buffer: when the lists are too long for it, they stay so for the later siblings.
            if (d + 2 == n && E == n && d >= 2 && MODE == CSM_ENUM_MODE_COUNT && S.pos[d] == 0 &&
                count_last_packed(S, P, pl, d, cnt, scans, probes))
                continue;
            // Descend into the next buffered candidate.
            const uint32_t c = S.buf[d][S.pos[d]];
            if (d == 1) {
                total += cnt * weight;  // the seed before this one is done
                cnt = 0;
            }
            __syncwarp();
            if (lane == 0) {
                S.pos[d]++;
                if (d == 1) {
                    const uint2 seed = seed_pair(P, pl, c);
                    S.f[0] = seed.x;
                    S.f[1] = seed.y;
                } else {
                    S.f[d] = c;
                }
            }
            __syncwarp();
            if (d == 1 && pl->seed_group == CSM_SEED_WEIGHT) weight = S.f[1];
            if (d + 1 == E) {
                cnt += tail_count(S, P, pl, probes);
                tails++;
                iter |= 7u;  // look for waiting warps after every long step
            } else {
                d++;
                if (lane == 0 && d + 2 == n) S.sl_state = 0;  // a new prefix f[0..n-3]
                enter_level(S, P, pl, d, 0, 0xFFFFFFFFu);
                // A chunk of a counting level with list intersections is a long step: look before it.
                if (PAIRS && d + 1 == E && pl->tail.pair_par && S.hi[d] >= 64u) iter |= 7u;
            }
            continue;
        }
        if (S.lo[d] >= S.hi[d]) {
            if (MODE == CSM_ENUM_MODE_COUNT && d + 1 == n && S.sl_state == 1) {
                // The shared last level is counted: keep its count for the candidates above.
                if (lane == 0) {
                    S.sl_count = cnt - sl_before;
                    S.sl_state = 2;
                }
                cnt = sl_before;
                __syncwarp();
            }
            if (d == L0) break;
            d--;
            continue;
        }
        if (LASTLOOP && d + 1 == n && E == n && d >= 2 && MODE == CSM_ENUM_MODE_COUNT && S.nbn[d] <= kLastLists + 1) {
            cnt += count_last_level(S, P, pl, L0, d, scans, probes, err, deadline);
            if (err & CSM_ERRBIT_TIMEOUT) break;
            continue;
        }
        // Scan the next 32 candidates of level d.
        const uint32_t idx = S.lo[d] + lane;
        bool ok = idx < S.hi[d];
        uint32_t cand = 0;
        if (d == 1) {
            if (ok) {
                const unsigned long long key = __ldg(P.keys + idx);
                const uint32_t x = P.kl.src(key), y = P.kl.dst(key);
                if (pl->seed_group == CSM_SEED_EDGE)
                    ok = __ldg(P.eff + idx) == P.phase && x != y && test_bit(nlf0, x) && test_bit(nlf1, y);
                else  // the first key of a list with batch edges (the leaf's NLF rule is implied)
                    ok = (idx == 0 || P.kl.list_of(__ldg(P.keys + idx - 1)) != P.kl.list_of(key)) &&
                         __ldg(P.seg_flagged + idx) > 0 && test_bit(nlf0, x);
                cand = idx;
            }
        } else {
            const uint32_t oldm = S.oldm[d];
            const uint32_t piv = S.piv[d];
            if (ok) {
                const uint32_t e = __ldg(P.g.pool + S.base[d] + idx);
                cand = e >> 1;
                scans++;
                ok = !(((oldm >> piv) & 1u) && (e & 1u));
                if (cand >= P.g.V) {
                    record_bad(P, CSM_BAD_ENTRY, e, S.base[d] + idx, d);
                    ok = false;
                }
            }
            for (uint32_t em = S.exm[d]; ok && em; em &= em - 1) ok = S.f[__ffs(em) - 1] != cand;
            // The NLF word is loaded now and tested after the probes, so its latency overlaps
            // theirs (probes are warp-wide and do not depend on it).
            const uint32_t nlf_id = S.nlf[d];
            const uint32_t nlf_word =
                !ok ? 0u : (nlf_id == CSM_NO_BITMAP ? 0xFFFFFFFFu : __ldg(bitmap(P, nlf_id) + (cand >> 5)));
            // Membership in the other backward lists.  The chunk's candidates ascend, so each list
            // keeps a cursor and is searched in the window from there on that the chunk spans.
            const uint32_t nbn = S.nbn[d], bb = S.bnb[d];
            const uint32_t last = 31 - __clz(__ballot_sync(0xffffffffu, idx < S.hi[d]));
            const uint32_t key = cand << 1, top = __shfl_sync(0xffffffffu, key, last);
            const uint32_t psize = S.psz[bb + piv];
            for (uint32_t k = 0; k < nbn; k++) {
                if (k == piv) continue;
                if (!__any_sync(0xffffffffu, ok)) break;
                const uint32_t slot = bb + k, size = S.psz[slot];
                uint32_t c0 = S.cur[slot];
                const uint32_t e = window_find(P.g.pool + S.poff[slot], size, c0, first_window(size, psize), key, top, last);
                if (ok) {
                    probes++;
                    ok = e != 0xFFFFFFFFu && !(((oldm >> k) & 1u) && (e & 1u));
                }
                __syncwarp();
                if (lane == 0) S.cur[slot] = c0;
                __syncwarp();
            }
            if (ok) ok = (nlf_word >> (cand & 31)) & 1u;
        }
        __syncwarp();
        if (lane == 0) S.lo[d] += 32u;
        const uint32_t mask = __ballot_sync(0xffffffffu, ok);
        const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
        if (MODE == CSM_ENUM_MODE_EXPAND && d == L0) {
            // One BFS level: survivors become items of depth d + 1.
            const uint32_t c = __popc(mask);
            unsigned long long r = 0;
            if (lane == 0 && c) r = atomicAdd(&P.ctrl->out_rows, (unsigned long long)c);
            r = __shfl_sync(0xffffffffu, r, 0);
            if (c && r + c > P.frontier_cap) {
                if (lane == 0) err |= CSM_ERRBIT_FRONTIER;
            } else if (ok) {
                WorkItem *o = expand_out + r + rank;
                o->plan = S.item_plan;
                o->depth = d + 1;
                o->lo = 0;
                o->hi = 0xFFFFFFFFu;
                if (d == 1) {
                    const uint2 seed = seed_pair(P, pl, cand);
                    o->f[0] = seed.x;
                    o->f[1] = seed.y;
                } else {
                    for (uint32_t k = 0; k < d; k++) o->f[k] = S.f[k];
                    o->f[d] = cand;
                }
            }
            __syncwarp();
        } else if (d + 1 == E && E < n && (pl->tail.lane_par || (PAIRS && pl->tail.pair_par))) {
            // Counting level before the tail: every surviving lane sizes its own tail.  Lists
            // shared by the chunk (parent matched above this level) are searched by the warp
            // with a cursor, as the probe lists are: the chunk's candidates ascend.
            uint32_t shared_hit = 0;
            if (d >= 2) {
                const DevTail *T = &pl->tail;
                const uint32_t nkeys = __ldg(&T->nkeys);
                const uint32_t last = 31 - __clz(__ballot_sync(0xffffffffu, idx < S.hi[d]));
                const uint32_t key = cand << 1, top = __shfl_sync(0xffffffffu, key, last);
                const uint32_t psize = S.psz[S.bnb[d] + S.piv[d]];
                for (uint32_t k = 0; k < nkeys; k++) {
                    if (__ldg(&T->key_parent[k]) >= d || !((__ldg(&T->single) >> k) & 1u)) continue;
                    if (!((__ldg(&T->key_excl[k]) >> d) & 1u)) continue;  // candidates never in this list
                    if (!__any_sync(0xffffffffu, ok)) break;
                    const uint32_t size = S.ts_size[k];
                    uint32_t c0 = S.ts_cur[k];
                    const uint32_t e =
                        window_find(P.g.pool + S.ts_off[k], size, c0, first_window(size, psize), key, top, last);
                    __syncwarp();
                    if (lane == 0) S.ts_cur[k] = c0;
                    __syncwarp();
                    if (ok) {
                        probes++;
                        if (e != 0xFFFFFFFFu && key_counts(__ldg(&T->key_old[k]), e)) shared_hit |= 1u << k;
                    }
                }
                __syncwarp();
            }
            unsigned long long t = 0;
            if (PAIRS && pl->tail.pair_par) {
                t = tail_count_pairs(S, P, pl, d, ok, cand, shared_hit, probes);
                iter |= 7u;
            } else if (ok) {
                if (d == 1) {
                    const uint2 seed = seed_pair(P, pl, cand);
                    t = tail_count_lane(S.ts_base, S.f, P, pl, 1, seed.x, seed.y, 0, probes);
                    if (pl->seed_group == CSM_SEED_WEIGHT) t *= seed.y;
                } else {
                    t = tail_count_lane(S.ts_base, S.f, P, pl, d, 0, cand, shared_hit, probes);
                }
            }
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            cnt += t;
            tails += __popc(mask);
        } else if (d + 1 == n) {
            if (MODE == CSM_ENUM_MODE_ROWS) {
                const uint32_t c = __popc(mask);
                unsigned long long r = 0;
                if (lane == 0 && c) r = atomicAdd(&P.ctrl->out_rows, (unsigned long long)c);
                r = __shfl_sync(0xffffffffu, r, 0);
                if (c && r + c > P.row_cap) {
                    if (lane == 0) err |= CSM_ERRBIT_OUTPUT;
                } else if (ok) {
                    if (d == 1) {
                        const unsigned long long key = __ldg(P.keys + cand);
                        uint32_t *row = P.rows + (r + rank) * P.row_words;
                        row[0] = pl->query;
                        row[1 + pl->order[0]] = P.kl.src(key);
                        row[1 + pl->order[1]] = P.kl.dst(key);
                    } else {
                        write_row(P, pl, S, d, cand, r + rank);
                    }
                }
            }
            cnt += __popc(mask);
            __syncwarp();
        } else {
            if (ok) S.buf[d][rank] = cand;
            __syncwarp();
            if (lane == 0) {
                S.nbuf[d] = (uint8_t)__popc(mask);
                S.pos[d] = 0;
            }
            __syncwarp();
        }
    }
    return total + cnt * weight;
}

// MINB resident blocks of 256 threads per SM: the register budget per thread follows from it.
// MODE: CSM_ENUM_MODE_* of the launch (each variant holds only its mode's code, which keeps the
// hot loop's instruction footprint small).
template <int MINB, bool LASTLOOP, bool PAIRS, int MODE>
__global__ void __launch_bounds__(256, MINB) k_enumerate(EnumParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    WarpState &S = reinterpret_cast<WarpState *>(smem)[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    if (P.abort_flag != nullptr && *(volatile const unsigned int *)P.abort_flag) return;
    if (MODE == CSM_ENUM_MODE_EXPAND ? !P.ctrl->go : P.ctrl->halt) return;
    const uint32_t src = P.ctrl->src;
    const WorkItem *frontier = src == 0 ? nullptr : P.frontier[src - 1];
    WorkItem *expand_out = MODE == CSM_ENUM_MODE_EXPAND ? P.frontier[src == 1 ? 1 : 0] : nullptr;
    // Per-lane work counters (statistics only), 32-bit to keep registers for the search; a
    // lane flushes them to the launch totals before they could wrap.
    uint32_t scans = 0, probes = 0, tails = 0, shared = 0;
    unsigned int err = 0;
    const unsigned long long deadline = P.time_limit_ns ? P.ctrl->t_start + P.time_limit_ns : 0ull;
    bool have_source = true;  // seed tickets / frontier not yet exhausted
    // A warp counts as active from its start: blocks that become resident late (the GPU shared
    // with other kernels, or more blocks than fit) join the count when they start, so warps
    // that ran out of work never wait for blocks that have not started.
    if (P.donate) {
        if (threadIdx.x == 0) atomicAdd(&P.ctrl->active, blockDim.x >> 5);
        __syncthreads();
    }
    while (!(err & CSM_ERRBIT_TIMEOUT)) {
        if (deadline) {
            unsigned int late = 0;
            if (lane == 0) late = device_ns() > deadline;
            if (__shfl_sync(0xffffffffu, late, 0)) {
                err |= CSM_ERRBIT_TIMEOUT;
                break;
            }
        }
        int got = 0;
        if (have_source) {
            got = take_ticket(S, P, frontier);
            if (got < 0) continue;  // a frontier item that failed its check
            if (!got) have_source = false;
        }
        if (!got) {
            if (!P.donate) break;  // nothing is handed out in this launch
            got = await_item(S, P, err, deadline);
            if (got < 0) continue;
            if (!got) break;
        }
        const unsigned long long c = run_item<LASTLOOP, PAIRS, MODE>(S, P, scans, probes, tails, shared, err, deadline, expand_out);
        if (lane == 0 && c) atomicAdd(P.counts + S.item_plan, c);
        if ((scans | probes | tails | shared) >= (1u << 30)) {
            atomicAdd(&P.ctrl->scan_entries, (unsigned long long)scans);
            atomicAdd(&P.ctrl->probes, (unsigned long long)probes);
            // The tail and shared-level counters are warp-uniform: one lane adds them.
            if (lane == 0) atomicAdd(&P.ctrl->tail_lists, (unsigned long long)tails);
            if (lane == 0) atomicAdd(&P.ctrl->shared_last, (unsigned long long)shared);
            scans = probes = tails = shared = 0;
        }
        __syncwarp();
    }
    unsigned long long scans64 = scans, probes64 = probes;
    for (int o = 16; o > 0; o >>= 1) {
        scans64 += __shfl_xor_sync(0xffffffffu, scans64, o);
        probes64 += __shfl_xor_sync(0xffffffffu, probes64, o);
    }
    if (lane == 0) {
        if (scans64) atomicAdd(&P.ctrl->scan_entries, scans64);
        if (probes64) atomicAdd(&P.ctrl->probes, probes64);
        if (tails) atomicAdd(&P.ctrl->tail_lists, (unsigned long long)tails);
        if (shared) atomicAdd(&P.ctrl->shared_last, (unsigned long long)shared);
        if (err) atomicOr(&P.ctrl->error, err);
    }
}

// Plan p: the key range of its seed relation, and the number of 32-key seed chunks.  A warp and a
// 32-ary search: about log32(m) dependent reads for each end.
__device__ void seed_range(const DevPlan *plans, uint32_t nplans, uint32_t p, const unsigned long long *keys, uint32_t m,
                           KeyLayout kl, uint32_t *seed_lo, uint32_t *chunks) {
    const uint32_t lane = lane_id();
    const uint32_t rel = plans[p].seed_rel;
    uint32_t end[2];
#pragma unroll
    for (uint32_t e = 0; e < 2; e++) {
        // First key whose relation is at least rel + e.
        uint32_t lo = e ? end[0] : 0u, hi = m;
        while (hi > lo) {
            const uint32_t step = (hi - lo + 31u) / 32u;
            const uint32_t i = lo + (lane + 1) * step - 1;
            const bool below = i < hi && kl.rel(__ldg(keys + i)) < rel + e;
            const uint32_t c = __popc(__ballot_sync(0xffffffffu, below));
            const uint32_t nhi = lo + (c + 1) * step - 1;
            lo += c * step;
            hi = nhi < hi ? nhi : hi;
            if (lo > hi) lo = hi;
        }
        end[e] = lo;
    }
    if (lane == 0) {
        seed_lo[p] = end[0];
        seed_lo[nplans + p] = end[1];
        chunks[p] = (end[1] - end[0] + 31u) / 32u;
    }
}

// Exclusive prefix of chunk counts, by one block of 1024 threads.
__device__ void ticket_prefix(const uint32_t *chunks, uint32_t nplans, uint32_t *prefix) {
    __shared__ uint32_t part[32];
    const uint32_t t = threadIdx.x, lane = lane_id();
    const uint32_t per = (nplans + blockDim.x - 1) / blockDim.x;
    uint32_t s = 0;
    for (uint32_t i = t * per; i < (t + 1) * per && i < nplans; i++) s += chunks[i];
    uint32_t incl = s;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    if (lane == 31) part[t >> 5] = incl;
    __syncthreads();
    if (t < 32) {
        uint32_t w = part[t];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += v;
        }
        part[t] = w;
    }
    __syncthreads();
    uint32_t acc = incl - s + (t >= 32 ? part[(t >> 5) - 1] : 0u);
    for (uint32_t i = t * per; i < (t + 1) * per && i < nplans; i++) {
        prefix[i] = acc;
        acc += chunks[i];
    }
    if (t == blockDim.x - 1) prefix[nplans] = acc;
}

// One block finds the ranges of few plans and their prefix in one launch; more plans (32 warps take
// more than four turns) get a grid for the ranges and a launch for the prefix.
constexpr uint32_t kOneBlockPlans = 128;

__global__ void __launch_bounds__(1024) k_seed_tickets(const DevPlan *plans, uint32_t nplans, const unsigned long long *keys,
                                                       uint32_t m, KeyLayout kl, uint32_t *seed_lo, uint32_t *chunks,
                                                       uint32_t *prefix) {
    for (uint32_t p = threadIdx.x >> 5; p < nplans; p += blockDim.x >> 5)
        seed_range(plans, nplans, p, keys, m, kl, seed_lo, chunks);
    __syncthreads();
    ticket_prefix(chunks, nplans, prefix);
}

__global__ void k_seed_ranges(const DevPlan *plans, uint32_t nplans, const unsigned long long *keys, uint32_t m,
                              KeyLayout kl, uint32_t *seed_lo, uint32_t *chunks) {
    const uint32_t p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (p < nplans) seed_range(plans, nplans, p, keys, m, kl, seed_lo, chunks);
}

__global__ void __launch_bounds__(1024) k_ticket_prefix(const uint32_t *chunks, uint32_t nplans, uint32_t *prefix) {
    ticket_prefix(chunks, nplans, prefix);
}

// Resets the control block for one phase.  The phase epoch (which marks queue slots ready) is the
// previous one plus one, kept on the device so that every phase on this scratch gets a fresh epoch
// whichever engine, stream or replayed graph issues it.
__global__ void k_phase_begin(EnumControl *ctrl, const uint32_t *nticket, uint32_t expand, unsigned long long target,
                              unsigned long long frontier_cap, unsigned int *pair_phase) {
    uint32_t *w = reinterpret_cast<uint32_t *>(ctrl);
    uint32_t epoch = ctrl->epoch + 1u;
    if (epoch == 0) epoch = 1;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < sizeof(EnumControl) / 4; i += blockDim.x) w[i] = 0u;
    __syncthreads();
    if (threadIdx.x != 0) return;
    const unsigned long long seeds = 32ull * *nticket;  // upper bound
    ctrl->epoch = epoch;
    ctrl->nticket = *nticket;
    ctrl->go = expand && seeds > 0 && seeds < target && seeds <= frontier_cap;
    ctrl->t_start = device_ns();
    if (pair_phase) ctrl->pair_phase = *pair_phase = *pair_phase + 1u;
}

// Tail values of the pendant plans (DevPlan.memo_tail): for every data vertex w at the counting level,
// the deep tail classes' count below it, without exclusions.  No prefix vertex can sit in their lists, but
// for the cut vertices (DevPlan.memo_cut), which settle_pendant takes off.  blockIdx.y names the table;
// the first of those that share tail values fills them.
__global__ void k_tail_values(EnumParams P, const uint32_t *desc, unsigned long long *memo) {
    const DevPlan *pl = P.plans + desc[3 * blockIdx.y];
    const uint32_t slot = desc[3 * blockIdx.y + 2];
    for (uint32_t t = 0; t < blockIdx.y; t++)
        if (desc[3 * t + 2] == slot) return;
    unsigned long long *out = memo + (size_t)slot * P.g.V;
    const DevTail *T = &pl->tail;
    const uint32_t c = pl->tail_start - 1u, nkeys = __ldg(&T->nkeys), deep = __ldg(&T->deep);
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < P.g.V; w += gridDim.x * blockDim.x) {
        uint32_t ksize[CSM_TAIL_MAXKEYS];
#pragma unroll 1
        for (uint32_t k = 0; k < nkeys; k++) {
            ksize[k] = 0;
            if (__ldg(&T->key_parent[k]) != c) continue;
            const uint32_t rel = __ldg(&T->key_rel[k]);
            const uint2 ms = list_of(P, rel, w, 900 + c);
            if (ms.y) ksize[k] = key_entries(P, rel, w, ms.y, __ldg(&T->key_old[k]));
        }
        out[w] = tail_product(P, pl, ksize, deep);
    }
}

// Table of a pendant plan (DevPlan.memo_slot): for every data vertex v, the count of its counting
// level c for a prefix whose vertex at memo_depth is v — the sum of the tail values of v's list
// under the flag rule and c's NLF filter.  A lane looks at one vertex (most have no list in the
// relation); the warp then scans the lists found, 32 entries at a time.
__global__ void k_pendant_counts(EnumParams P, const uint32_t *desc, unsigned long long *memo) {
    const uint32_t lane = threadIdx.x & 31u;
    const DevPlan *pl = P.plans + desc[3 * blockIdx.y];
    unsigned long long *out = memo + (size_t)desc[3 * blockIdx.y + 1] * P.g.V;
    const unsigned long long *value = memo + (size_t)desc[3 * blockIdx.y + 2] * P.g.V;
    const uint32_t c = pl->tail_start - 1u;
    const DevLevel *lv = &pl->lv[c];
    const uint32_t rel = __ldg(&lv->bn_rel[0]);
    const bool old = (__ldg(&lv->old_mask) & 1u) != 0;
    const uint32_t nlf_id = __ldg(&lv->nlf_bitmap);
    const uint32_t *nlf = nlf_id == CSM_NO_BITMAP ? nullptr : bitmap(P, nlf_id);
    uint32_t scans = 0;
    const uint32_t nw = gridDim.x * (blockDim.x >> 5);
    for (uint32_t base = 32u * (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); base < P.g.V; base += 32u * nw) {
        const uint32_t v = base + lane;
        const uint2 ms = v < P.g.V ? list_of(P, rel, v, 900 + c) : make_uint2(0u, 0u);
        unsigned long long mine = 0;
        for (uint32_t todo = __ballot_sync(0xffffffffu, ms.y != 0); todo; todo &= todo - 1) {
            const uint32_t l = __ffs(todo) - 1;
            const uint32_t off = __shfl_sync(0xffffffffu, ms.x, l), size = __shfl_sync(0xffffffffu, ms.y, l);
            unsigned long long acc = 0;
            for (uint32_t i = lane; i < size; i += 32) {
                const uint32_t e = __ldg(P.g.pool + off + i), w = e >> 1;
                scans++;
                bool ok = !(old && (e & 1u));
                if (w >= P.g.V) {
                    record_bad(P, CSM_BAD_ENTRY, e, off + i, 900 + c);
                    ok = false;
                }
                if (ok && (!nlf || test_bit(nlf, w))) acc += value[w];
            }
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == l) mine = acc;
        }
        if (v < P.g.V) out[v] = mine;
    }
    unsigned long long s64 = scans;
    for (int o = 16; o > 0; o >>= 1) s64 += __shfl_xor_sync(0xffffffffu, s64, o);
    if (lane == 0 && s64) atomicAdd(&P.ctrl->scan_entries, s64);
}

// Between two expansion launches.  The level just written becomes the source of the next launch,
// and the last block to finish decides whether that launch expands it further: only when an upper
// bound of what it would write (the sum of every item's smallest candidate list) fits the frontier,
// so no level overflows.  Deciding here instead of on the host takes two host synchronisations out
// of every level (64 updates, batch and inverse: 0.74 -> 0.51 ms; netflow 262,144: 22 -> 13 ms);
// launches after the last level find go == 0 and return.
__global__ void k_expand_decide(EnumParams P, uint32_t last, unsigned long long target) {
    EnumControl *ctrl = P.ctrl;
    if (!ctrl->go) return;  // no expansion ran: the state is already the counting launch's
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t out = ctrl->src == 1 ? 1u : 0u;  // the buffer the expansion wrote
    const unsigned long long n = ctrl->out_rows;
    const bool failed = (ctrl->error & (CSM_ERRBIT_FRONTIER | CSM_ERRBIT_TIMEOUT | CSM_ERRBIT_CORRUPT)) != 0;
    const bool stop = failed || last || n == 0 || n >= target;
    if (!stop) {
        const unsigned long long nw = (unsigned long long)gridDim.x * (blockDim.x >> 5);
        unsigned long long acc = 0;
        for (unsigned long long i = (blockIdx.x * (blockDim.x >> 5)) + (threadIdx.x >> 5); i < n; i += nw) {
            const WorkItem *it = P.frontier[out] + i;
            const DevPlan *pl = P.plans + it->plan;
            const uint32_t d = it->depth;
            if (d == 0 || d >= pl->expand_stop) {
                if (lane == 0) acc += 1;  // passes through unchanged (seed chunks of plans that expand nothing too)
                continue;
            }
            const DevLevel *lv = &pl->lv[d];
            uint32_t sz = 0xFFFFFFFFu;
            if (lane < lv->nbn) sz = list_of(P, lv->bn_rel[lane], it->f[lv->bn_depth[lane]], 800 + d).y;
            for (int o = 16; o > 0; o >>= 1) sz = min(sz, __shfl_xor_sync(0xffffffffu, sz, o));
            if (lane == 0) acc += sz;
        }
        if (lane == 0 && acc) atomicAdd(&ctrl->expand_bound, acc);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x != 0 || atomicAdd(&ctrl->blocks_done, 1u) != gridDim.x - 1) return;
    __threadfence();
    ctrl->blocks_done = 0;
    ctrl->levels++;
    if (failed) {
        ctrl->halt = 1;
        ctrl->go = 0;
        return;
    }
    ctrl->src = 1 + out;
    ctrl->ticket = 0;
    ctrl->nticket = n;
    ctrl->out_rows = 0;
    if (n > ctrl->max_front) ctrl->max_front = n;
    ctrl->go = !stop && *(volatile unsigned long long *)&ctrl->expand_bound <= P.frontier_cap;
    ctrl->expand_bound = 0;
    ctrl->t_start = device_ns();
}

}  // namespace

size_t enum_smem_bytes(int warps_per_block) { return sizeof(WarpState) * (size_t)warps_per_block; }

namespace {
using EnumKernel = void (*)(EnumParams);
template <int MINB>
EnumKernel enum_kernel_mode(bool last_loop, bool pairs, uint32_t mode) {
    if (mode == CSM_ENUM_MODE_EXPAND) return k_enumerate<MINB, false, false, CSM_ENUM_MODE_EXPAND>;
    if (mode == CSM_ENUM_MODE_ROWS) return k_enumerate<MINB, false, false, CSM_ENUM_MODE_ROWS>;
    if (pairs)
        return last_loop ? k_enumerate<MINB, true, true, CSM_ENUM_MODE_COUNT> : k_enumerate<MINB, false, true, CSM_ENUM_MODE_COUNT>;
    return last_loop ? k_enumerate<MINB, true, false, CSM_ENUM_MODE_COUNT> : k_enumerate<MINB, false, false, CSM_ENUM_MODE_COUNT>;
}

EnumKernel enum_kernel(int occupancy, bool last_loop, bool pairs, uint32_t mode) {
    switch (occupancy) {
        case 6: return enum_kernel_mode<6>(last_loop, pairs, mode);
        case 5: return enum_kernel_mode<5>(last_loop, pairs, mode);
        default: return enum_kernel_mode<4>(last_loop, pairs, mode);
    }
}
}  // namespace

int enum_blocks_per_sm(int warps_per_block, int occupancy) {
    // The smallest residency of the variants: a persistent grid must fit each of them.
    const size_t smem = enum_smem_bytes(warps_per_block);
    int best = 1 << 30;
    for (int v = 0; v < 6; v++) {
        EnumKernel k = enum_kernel(occupancy, v & 1, v & 2, v < 4 ? CSM_ENUM_MODE_COUNT : (uint32_t)(v - 3));
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int nb = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, warps_per_block * 32, smem) != cudaSuccess) return 1;
        best = nb < best ? nb : best;
    }
    return best > 0 ? best : 1;
}

void launch_enumerate(const EnumParams &p, int blocks, int warps_per_block, int occupancy, cudaStream_t s) {
    const size_t smem = enum_smem_bytes(warps_per_block);
    EnumKernel k = enum_kernel(occupancy, p.last_loop != 0, p.pairs != nullptr, p.mode);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<blocks, warps_per_block * 32, smem, s>>>(p);
}

void launch_seed_tickets(const DevPlan *plans, uint32_t nplans, const unsigned long long *keys, uint32_t m,
                         KeyLayout kl, uint32_t *seed_lo, uint32_t *ticket_prefix, cudaStream_t s) {
    // seed_lo holds three arrays of nplans: first key, end key, chunk count.
    uint32_t *chunks = seed_lo + 2 * nplans;
    if (nplans <= kOneBlockPlans) {
        k_seed_tickets<<<1, 1024, 0, s>>>(plans, nplans, keys, m, kl, seed_lo, chunks, ticket_prefix);
        return;
    }
    k_seed_ranges<<<(nplans + 3) / 4, 128, 0, s>>>(plans, nplans, keys, m, kl, seed_lo, chunks);
    k_ticket_prefix<<<1, 1024, 0, s>>>(chunks, nplans, ticket_prefix);
}

void launch_phase_begin(EnumControl *ctrl, const uint32_t *ticket_prefix, uint32_t nplans, bool expand,
                        unsigned long long target, unsigned long long frontier_cap, unsigned int *pair_phase,
                        cudaStream_t s) {
    k_phase_begin<<<1, 128, 0, s>>>(ctrl, ticket_prefix + nplans, expand ? 1u : 0u, target, frontier_cap, pair_phase);
}

void launch_expand_decide(const EnumParams &p, bool last, unsigned long long target, cudaStream_t s) {
    k_expand_decide<<<296, 256, 0, s>>>(p, last ? 1u : 0u, target);
}

void launch_pendant_tables(const EnumParams &p, const uint32_t *desc, uint32_t ntables, unsigned long long *memo,
                           cudaStream_t s) {
    // Enough blocks for one pass over the vertices, at most eight per SM and table.
    const uint32_t blocks = p.g.V / 256u + 1u < 148u * 8u ? p.g.V / 256u + 1u : 148u * 8u;
    k_tail_values<<<dim3(blocks, ntables), 256, 0, s>>>(p, desc, memo);
    k_pendant_counts<<<dim3(blocks, ntables), 256, 0, s>>>(p, desc, memo);
}

}  // namespace csm
