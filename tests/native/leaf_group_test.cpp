// Host-only check of group_leaf_seeds and extend_pendant (gcsm-bu_b200/csrc/plan.cpp): on random
// labelled queries and random data graphs with some edges marked as batch edges, the plan that starts
// once per data vertex of the inner endpoint, and the plan whose counting level is settled from
// per-vertex sums, count what the plan that starts at every batch edge counts.  All device forms are
// evaluated by the same small interpreter (levels, flag rules, exclusions, candidate bitmaps, tail
// polynomial, tables).
#include <algorithm>
#include <cstdio>
#include <map>
#include <random>
#include <set>
#include <tuple>
#include <vector>

#include "plan.h"
#include "query.h"

using namespace csm;

namespace {

struct Entry {
    uint32_t v;
    bool batch;
};

struct Graph {
    uint32_t n = 0;
    std::map<std::pair<int, uint32_t>, std::vector<Entry>> lists;  // (relation, vertex)
    const std::vector<Entry> &list(int rel, uint32_t v) const {
        static const std::vector<Entry> none;
        auto it = lists.find({rel, v});
        return it == lists.end() ? none : it->second;
    }
    // 0 = absent, 1 = present, 2 = present and a batch edge
    int entry(int rel, uint32_t v, uint32_t w) const {
        for (const Entry &e : list(rel, v))
            if (e.v == w) return e.batch ? 2 : 1;
        return 0;
    }
    // Candidate bitmaps (the NLF rule): per bitmap the groups that a vertex needs, a relation and how many
    // neighbours in it.
    std::vector<std::vector<std::pair<int, uint32_t>>> groups;
    bool candidate(uint32_t bitmap, uint32_t v) const {
        if (bitmap == CSM_NO_BITMAP) return true;
        for (auto &g : groups[bitmap])
            if (list(g.first, v).size() < g.second) return false;
        return true;
    }
};

bool counts(int rule, bool batch) { return rule == CSM_KEY_ANY || batch == (rule == CSM_KEY_BATCH); }

// The tail classes in `classes` for the prefix f; `depths` of it are set.
long long tail(const Graph &g, const DevPlan &p, const std::vector<DevTailTerm> &terms, const uint32_t *f,
               unsigned classes, int depths) {
    const DevTail &t = p.tail;
    std::vector<long long> size(t.nmasks, 0);
    for (int mi = 0; mi < t.nmasks; mi++)
        for (uint32_t w = 0; w < g.n; w++) {
            if (t.key_parent[__builtin_ctz(t.mask[mi])] >= depths) continue;  // of a class not asked for
            bool ok = true;
            for (int k = 0; ok && k < t.nkeys; k++) {
                if (!((t.mask[mi] >> k) & 1u)) continue;
                const int e = g.entry(t.key_rel[k], f[t.key_parent[k]], w);
                ok = e && counts(t.key_old[k], e == 2);
                for (int j = 0; ok && j < depths; j++)
                    if (((t.key_excl[k] >> j) & 1u) && f[j] == w) ok = false;
            }
            size[mi] += ok;
        }
    long long total = 1;
    for (int c = 0; c < t.nclasses; c++) {
        if (!((classes >> c) & 1u)) continue;
        long long s = 0;
        for (int i = t.class_term_begin[c]; i < t.class_term_begin[c + 1]; i++) {
            long long prod = terms[i].coef;
            for (int j = 0; j < terms[i].nf; j++) prod *= size[terms[i].f[j]];
            s += prod;
        }
        total *= s;
    }
    return total;
}

// What hangs off vertex w at the counting level alone: a table entry of its own.
long long tail_value(const Graph &g, const DevPlan &p, const std::vector<DevTailTerm> &terms, uint32_t w) {
    uint32_t f[CSM_MAXQV];
    std::fill(f, f + CSM_MAXQV, 0xFFFFFFFFu);  // no prefix
    f[p.tail_start - 1] = w;
    return tail(g, p, terms, f, p.tail.deep, p.tail_start);
}

// Vertices in list (ra, a) and in list (rb, b), each under its rule.
long long common(const Graph &g, int ra, uint32_t a, int rule_a, int rb, uint32_t b, int rule_b) {
    long long n = 0;
    for (const Entry &e : g.list(ra, a)) {
        const int x = g.entry(rb, b, e.v);
        n += counts(rule_a, e.batch) && x && counts(rule_b, x == 2);
    }
    return n;
}

// A pendant counting level below the prefix f[0..c-1]: the sum over its list, without exclusions, less
// the prefix vertices that the sum should not hold, times what hangs off the prefix.  As on the device, the
// cut vertices are taken off without a look at the level's candidate bitmap: where extend_pendant allows a cut,
// a vertex next to a cut vertex passes it.
long long settle(const Graph &g, const DevPlan &p, const std::vector<DevTailTerm> &terms, const uint32_t *f) {
    const int c = p.tail_start - 1, md = p.memo_depth;
    const DevLevel &lv = p.lv[c];
    const bool old = lv.old_mask & 1u;
    long long sum = 0;
    for (const Entry &e : g.list(lv.bn_rel[0], f[md]))
        if (!(old && e.batch) && g.candidate(lv.nlf_bitmap, e.v)) sum += tail_value(g, p, terms, e.v);
    for (int j = 0; j < c; j++) {
        if (!((lv.excl_mask >> j) & 1u) || j == md) continue;
        const int x = g.entry(lv.bn_rel[0], f[md], f[j]);
        if (!x || (old && x == 2) || !g.candidate(lv.nlf_bitmap, f[j])) continue;
        sum -= tail_value(g, p, terms, f[j]);
        for (int i = 0; i < c; i++) {
            if (!((p.memo_cut >> i) & 1u)) continue;
            const int y = g.entry(p.tail.key_rel[p.cut_key], f[j], f[i]);
            sum += y && counts(p.tail.key_old[p.cut_key], y == 2);
        }
    }
    for (int i = 0; i < c; i++)
        if ((p.memo_cut >> i) & 1u)
            sum -= common(g, lv.bn_rel[0], f[md], old ? CSM_KEY_OLD : CSM_KEY_ANY, p.cut_rel, f[i], p.tail.key_old[p.cut_key]);
    return sum * tail(g, p, terms, f, ~(unsigned)p.tail.deep, c);
}

long long walk(const Graph &g, const DevPlan &p, const std::vector<DevTailTerm> &terms, uint32_t *f, int d) {
    if (d == p.n) return 1;
    if (p.memo_slot == CSM_MEMO_PENDING && d + 1 == p.tail_start) return settle(g, p, terms, f);
    if (d == p.tail_start) return tail(g, p, terms, f, ~0u, d);
    const DevLevel &lv = p.lv[d];
    long long total = 0;
    for (const Entry &e : g.list(lv.bn_rel[0], f[lv.bn_depth[0]])) {
        bool ok = true;
        for (int k = 0; ok && k < lv.nbn; k++) {
            const int x = g.entry(lv.bn_rel[k], f[lv.bn_depth[k]], e.v);
            ok = x && !(((lv.old_mask >> k) & 1u) && x == 2);
        }
        for (int j = 0; ok && j < d; j++)
            if (((lv.excl_mask >> j) & 1u) && f[j] == e.v) ok = false;
        if (!ok || !g.candidate(lv.nlf_bitmap, e.v)) continue;
        f[d] = e.v;
        total += walk(g, p, terms, f, d + 1);
    }
    return total;
}

long long count(const Graph &g, const DevPlan &p, const std::vector<DevTailTerm> &terms) {
    long long total = 0;
    for (uint32_t v = 0; v < g.n; v++) {
        uint32_t batch = 0;
        for (const Entry &e : g.list(p.seed_rel, v)) batch += e.batch;
        // The position without a query vertex holds a number: it must never be read as a vertex.
        uint32_t f[CSM_MAXQV] = {v, batch};
        if (!g.candidate(p.nlf0, v)) continue;
        if (p.seed_group != CSM_SEED_EDGE) {
            if (batch) total += (p.seed_group == CSM_SEED_WEIGHT ? batch : 1) * walk(g, p, terms, f, 2);
            continue;
        }
        for (const Entry &e : g.list(p.seed_rel, v)) {
            if (!e.batch || !g.candidate(p.nlf1, e.v)) continue;
            f[1] = e.v;
            total += walk(g, p, terms, f, 2);
        }
    }
    return total;
}

}  // namespace

int main() {
    std::mt19937 rng(77);
    int grouped[3] = {0, 0, 0}, nonzero = 0, pendant = 0, cut = 0, kept = 0;
    for (int qn = 0; qn < 600; qn++) {
        const uint32_t nv = 2 + rng() % 6, nlab = 1 + rng() % 4;
        std::vector<uint32_t> vl(nv), src, dst, el;
        for (auto &x : vl) x = rng() % nlab;
        std::set<std::pair<uint32_t, uint32_t>> seen;
        for (uint32_t v = 1; v < nv; v++) {
            const uint32_t p = rng() % v;
            src.push_back(p), dst.push_back(v), el.push_back(rng() % 2);
            seen.insert({p, v});
        }
        for (int e = (int)(rng() % 3); e > 0; e--) {
            uint32_t a = rng() % nv, b = rng() % nv;
            if (a > b) std::swap(a, b);
            if (a == b || !seen.insert({a, b}).second) continue;
            src.push_back(a), dst.push_back(b), el.push_back(rng() % 2);
        }
        Query q;
        if (!build_query(nv, vl.data(), (uint32_t)src.size(), src.data(), dst.data(), el.data(), q).empty()) return 1;
        std::map<std::tuple<uint32_t, uint32_t, uint32_t>, uint16_t> rels;
        RelOf rel_of = [&](uint32_t u, uint32_t uu) -> uint16_t {
            auto k = std::make_tuple(q.vlabel[u], q.edge_label(u, uu), q.vlabel[uu]);
            return rels.emplace(k, (uint16_t)rels.size()).first->second;
        };
        for (auto &e : q.qe_list) rel_of(e.first, e.second), rel_of(e.second, e.first);
        EdgeStats st;
        st.card.assign(nv * nv, 1);
        st.avg.assign(nv * nv, 1.f);
        for (auto &x : st.avg) x = 1.f + (float)(rng() % 100);
        PlanOptions po;
        po.order = (Order)(qn % 4);
        std::vector<HostPlan> plans = build_plans(q, 0, 0, st, po, rel_of);
        // A data graph of the query's labels; two labelled edges of one pair are two edges.
        Graph g;
        g.n = 14;
        std::vector<uint32_t> gl(g.n);
        for (auto &x : gl) x = rng() % nlab;
        for (uint32_t a = 0; a < g.n; a++)
            for (uint32_t b = a + 1; b < g.n; b++)
                for (uint32_t l = 0; l < 2; l++) {
                    if (rng() % 5 > 2) continue;
                    const bool batch = rng() % 3 == 0;
                    for (auto e : {std::make_pair(a, b), std::make_pair(b, a)}) {
                        auto it = rels.find(std::make_tuple(gl[e.first], l, gl[e.second]));
                        if (it != rels.end()) g.lists[{it->second, e.first}].push_back({e.second, batch});
                    }
                }
        g.groups.resize(nv);
        for (uint32_t u = 0; u < nv; u++)
            for (auto &grp : q.nlf[u])
                g.groups[u].push_back({rels.at(std::make_tuple(q.vlabel[u], grp.elabel, grp.vlabel)), (uint32_t)grp.count});
        for (size_t i = 0; i < plans.size(); i++) {
            HostPlan hp = plans[i];
            const long long want = count(g, plans[i].dev, plans[i].terms);
            const bool did = group_leaf_seeds(q, 0, rel_of, hp);
            grouped[hp.dev.seed_group]++;
            const auto &e = q.qe_list[i];
            if (did != (nv > 2 && (q.degree(e.first) == 1 || q.degree(e.second) == 1))) {
                std::printf("FAIL grouping of query %d plan %zu\n", qn, i);
                return 1;
            }
            const long long got = count(g, hp.dev, hp.terms);
            nonzero += did && want > 0;
            for (HostPlan ep : {plans[i], hp}) {
                if (!extend_pendant(q, rel_of, ep)) continue;
                const long long settled = count(g, ep.dev, ep.terms);
                pendant += want > 0;
                cut += want > 0 && ep.dev.memo_cut;
                if (settled != want) {
                    std::printf("FAIL query %d plan %zu: %lld settled, %lld counted\n", qn, i, settled, want);
                    return 1;
                }
            }
            HostPlan rp = plans[i];
            rewrite_plan(q, 0, rel_of, rp);
            if (count(g, rp.dev, rp.terms) != want) {
                std::printf("FAIL query %d plan %zu: its rewritten form counts otherwise than %lld\n", qn, i, want);
                return 1;
            }
            // A leaf in the tail must not cost the plan its counting of 32 prefixes at once.
            if (rp.dev.seed_group == CSM_SEED_TAIL && rp.dev.memo_slot == CSM_NO_MEMO && counted_by_lane(plans[i].dev) &&
                !counted_by_lane(rp.dev)) {
                std::printf("FAIL query %d plan %zu: grouped into a tail that is counted one prefix at a time\n", qn, i);
                return 1;
            }
            kept += did && rp.dev.seed_group == CSM_SEED_EDGE && !counted_by_lane(hp.dev);
            if (got != want) {
                std::printf("FAIL query %d plan %zu: %lld per inner vertex, %lld per batch edge\n", qn, i, got, want);
                return 1;
            }
        }
    }
    if (grouped[CSM_SEED_WEIGHT] < 50 || grouped[CSM_SEED_TAIL] < 50 || nonzero < 100 ||
        pendant < 50 || cut < 20 || kept < 5)
        return std::printf("too few plans: %d weighted, %d in the tail, %d of them with matches, %d pendant, %d cut, %d not grouped\n",
                           grouped[1], grouped[2], nonzero, pendant, cut, kept), 1;
    std::printf("ok %d weighted, %d in the tail, %d of them with matches, %d pendant, %d of them cut, %d not grouped\n", grouped[1], grouped[2],
                nonzero, pendant, cut, kept);
    return 0;
}
