// Host check of assign_pendant_tables (gcsm-bu_b200/csrc/plan.cpp): which pendant plans of an engine get a
// table, and which share one.
#include <cstdio>
#include <map>
#include <random>
#include <tuple>
#include <utility>
#include <vector>

#include "plan.h"
#include "query.h"

using namespace csm;

namespace {

struct Plans {
    std::vector<HostPlan> plans;
    std::vector<char> own;  // pendant without extend_pendant
    std::vector<int> query;
    std::map<std::tuple<uint32_t, uint32_t, uint32_t>, uint16_t> rels;
    uint32_t bitmaps = 0;
    int nq = 0;

    bool add(const std::vector<uint32_t> &vl, const std::vector<std::pair<uint32_t, uint32_t>> &edges) {
        std::vector<uint32_t> src, dst, el(edges.size(), 0);
        for (auto &e : edges) src.push_back(e.first), dst.push_back(e.second);
        Query q;
        if (!build_query((uint32_t)vl.size(), vl.data(), (uint32_t)edges.size(), src.data(), dst.data(), el.data(), q).empty())
            return false;
        RelOf rel_of = [&](uint32_t u, uint32_t uu) -> uint16_t {
            auto k = std::make_tuple(q.vlabel[u], q.edge_label(u, uu), q.vlabel[uu]);
            return rels.emplace(k, (uint16_t)rels.size()).first->second;
        };
        EdgeStats st;
        st.card.assign(q.nv * q.nv, 1);
        st.avg.assign(q.nv * q.nv, 1.f);
        for (HostPlan &hp : build_plans(q, (uint16_t)nq, bitmaps, st, PlanOptions{}, rel_of)) {
            own.push_back(hp.dev.memo_slot == CSM_MEMO_PENDING);
            extend_pendant(q, rel_of, hp);
            plans.push_back(hp);
            query.push_back(nq);
        }
        bitmaps += q.nv;
        nq++;
        return true;
    }
};

#define CHECK(c) \
    if (!(c)) return std::printf("FAIL line %d: %s\n", __LINE__, #c), 1

}  // namespace

int main() {
    // Twenty queries whose prefix shares a label with the counting level or its tail, then one that is
    // pendant as it stands.
    Plans p;
    std::mt19937 rng(3);
    for (uint32_t i = 0; i < 20; i++) {
        const uint32_t a = 10 + i, b = 40 + i, c = 70 + i, e = 100 + i;
        CHECK(p.add(i % 2 ? std::vector<uint32_t>{a, b, c, a, e} : std::vector<uint32_t>{a, b, c, b, e},
                    {{0, 1}, {1, 2}, {2, 3}, {3, 4}}));
    }
    const int last = p.nq;
    CHECK(p.add({0, 1, 2, 3, 4, 5}, {{0, 1}, {1, 2}, {2, 0}, {2, 3}, {3, 4}, {4, 5}}));
    int own = 0, extended = 0;
    for (size_t i = 0; i < p.plans.size(); i++) {
        own += p.own[i] && p.query[i] == last;
        extended += !p.own[i] && p.plans[i].dev.memo_slot == CSM_MEMO_PENDING;
    }
    CHECK(own > 0 && extended > 16);
    for (auto [max_sums, max_tables] : {std::pair<size_t, size_t>{0, 400}, {1, 400}, {16, 400}, {16, 32}, {16, 20}, {16, 7},
                                        {16, 1}, {16, 0}, {200, 400}}) {
        std::vector<HostPlan> plans = p.plans;
        size_t ntables = 0;
        const std::vector<uint32_t> tables = assign_pendant_tables(plans, p.own, max_sums, max_tables, ntables);
        const size_t sums = tables.size() / 3;
        CHECK(sums <= max_sums && ntables <= 2 * sums && ntables >= sums && ntables <= max_tables);
        CHECK(max_tables > 20 || sums >= max_tables / 2);  // the room there is gets used
        int with = 0, without = 0;
        for (size_t i = 0; i < plans.size(); i++) {
            const DevPlan &dp = plans[i].dev;
            if (dp.memo_slot == CSM_NO_MEMO) continue;
            if (dp.memo_slot == CSM_MEMO_PENDING) {
                without++;
                // A plan goes without only when no table is left.
                CHECK((sums == max_sums || ntables + 2 > max_tables) && (max_sums < 16 || max_tables < 20 || !p.own[i]));
                continue;
            }
            with++;
            // Its table is described by a plan with the same counting level.
            bool found = false;
            for (size_t t = 0; t < sums; t++) {
                const DevPlan &rep = plans[tables[3 * t]].dev;
                if (tables[3 * t + 1] != dp.memo_slot) continue;
                found = rep.memo_slot == dp.memo_slot && rep.memo_tail == dp.memo_tail && tables[3 * t + 2] == dp.memo_tail &&
                        rep.lv[rep.tail_start - 1].bn_rel[0] == dp.lv[dp.tail_start - 1].bn_rel[0] &&
                        rep.lv[rep.tail_start - 1].nlf_bitmap == dp.lv[dp.tail_start - 1].nlf_bitmap;
            }
            CHECK(found && dp.memo_slot < ntables && dp.memo_tail < dp.memo_slot);
        }
        CHECK(with + without == own + extended);
        CHECK(max_sums < 200 || without == 0);
    }
    std::printf("ok %d plans pendant as they stand, %d extended\n", own, extended);
    return 0;
}
