// Matching-order planner.
//
// One plan per (query, updated query edge i).  The vertex-selection rules follow the
// reference's PlanManager (graph/plan.cpp): the BFS indexing order (plan.cpp:1548-1602),
// the GAMMA order (plan.cpp:1843-2116), the GCSM v2 order (plan.cpp:386-782) and the RI order
// (plan.cpp:195-385), with backward neighbours sorted by the average degree of their relation
// (plan.cpp:471-486).  Every order here starts with the endpoints of the updated edge, so that
// every partial embedding grows from a batch edge; where the reference's GCSM and RI rules
// pick another start, their vertex priority is kept and re-anchored at the updated edge.
#pragma once

#include <functional>
#include <string>
#include <vector>

#include "common.h"
#include "query.h"

namespace csm {

enum class Order { kIndexing = 0, kGamma = 1, kGcsm = 2, kRi = 3 };

struct PlanOptions {
    Order order = Order::kGcsm;
    bool cartesian = true;
    bool materialize = false;
};

// Summary of the candidate index per directed query edge (GetSummary, match_gpu.cu:589-609):
// card[u*nv+uu] = number of candidate edges, avg[u*nv+uu] = card / number of sources.
struct EdgeStats {
    std::vector<uint32_t> card;
    std::vector<float> avg;
};

struct HostPlan {
    std::vector<uint8_t> order;                 // query vertices by depth
    std::vector<std::vector<uint8_t>> bn;       // per depth: depths of backward neighbours
    int tail_start = 0;
    std::vector<DevTailTerm> terms;             // tail polynomial
    DevPlan dev;                                // packed form (term_begin set by the engine)
};

using RelOf = std::function<uint16_t(uint32_t u, uint32_t uu)>;  // relation of query edge u->uu

// Builds the plans of every query edge of `q`, in qe_list_ order.
std::vector<HostPlan> build_plans(const Query &q, uint16_t query_id, uint32_t nlf_base,
                                  const EdgeStats &st, const PlanOptions &opt, const RelOf &rel_of);

// Rewrites the device form of the plan of a query edge with a leaf endpoint so that its seeds are
// the data vertices of the inner endpoint instead of the batch edges (DevPlan.seed_group); order,
// bn and tail_start keep describing the plan it stands for.  Returns whether it did: not for edges
// without a leaf, queries of two vertices or row-materialising plans, nor where the leaf has to be counted
// in the tail and the query has CSM_MAXQV vertices or the tail would exceed the device tables.
bool group_leaf_seeds(const Query &q, uint32_t nlf_base, const RelOf &rel_of, HostPlan &hp);

// Whether a plan has a tail that is counted for 32 prefixes at once: its masks are single keys, pairs, or
// triples with two keys above the counting level.
bool counted_by_lane(const DevPlan &dp);

// Marks the device form of a plan as pendant (DevPlan.memo_slot) where it is not already and its
// counting level allows it.  Returns whether it did.
bool extend_pendant(const Query &q, const RelOf &rel_of, HostPlan &hp);

// Rewrites the device form of a plan as group_leaf_seeds and extend_pendant allow, where that is the form
// that counts faster.  Returns whether the plan was pendant without extend_pendant.
bool rewrite_plan(const Query &q, uint32_t nlf_base, const RelOf &rel_of, HostPlan &hp);

// Table slots (DevPlan.memo_slot, memo_tail) of the pendant plans of an engine.  Plans with the same
// counting level and deep tail classes read one table: its entries do not depend on the depths or on the
// query.  The tail values it sums are a table too, shared by what hangs off the counting vertex alone.
// At most `max_sums` tables of sums, and `max_tables` with the tail values; further plans stay CSM_MEMO_PENDING.  Plans marked in `first` (those
// that are pendant without extend_pendant) come first, whatever queries were registered before theirs: such
// a query after twenty that need extend_pendant took 10.2 ms at 250,007 updates, before them 5.2.
// Returns, per table of sums: a plan that reads it, its slot, the slot of its tail values.
std::vector<uint32_t> assign_pendant_tables(std::vector<HostPlan> &plans, const std::vector<char> &first, size_t max_sums,
                                            size_t max_tables, size_t &ntables);

// Text description, one block per query edge, in the spirit of PlanManager::PrintOrders.
std::string describe_plans(const Query &q, const std::vector<HostPlan> &plans);

// Exposed for tests: the bare vertex orders.
std::vector<uint8_t> indexing_order(const Query &q, uint32_t u0, uint32_t u1);

}  // namespace csm
