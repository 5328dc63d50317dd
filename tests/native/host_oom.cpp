// A batch with rows whose host memory runs out: the call returns a status, and the engine refuses what follows,
// since the batch is only partly applied.  The failure is made here, by this program's operator new[].
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "../../include/csm.h"

static bool armed = false;

void *operator new[](std::size_t n) {
    if (armed && n > 4096) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete[](void *p) noexcept { std::free(p); }
void operator delete[](void *p, std::size_t) noexcept { std::free(p); }

#define CHECK(c) \
    if (!(c)) return std::printf("FAIL line %d: %s\n", __LINE__, #c), 1

int main() {
    csm_config cfg;
    csm_default_config(&cfg);
    cfg.materialize_rows = 1 << 16;
    cfg.frontier_bytes = 1 << 20;
    csm_engine *e = nullptr;
    CHECK(csm_create(&e, &cfg) == CSM_OK);
    // One edge as the query, its ends of one label: two rows for every edge of a batch.
    const uint32_t ql[] = {0, 0}, qs[] = {0}, qd[] = {1}, qe[] = {0};
    CHECK(csm_load_query(e, 2, ql, 1, qs, qd, qe, nullptr) == CSM_OK);
    const uint32_t n = 2000, m = n / 2;
    std::vector<uint32_t> vl(n, 0), s, d, l(m, 0);
    for (uint32_t i = 0; i < m; i++) s.push_back(2 * i), d.push_back(2 * i + 1);
    CHECK(csm_load_graph(e, n, vl.data(), m, s.data(), d.data(), l.data()) == CSM_OK);
    std::vector<uint8_t> del(m, 1);
    csm_batch_result r;
    CHECK(csm_apply_batch(e, 10, s.data(), d.data(), l.data(), del.data(), &r) == CSM_OK && r.negative == 20);
    armed = true;
    const csm_status st = csm_apply_batch(e, m, s.data(), d.data(), l.data(), del.data(), &r);
    armed = false;
    CHECK(st == CSM_ERR_OOM);
    CHECK(csm_apply_batch(e, 10, s.data(), d.data(), l.data(), nullptr, &r) == CSM_ERR_STATE);
    csm_destroy(e);
    std::printf("ok\n");
    return 0;
}
