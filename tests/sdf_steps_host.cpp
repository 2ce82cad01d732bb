// The step control of the GPU SDF build (csrc/sdf_steps.h) with a thread for each CTA.
//
// Arguments: ctas k0 k1 limit, then the last step of each of the three levels (cells of distance k0..last, a
// few of each; k0 - 1: none), then for each CTA when it starts: -1 at once, l once level l has no cell left,
// 3 once none is left in any level, 4 after every other CTA has returned. Prints "error" if a wait met its limit, else
// the last step of each level, and fails if a cell was not looked at exactly once in each step of its level.
#include <sched.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "sdf_steps.h"

namespace {
struct Mem {
    template <class T>
    T add(T *p, T v) const { return __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
    uint32_t count(uint32_t *p, uint32_t n) const {
        uint32_t v = load(p);
        while (!__atomic_compare_exchange_n(p, &v, v + 1u < n ? v + 1u : 0u, true, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {
        }
        return v;
    }
    template <class T>
    T load(const T *p) const { return __atomic_load_n(p, __ATOMIC_RELAXED); }
    void store(uint32_t *p, uint32_t v) const { __atomic_store_n(p, v, __ATOMIC_RELAXED); }
    void fence() const { __atomic_thread_fence(__ATOMIC_SEQ_CST); }
    void pause() const { sched_yield(); }
};
}  // namespace

int main(int argc, char **argv) {
    auto arg = [&](int i) { return i < argc ? std::atoi(argv[i]) : -1; };
    const uint32_t ctas = arg(1), k0 = arg(2), k1 = arg(3), limit = arg(4);
    const Mem m;
    wxk::SdfCtl c{};
    std::vector<uint32_t> dist[3], seen[3];
    const uint32_t per = 3 * ctas + 1;  // cells of one distance
    for (int l = 0; l < 3; l++) {
        for (uint32_t k = k0; (int)k <= arg(5 + l); k++) dist[l].insert(dist[l].end(), per, k);
        seen[l].assign(dist[l].size() * (k1 + 1), 0);
        c.left[l] = dist[l].size();
    }
    std::atomic<uint32_t> returned{0};
    auto cta = [&](uint32_t j) {
        const int when = arg(8 + (int)j);
        auto wait = [&](auto ready) {
            while (!ready()) sched_yield();
        };
        auto done = [&](int l) { return m.load(&c.left[l]) == 0ull || m.load(&c.error); };
        if (when >= 0 && when < 3) wait([&] { return done(when); });
        if (when == 3) wait([&] { return done(0) && done(1) && done(2); });
        if (when == 4) wait([&] { return returned == ctas - 1u; });
        uint32_t ticket;
        uint32_t w = wxk::steps_enter(m, &c, ctas, k0, k1, limit, &ticket);
        while (wxk::steps_done(w) != wxk::kStepsAllDone && wxk::steps_k(w) < k1) {
            const uint32_t k = wxk::steps_k(w) + 1u;
            for (int l = 0; l < 3; l++) {
                if ((wxk::steps_done(w) >> l) & 1u) continue;
                unsigned long long found = 0;
                for (size_t i = ticket; i < dist[l].size(); i += wxk::steps_ctas(w)) {
                    seen[l][i * (k1 + 1) + k]++;  // a cell has one owner in a step: threads never share an element at a time
                    found += dist[l][i] == k;
                }
                if (found) m.add(&c.left[l], 0ull - found);
            }
            w = wxk::steps_next(m, &c, ticket, w, k1, limit);
        }
        returned++;
    };
    std::vector<std::thread> th;
    for (uint32_t j = 0; j < ctas; j++) th.emplace_back(cta, j);
    for (auto &t : th) t.join();
    if (c.error) {
        std::puts("error");
        return 0;
    }
    int bad = 0;
    for (int l = 0; l < 3; l++) {
        const uint32_t last = dist[l].empty() ? k0 - 1u : std::min(dist[l].back(), k1);
        for (size_t i = 0; i < dist[l].size(); i++)
            for (uint32_t k = 0; k <= k1; k++) bad += seen[l][i * (k1 + 1) + k] != (k >= k0 && k <= last ? 1u : 0u);
    }
    std::printf("%u %u %u\n", c.last[0], c.last[1], c.last[2]);
    if (bad) std::printf("%d cells not looked at once a step\n", bad);
    return bad != 0;
}
