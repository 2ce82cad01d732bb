// sdf_steps.h — how the CTAs of k_sdf_levels (sdf.cu) go from one step to the next.
//
// Which CTAs take part is settled at every barrier and nowhere else: a CTA draws a ticket when it
// starts, and the release word of a step says how many tickets the next step is divided among.
// Ticket 0 opens the first step after a short wait for the others; a CTA that starts later than
// that waits for the next release, and one that starts after the last step returns. So the wait is
// only ever for CTAs that are running, whatever else holds the SMs (a render on another stream, a
// process limited to a part of them) and however many of the launch's CTAs fit. What a step does
// (the levels that still have cells) is part of the same word: no CTA derives it from counters that
// others are changing.
//
// M: relaxed loads and stores, an atomic add that returns the old value, an atomic count from 0 to
// n - 1 and round again that does too, a fence that orders all earlier accesses of the CTA before all
// later ones, and a pause. The kernel's are in sdf.cu.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define WX_STEPS __device__ __forceinline__
#else
#define WX_STEPS inline
#endif

namespace wxk {

struct SdfCtl {
    // Cleared before each launch.
    uint32_t started;  // tickets drawn
    uint32_t arrived;  // CTAs at the barrier of the current step
    uint32_t release;  // word of the last finished step (steps_word), 0 before the first step is open
    uint32_t unused;
    // Kept over the launches of a build.
    uint32_t error;    // a wait hit its bound
    uint32_t n_ovf;    // overflow entries
    uint32_t last[3];  // last step of N5, N4, leaves
    uint32_t unused2;
    unsigned long long left[3];   // cells of N5, N4 and leaves without a distance
    unsigned long long inactive;  // leaf cells without a distance at the start
};

// A finished step k (12 bits), the CTAs of the next one (16 bits) and the levels without open cells (bit each of N5,
// N4, leaves).
constexpr uint32_t kStepsMaxCtas = 65535u, kStepsAllDone = 7u;
WX_STEPS uint32_t steps_word(uint32_t k, uint32_t ctas, uint32_t done) { return (k << 19) | (ctas << 3) | done; }
WX_STEPS uint32_t steps_k(uint32_t w) { return w >> 19; }
WX_STEPS uint32_t steps_ctas(uint32_t w) { return (w >> 3) & kStepsMaxCtas; }
WX_STEPS uint32_t steps_done(uint32_t w) { return w & 7u; }

// Polls that ticket 0 waits for the launch's other CTAs (8 us; on an idle chip they start within 2 us).
constexpr uint32_t kStepsStartPolls = 32u;

template <class M>
WX_STEPS uint32_t steps_publish(M m, SdfCtl *c, uint32_t k) {
    // All loads in flight together: every other CTA waits for this one.
    const uint32_t ctas = m.load(&c->started), error = m.load(&c->error);
    const unsigned long long n5 = m.load(&c->left[0]), n4 = m.load(&c->left[1]), n3 = m.load(&c->left[2]);
    const uint32_t done = (n5 ? 0u : 1u) | (n4 ? 0u : 2u) | (n3 ? 0u : 4u);
    const uint32_t w = steps_word(k, ctas, error ? kStepsAllDone : done);
    m.store(&c->release, w);
    return w;
}

// The word of step k, or of a later one, that has a place for this ticket or ends the launch (whose last step is k1).
// After `limit` polls, or once another CTA has met its limit: the error flag, and a word with nothing left to do.
template <class M>
WX_STEPS uint32_t steps_wait(M m, SdfCtl *c, uint32_t ticket, uint32_t k, uint32_t k1, uint32_t limit) {
    for (uint32_t polls = 1;; polls++) {
        const uint32_t w = m.load(&c->release);
        if (w != 0u && steps_k(w) >= k &&
            (ticket < steps_ctas(w) || steps_done(w) == kStepsAllDone || steps_k(w) >= k1)) {
            m.fence();
            return w;
        }
        if (polls >= limit || m.load(&c->error) != 0u) {
            m.store(&c->error, 1u);
            return steps_word(k, 0u, kStepsAllDone);
        }
        m.pause();
    }
}

// Once per CTA, before its first step: its ticket, and the word whose next step is its first.
template <class M>
WX_STEPS uint32_t steps_enter(M m, SdfCtl *c, uint32_t ctas, uint32_t k0, uint32_t k1, uint32_t limit, uint32_t *ticket) {
    *ticket = m.add(&c->started, 1u);
    if (*ticket != 0u) return steps_wait(m, c, *ticket, k0 - 1u, k1, limit);
    for (uint32_t polls = 0; polls < kStepsStartPolls && m.load(&c->started) < ctas; polls++) m.pause();
    return steps_publish(m, c, k0 - 1u);
}

// At the end of the step after word w; the CTA's part of it is written. Returns the word of that step.
template <class M>
WX_STEPS uint32_t steps_next(M m, SdfCtl *c, uint32_t ticket, uint32_t w, uint32_t k1, uint32_t limit) {
    const uint32_t k = steps_k(w) + 1u;
    m.fence();
    if (m.count(&c->arrived, steps_ctas(w)) != steps_ctas(w) - 1u) return steps_wait(m, c, ticket, k, k1, limit);
    m.fence();  // before the release: the count is back at 0, and the other CTAs' writes are before this one's release
    for (uint32_t l = 0; l < 3u; l++)
        if (!((steps_done(w) >> l) & 1u)) c->last[l] = k;
    return steps_publish(m, c, k);
}

}  // namespace wxk
