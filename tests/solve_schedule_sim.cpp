// Steps the decisions of a one-launch solve (csrc/gcut_schedule.h) for two CTAs, one of which
// is always a whole step ahead: it has decided the next step and done that step's counting
// before the other reads the counters of the step both have finished.  The steps' outcomes are
// random.  Then grid barriers around the wrap of their arrival counts.  Prints the first
// disagreement and returns 1, else returns 0.
#include <cstdio>
#include <cstring>
#include <random>

#include "gcut_schedule.h"

using namespace gcut;

namespace {

bool same(const SolveState& a, const SolveState& b) {
  return a.step == b.step && a.cyc == b.cyc && a.n == b.n && a.pulse == b.pulse && a.pulses == b.pulses &&
         a.iters == b.iters && a.qk == b.qk && a.fk == b.fk && a.stamp == b.stamp && a.prev == b.prev &&
         a.cycles == b.cycles && a.cap == b.cap && a.hlim == b.hlim && a.rounds == b.rounds && a.err == b.err;
}

bool makes_list(int step) { return step == ST_LIST || step == ST_BFS_FIRST || step == ST_BFS; }
bool floods(int step) { return step == ST_FLOOD_FIRST || step == ST_FLOOD; }

int run(unsigned seed, bool ahead_is_cta0) {
  std::mt19937 rng(seed);
  auto pick = [&](int n) { return (int)(rng() % (unsigned)n); };
  SolvePlan plan{};
  plan.stamp0 = pick(4);
  plan.warm = pick(2);
  plan.fresh = plan.warm ? pick(2) : 1;
  plan.iters = 3;
  plan.pulses = 1 + pick(3);
  plan.max_rounds = plan.max_cycles = 1000;
  plan.cap = kFirstCap;
  SolveState ahead{};
  ahead.cap = plan.cap;
  ahead.hlim = kFirstLimit;
  ahead.stamp = plan.stamp0 + plan.warm;
  ahead.step = plan.warm ? ST_FLOOD_FIRST : ST_LIST;
  SolveState behind = ahead;
  int32_t ctl[CTL_N] = {};
  int listed = 0;       // tiles of the worklist in the making
  int last_total = 0;   // tiles queued in the step both have finished
  for (int k = 0; k < 300 && ahead.step != ST_END; ++k) {
    const int step = ahead.step;
    const bool last_pulse = step == ST_PULSE && ahead.pulse == ahead.pulses - 1;   // queues nothing
    const int total = step == ST_LIST || last_pulse || pick(3) ? 0 : 1 + pick(5);
    const int tiles = makes_list(step) && pick(3) == 0 ? 1 + pick(5) : 0;
    const int hits = floods(step) && pick(2);
    if (step == ST_BFS_FIRST) listed = 0;
    // the step counts from zero (a list that follows a relabel: from what that listed)
    const int from = floods(step) ? ctl[CTL_H0 + ahead.stamp % 3] : ctl[list_slot(ahead)];
    if ((step == ST_FLOOD_FIRST || step == ST_PULSE) ? from != 0 : makes_list(step) && from != listed)
      return std::printf("seed %u: step %d counts from %d\n", seed, step, from), 1;
    auto clear = [&](const SolveState& s) {
      if (list_slot_cleared(s) >= 0) ctl[list_slot_cleared(s)] = 0;
      if (s.step == ST_FLOOD_FIRST) ctl[CTL_H0 + (s.stamp + 1) % 3] = 0;
    };
    if (ahead_is_cta0) clear(ahead);
    if (floods(step)) ctl[CTL_H0 + ahead.stamp % 3] += hits;
    else ctl[list_slot(ahead)] += step == ST_PULSE ? total : tiles;
    listed = step == ST_PULSE ? 0 : listed + tiles;
    // the other CTA leaves the barrier of the step before only now
    if (k > 0) next_step(ctl, 1000, plan, behind, last_total);
    if (!same(ahead, behind))
      return std::printf("seed %u: one CTA at step %d with a list of %d, another at step %d with %d\n", seed,
                         ahead.step, ahead.n, behind.step, behind.n), 1;
    if (!ahead_is_cta0) clear(behind);
    next_step(ctl, 1000, plan, ahead, total);
    last_total = total;
    if (makes_list(step) && ahead.step == ST_PULSE && ahead.n != listed)
      return std::printf("seed %u: a list of %d for %d tiles\n", seed, ahead.n, listed), 1;
  }
  return 0;
}

// Barriers of `ctas` CTAs whose words start `left` uses before their arrivals reach a multiple of
// 2^32: every use is over at its last arrival only, and its sum is what the CTAs queued.
int barriers(unsigned ctas, unsigned left, unsigned seed) {
  std::mt19937 rng(seed);
  SolveState s{};
  const unsigned long long uses = (1ull << 32) / ctas - left;
  s.bar = 2 * uses;
  unsigned long long word[2] = {(uses * ctas) & 0xffffffffull, (uses * ctas) & 0xffffffffull};
  for (int k = 0; k < 40; ++k) {
    unsigned long long& w = word[s.bar & 1];
    unsigned want = 0;
    const unsigned zero = rng() % ctas;   // CTA 0 comes at any time among the others
    for (unsigned c = 0; c < ctas; ++c) {
      if (bar_full(s, ctas, w)) return std::printf("%u CTAs: over after %u\n", ctas, c), 1;
      s.push = rng() % 3 ? 0 : rng() % 1000;
      want += s.push;
      w += bar_add(s, c == zero);
      if (w & GC_BAR_ABORT) return std::printf("%u CTAs: aborted\n", ctas), 1;
    }
    if (!bar_full(s, ctas, w)) return std::printf("%u CTAs: not over\n", ctas), 1;
    const unsigned got = bar_pass(s, ctas, w);
    if (got != want) return std::printf("%u CTAs: a sum of %u, not %u\n", ctas, got, want), 1;
  }
  return 0;
}

// A barrier waits longer than a pulse can take: 2 us a sweep, all sweeps of all a CTA's tiles.
int waits() {
  for (const int iters : {1, 1000, 10000000, 2147483647})
    for (const int n : {1, 444, 445, 1 << 26})
      for (const unsigned ctas : {1u, 444u}) {
        SolveState s{};
        s.step = ST_PULSE;
        s.n = n;
        s.iters = iters;
        const double takes = 2e3 * iters * ((n + ctas - 1) / ctas);
        const unsigned long long ns = bar_wait_ns(s, ctas);
        if ((double)ns < (takes < 4e18 ? takes : 4e18))
          return std::printf("%d tiles, %u CTAs, %d sweeps: %llu ns\n", n, ctas, iters, ns), 1;
      }
  return 0;
}

// Any positive option gives positive counts in every cycle, none below the first cycle's.
int counts() {
  for (const int k : {1, 3, 17, 2147483644, 2147483645, 2147483647})
    for (int cycle = 0; cycle < 40; ++cycle) {
      const volatile int sweeps = cycle_iters(k, cycle), pulses = cycle_pulses(k, cycle);
      if (sweeps < k || pulses < k)
        return std::printf("%d: %d sweeps, %d pulses in cycle %d\n", k, sweeps, pulses, cycle), 1;
    }
  return 0;
}

}  // namespace

int main() {
  if (waits() || counts()) return 1;
  for (unsigned ctas : {1u, 2u, 3u, 128u, 443u, 444u})
    for (unsigned left = 0; left < 8; ++left)
      if (barriers(ctas, left, 8 * ctas + left)) return 1;
  for (unsigned seed = 0; seed < 20000; ++seed)
    for (int cta0 = 0; cta0 < 2; ++cta0)
      if (run(seed, cta0)) return 1;
  return 0;
}
