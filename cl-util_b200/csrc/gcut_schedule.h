// Decisions of a solve: which step follows which, on what schedule, and where the steps of the
// one-launch solve (k_solve) count what they queue.  No CUDA types, and it compiles as plain
// C++ too, so that a host program can take the same decisions step by step.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GC_HD __device__ __host__ __forceinline__
#else
#define GC_HD inline
#endif

#define GC_HINF 0x3fffffff

namespace gcut {

// Device-side loop control words.  In the host-driven loops the last CTA of every frontier
// round advances the round parity; k_solve keeps its loop state in shared memory and uses the
// rotating counters (CTL_Q0.., CTL_F0.., CTL_H0..) and the totals.
enum CtlSlot {
  CTL_RND = 0,        // frontier round number (its parity selects the mark buffer)
  CTL_DONE = 1,       // CTAs finished in the current round
  CTL_LASTCNT = 2,    // tiles the last finished round queued for the next
  CTL_ROUNDS = 3,     // rounds of the current frontier loop
  CTL_BFS_TOTAL = 4,  // BFS rounds of the solve
  CTL_FLOOD_TOTAL = 5,
  CTL_CYCLES = 6,     // global-relabel cycles of the solve
  CTL_ERR = 7,        // 1: round cap, 2: cycle cap, 3: copy wait gave up, 4: self-check,
                      // 5: grid-barrier wait gave up
  CTL_MAXROUNDS = 8,
  CTL_PULSE = 10,     // discharge launches since the last list rebuild (parity = worklist)
  CTL_DDONE = 11,     // CTAs finished in the current discharge launch
  CTL_BAD = 12,       // first out-of-range worklist value seen by a self-check
  CTL_BADWHERE = 13,  // 1: worklist append, 2: worklist length, 3: list length, 4: image id
                      // (or tile) of the selection, 5: frontier append, 6: frontier length,
                      // 9: selection size
  CTL_NCHECK = 15,    // flood checks run (k_flood_check launches)
  CTL_NACT = 16,      // active-list rebuilds run (k_active_list launches)
  CTL_LEFT = 17,      // images still running after the last flood check
  CTL_SCANERR = 18,   // the scan state's error word, as the last active list saw it
  // k_solve's counters, three of each: a step reads one (filled by the step before), adds to
  // the next and clears the third, so one grid barrier per step orders all three uses (the
  // worklists': list_slot)
  CTL_Q0 = 20,        // worklist lengths
  CTL_F0 = 24,        // frontier lengths
  CTL_H0 = 28,        // images whose flood reached a sink
  CTL_N = 64          // the control words fill 256 bytes; the per-image sums follow them
};

// The schedule of a solve: pulses and sweeps of cycle `cycle` (0, 1, ...) from the handle's
// options, and the relabel's distance cap (its first value, and the next after `cap`).
//
// A cycle costs a flood and a relabel over the images left (60 us at 2048^2) besides its
// pulses (10 us each on a few hundred tiles).  Most solves end after one or two cycles, which
// the options' own schedule suits; the excess left after that has to travel far, and then more
// work between relabels pays: three more sweeps from the second cycle, twice the pulses with
// each from the third.  Mean over 12 seeds against the fixed schedule 3 x 2 (and its worst
// seed), one B200: 2048^2 1740 -> 515 us (13133 -> 3216), 512^2 424 -> 241, 803x607 under the
// lamda rule 690 -> 317, 4096^2 image 1108 -> 974.
GC_HD int cycle_pulses(int pulses, int cycle) {
  const int most = pulses > 16 ? pulses : 16;
  const int shift = cycle < 2 ? 0 : cycle - 1 < 4 ? cycle - 1 : 4;
  const long long p = (long long)pulses << shift;
  return p < most ? (int)p : most;
}
GC_HD int cycle_iters(int iters, int cycle) {
  return cycle == 0 || iters > 0x7fffffff - 3 ? iters : iters + 3;   // (any positive count is an option)
}
// Active heights before the first relabel, whose trivial labels (0 at sinks, 1 elsewhere) say
// little: below 4, excess far from a sink stops rising after three sweeps instead of keeping
// its warps busy.  (3: more cycles; unlimited: 512^2 3 %, 64 grids 4 % slower.)
constexpr int kFirstLimit = 4;
// The first relabel reaches 8 pixels around the sinks: what is further out gets its distances
// with a later cap, if it is still active then.  (Mean us over 12 seeds, caps 4 / 8 / 10: 64 grids
// 5025 / 4613 / 4844, 1920x1080 models 290 / 264 / 272, 4096^2 image 727 / 686 / 682; over 9 seeds,
// caps 16 / 8: models 287 / 273, 12 sessions 516 / 491, strokes at 4096^2 145 / 140.)
constexpr int kFirstCap = 8;
constexpr int kLastCap = 1 << 12;   // above it: exact distances
GC_HD int next_cap(int cap) { return cap >= kLastCap ? GC_HINF : cap * 2; }
// initial_relabel: the relabel before the first pulses is exact, and the caps start after it.
GC_HD int first_cap(int initial_relabel) { return initial_relabel ? GC_HINF : kFirstCap; }
GC_HD int cap_after(int cap, bool initial) { return initial && cap >= GC_HINF ? kFirstCap : next_cap(cap); }

// What the decisions of a one-launch solve depend on.
struct SolvePlan {
  int stamp0;               // every stamp in img_hit is at most this; the floods take the next ones
  int warm, fresh;          // some selected image continues from a flow / is freshly uploaded
  int iters, pulses;        // sweeps per discharge, discharges per cycle
  int max_rounds, max_cycles;
  int cap;                  // distance cap of the first relabel (first_cap)
};

// The solve's loop state, one copy per CTA in shared memory, written by thread 0 only (inside
// solve_barrier): the same in every CTA, because it follows from the same counters.  Kept out
// of registers: what a step spills is reloaded from L2, since the barriers' fences empty L1.
enum SolveStep { ST_LIST, ST_PULSE, ST_FLOOD_FIRST, ST_FLOOD, ST_BFS_FIRST, ST_BFS, ST_END };
struct SolveState {
  int step;
  int cyc;                  // 0 before the first pulses (warm images' flood, first list)
  int n;                    // tiles of the step's list
  int pulse, pulses, iters; // of the cycle
  int qk, fk;               // worklists and frontier steps so far (counter slots mod 3)
  int stamp, prev;          // the flood's stamp, the one before it (0: none)
  int cycles, cap, hlim;    // finished cycles; the next relabel's cap, the last one's limit
  int rounds;               // of the flood or relabel that runs
  int nf, nb, np;           // flood rounds, relabel rounds, pulses of the solve
  int err;
  int push;                 // tiles this CTA has queued since the last barrier
  unsigned long long bar;   // barriers passed
  unsigned last[2];         // sum halves that the barrier words' last uses left
};

// A grid barrier word: the low half counts arrivals, bits 32-62 hold a sum over the CTAs (tiles
// queued since the last barrier), bit 63 ends the solve.  Barriers alternate between two words,
// and no CTA reaches a word's next use before all have left this one, so a use is over exactly
// when the low half stands at the arrivals of all uses so far, modulo 2^32: no number of
// barriers is too many.  When the low half wraps, its carry adds one to the sum of that use.
constexpr unsigned long long GC_BAR_ABORT = 1ull << 63;
GC_HD unsigned long long bar_arrivals(const SolveState& s, unsigned ctas) {   // before this use
  return (s.bar >> 1) * ctas;
}
// What a CTA adds; CTA 0 takes out what the word's last use left in the sum half, which so never
// falls below zero.
GC_HD unsigned long long bar_add(const SolveState& s, bool cta0) {
  const unsigned long long add = ((unsigned long long)(unsigned)s.push << 32) + 1ull;
  return cta0 ? add - ((unsigned long long)s.last[s.bar & 1] << 32) : add;
}
GC_HD bool bar_full(const SolveState& s, unsigned ctas, unsigned long long word) {
  return (unsigned)word == (unsigned)(bar_arrivals(s, ctas) + ctas);
}
// How long a CTA waits for the others, in ns: 5 s, far beyond any step's passes over the largest
// pool, and 4 us a sweep of the tiles a CTA may have in a pulse (a sweep takes 0.5 to 2 us; how
// many there are is the caller's option, without a limit).
GC_HD unsigned long long bar_wait_ns(const SolveState& s, unsigned ctas) {
  if (s.step != ST_PULSE) return 5000000000ull;
  const unsigned long long sweeps = ((unsigned)s.n / ctas + 1ull) * (unsigned)s.iters;
  const unsigned long long most = 1ull << 50;
  return 5000000000ull + 4000ull * (sweeps < most ? sweeps : most);
}
// The sum of a use that is over; passes the barrier.
GC_HD unsigned bar_pass(SolveState& s, unsigned ctas, unsigned long long word) {
  const unsigned long long before = bar_arrivals(s, ctas);
  const unsigned sum = (unsigned)(word >> 32) & 0x7fffffffu;
  s.push = 0;
  s.last[s.bar & 1] = sum;
  ++s.bar;
  return sum - (unsigned)(((before + ctas) >> 32) - (before >> 32));
}

// Worklist counter that a step adds the tiles it lists to (a pulse: the next worklist's), and
// the one that it clears for a later step (-1: none).  next_step reads a list's or relabel's
// counter after the barrier, when other CTAs may be in the next step already: so a relabel that
// starts over because it listed nothing counts in the next slot, and a slot is cleared a step
// before it is counted in and not in the step after its reading.
GC_HD int list_slot(const SolveState& s) { return CTL_Q0 + (s.step == ST_PULSE ? s.qk + 1 : s.qk) % 3; }
GC_HD int list_slot_cleared(const SolveState& s) {
  return s.step == ST_PULSE ? CTL_Q0 + (s.qk + 2) % 3 : s.step == ST_BFS_FIRST ? CTL_Q0 + (s.qk + 1) % 3 : -1;
}

GC_HD void begin_cycle(const SolvePlan& A, SolveState& s, int list) {
  ++s.cyc;
  s.n = list;
  s.pulse = 0;
  s.pulses = cycle_pulses(A.pulses, s.cycles);
  s.iters = cycle_iters(A.iters, s.cycles);
  s.step = ST_PULSE;
}

// The step after `s.step`, which the whole grid has finished; total: tiles queued in it; ctl:
// the control words; nt: tiles of the pool.
GC_HD void next_step(const volatile int32_t* ctl, int nt, const SolvePlan& A, SolveState& s, int total) {
  int list = -1;   // >= 0: a cycle begins with a worklist of this length
  s.n = total;
  switch (s.step) {
    case ST_LIST:
      list = ctl[list_slot(s)];
      break;
    case ST_PULSE:
      ++s.qk;
      ++s.np;
      if (++s.pulse < s.pulses && total > 0) break;
      s.step = ST_FLOOD_FIRST;
      s.prev = s.stamp == A.stamp0 ? 0 : s.stamp;
      ++s.stamp;
      break;
    case ST_FLOOD_FIRST:
    case ST_FLOOD: {
      ++s.fk;
      ++s.nf;
      ++s.rounds;
      if (total > 0) {
        s.step = ST_FLOOD;
        if (s.rounds >= A.max_rounds) s.err = 1;
        break;
      }
      const int left = ctl[CTL_H0 + s.stamp % 3];   // images that met a sink
      if (s.cyc > 0) ++s.cycles;
      s.rounds = 0;
      s.step = left > 0 ? ST_BFS_FIRST : s.cyc == 0 && A.fresh ? ST_LIST : ST_END;
      break;
    }
    case ST_BFS_FIRST:
    case ST_BFS:
      ++s.fk;
      ++s.nb;
      ++s.rounds;
      if (total > 0) {
        s.step = ST_BFS;
        if (s.rounds >= A.max_rounds) s.err = 1;
        break;
      }
      s.rounds = 0;
      list = ctl[list_slot(s)];
      if (list == 0 && s.cap < GC_HINF) {   // no excess within the cap of a sink: further out
        s.cap = next_cap(s.cap);
        ++s.qk;   // this list's counter may still be read; the list is empty
        s.step = ST_BFS_FIRST;
        list = -1;
        break;
      }
      s.hlim = s.cap < GC_HINF ? s.cap + 1 : GC_HINF;
      s.cap = cap_after(s.cap, s.cyc == 0 && A.cap >= GC_HINF);   // further out with every cycle
      if (s.cyc == 0 && A.fresh) {
        s.step = ST_LIST;
        list = -1;
      }
      break;
  }
  if (list >= 0) {
    if (list == 0 && s.step != ST_LIST) {
      s.step = ST_END;
    } else if (s.cycles >= A.max_cycles) {
      s.err = 2;
    } else {
      begin_cycle(A, s, list);
      if (list == 0) {   // no fresh tile is near a sink: straight to the flood
        s.step = ST_FLOOD_FIRST;
        s.prev = s.stamp == A.stamp0 ? 0 : s.stamp;
        ++s.stamp;
      }
    }
  }
  if (s.n < 0 || s.n > nt) s.err = 4;   // self-check: a list holds each tile at most once
  if (s.err) s.step = ST_END;
}

}  // namespace gcut
