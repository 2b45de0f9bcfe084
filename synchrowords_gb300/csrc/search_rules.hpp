// Which levels of an exact search run the dominance reductions (exact.cu).
#pragma once
#include <cmath>
#include <cstdint>

#include "synchrowords.h"

namespace sw {

// The last reduced level of a side: time of its checks, share of the distinct
// children they dropped, rows it was expanded from.
struct Reduction {
  double seconds = 0, dropped = 0;
  uint32_t parents = 0;
};

// left_out: the checks would have run but for their cost.
struct LevelRule {
  bool reduce, left_out;
};

// The checks must save kReduceGain times less than they cost to be left out, and
// a search that leaves them out switches to the bounded phase at kSwitchUnreduced
// of the projection, since each further level then enlarges what that phase
// starts from.  Sum over 18 LearnedBeam + Exact n=256 / 12 Beam + Exact n=300
// searches, ms: no rule 469 / 533; gain 0.6 333 / 640, 1 349 / 605, 1.4 with the
// earlier switch 365 / 519, 2 365 / 547 (512 with it), 4 388 / 544.
constexpr double kReduceGain = 1.4, kSwitchUnreduced = 0.5;

// Whether lists of `bytes` now stay below a quarter of the budget, where the checks
// come on again, for `levels` more lengths (each side grows ~1.7x when its turn
// comes, 1.3x a length).  A search that will get there gains nothing by larger
// lists: Beam + Exact n = 384, 12 GB, 10.6 s with its checks left out until then, 5.6 with
// them; the others of n = 320 to 384 whose bounded phase does not fit take 4.3 s
// without, 4.9 with this limit, 6.3 with their checks throughout.
inline bool lists_stay_small(double bytes, uint64_t levels, double budget) {
  return 4.0 * bytes * std::pow(1.3, (double)levels) <= budget;
}

// A level expanded from `rows` rows, `rest` seconds (0: not known) before the
// projected end of the search.  The checks pay with a word behind the bound (the
// bounded phase expands the backward list from its size at the switch) and where
// the lists press on the memory budget (past a quarter of it).  Left to this rule
// ('auto'), they run only while what they drop saves more of the rest than they
// cost (their time grows with the square of the rows), except where running out of
// memory would end the search (no bounded phase to go on in): the larger lists ran
// out up to two lengths earlier (n = 320, 100 MB).
inline LevelRule reductions_of_level(int mode, bool has_word, bool bounded_phase, bool pressure, const Reduction& last,
                                     uint64_t rows, double rest) {
  const bool wanted = mode == SW_REDUCE_ALWAYS || (mode == SW_REDUCE_AUTO && has_word);
  if (pressure || !wanted) return {pressure, false};
  if (mode == SW_REDUCE_AUTO && bounded_phase && last.parents && rest > 0) {
    const double g = (double)rows / last.parents;
    if (last.seconds * g * g > kReduceGain * last.dropped * rest) return {false, true};
  }
  return {true, false};
}

}  // namespace sw
