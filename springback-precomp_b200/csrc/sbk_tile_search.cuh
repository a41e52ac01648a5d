// The line search of the tile kernel's local iteration: what the reference does
// when the full Newton step of a definite K_aa is refused (line_search and
// search_norm, IncompatibleModes.cpp:359-456), as a state per element instead
// of a call. A trial is a pass of the tile's next round at alpha + t dir;
// search_after takes its outcome, and either accepts it, sets the next trial,
// or hands the element on: where no step is found, and where K_aa is
// indefinite (the shifted direction, Levenberg-Marquardt), the single kernel
// starts the element again.
//
// One lane runs it over the element's record: a few comparisons a trial. Handed
// to the single kernel as well, the some hundred elements of 80,000 that
// search held the GPU for 3.5 ms at the end of an evaluation.
#pragma once

#include "sbk_element_math.cuh"
#include "sbk_tile.h"

namespace sbk {

struct TileElement;

enum TileStage {
  kStageNewton,   // the full Newton step
  kStageShrink,   // it halved while it is not evaluated
  kStageSection,  // the search on the directional residual
  kStageReturn,   // its last evaluated point again
  kStageNorm,     // search_norm
  kStageBest      // its best point again
};

template <class E>
__device__ __forceinline__ int search_trial(E& e, int stage, double t) {
  for (int i = 0; i < 9; ++i) e.at[i] = e.alpha[i] + t * e.dir[i];
  e.stage = stage;
  return 0;
}

template <class E>
__device__ __forceinline__ double search_slope(const E& e, const double* r) {
  double v = 0.0;
  for (int i = 0; i < 9; ++i) v += e.dir[i] * r[i];
  return v;
}

// After a trial of element e: evaluated, with the residual norm `full`,
// within the tolerance (`met`) or reducing it enough (`reduced`). Returns 0
// with the next trial set, 1 to accept this one, 2 to hand the element on.
template <class E>
__device__ __noinline__ int search_after(E& e, TileSearch& s, bool evaluated, double full, bool met, bool reduced) {
  const double infinity = __longlong_as_double(0x7ff0000000000000LL);
  switch (e.stage) {
    case kStageNewton:
      s.reach = 1.0;
      s.halvings = 0;
      // fall through: the line search's first trial
    case kStageShrink: {
      if (!evaluated) {
        if (s.halvings < kMaxLineSearch) {
          ++s.halvings;
          s.reach *= 0.5;
          return search_trial(e, kStageShrink, s.reach);
        }
        return 2;
      }
      if (reduced || met) return 1;
      const double phi0 = search_slope(e, e.r0), phi1 = search_slope(e, e.r);
      if (!(phi0 < 0.0) || !(phi1 > 0.0) || !isfinite(phi1)) {
        s.best_step = 0.0;
        s.best = e.res;
        s.last_is_best = 0;
        s.count = 0;
        s.step = 0.5 * s.reach;
        return search_trial(e, kStageNorm, s.step);
      }
      s.phi0 = phi0;
      s.s0 = 0.0, s.f0 = phi0, s.s1 = s.reach, s.f1 = phi1;
      s.side = 0;
      s.count = 0;
      const double width = s.s1 - s.s0;
      s.step = fmin(fmax((s.s0 * s.f1 - s.s1 * s.f0) / (s.f1 - s.f0), s.s0 + 0.1 * width), s.s1 - 0.1 * width);
      return search_trial(e, kStageSection, s.step);
    }
    case kStageSection: {
      const double f = evaluated ? search_slope(e, e.r) : infinity;
      if (evaluated && fabs(f) <= kLineSearchRatio * fabs(s.phi0)) return 1;
      if (!evaluated || f > 0.0) {
        s.s1 = s.step;
        s.f1 = evaluated ? f : 0.5 * s.f1;
        if (s.side == 1) s.f0 *= 0.5;
        s.side = 1;
      } else {
        s.s0 = s.step;
        s.f0 = f;
        if (s.side == -1) s.f1 *= 0.5;
        s.side = -1;
      }
      if (++s.count < kMaxLineSearch) {
        const double width = s.s1 - s.s0;
        s.step = fmin(fmax((s.s0 * s.f1 - s.s1 * s.f0) / (s.f1 - s.f0), s.s0 + 0.1 * width), s.s1 - 0.1 * width);
        return search_trial(e, kStageSection, s.step);
      }
      if (evaluated) return 1;
      return s.s0 == 0.0 ? 2 : search_trial(e, kStageReturn, s.s0);
    }
    case kStageNorm: {
      bool stop = false;
      s.last_is_best = 0;
      if (evaluated) {
        if (full < s.best) {
          s.last_is_best = 1;
          s.best = full;
          s.best_step = s.step;
        }
        stop = reduced;
      }
      if (!stop && ++s.count < kMaxLineSearch) {
        s.step *= 0.5;
        return search_trial(e, kStageNorm, s.step);
      }
      if (s.best_step == 0.0) return 2;
      return s.last_is_best ? 1 : search_trial(e, kStageBest, s.best_step);
    }
    default:  // kStageReturn, kStageBest
      // A point that evaluated before can fail now: its return starts from
      // the closest point of the trial in between. The sums are then another
      // trial's, so the element goes on as after any search that fails.
      return evaluated ? 1 : 2;
  }
}

}  // namespace sbk
