// held_run.h -- the order of the steps, questions and timings of a run with
// images held in place.  Host code only; the calls it orders are capi.cu's.
#pragma once

namespace lbmpsm {

// When a run asks whether the particle table has settled: before its second to
// fourth step (a table that particles have just moved over settles with the
// second or third map), while enough steps are left to be worth the wait.
struct SettleQuestions {
  static constexpr int MAX = 3;
  int asked = 0;
  bool settled = false;
  bool due(int done, int left, int min_left = 4) const {
    return !settled && done >= 1 && asked < MAX && left >= min_left;
  }
};

// One call of a group: nsteps steps, with tune (nsteps >= 8) the two plans timed
// on the way.  Ops:
//   int ask(bool& settled)   whether every member's table has settled (waits)
//   int step(bool map)       one step, with the maps or without
//   int plan(int which)      the steps that follow take this plan (drops graphs)
//   int ready(bool map)      prepares what steps of the plan need for their launch
//   int start(), stop(int which)   around a plan's timed steps
//   int choose()             takes the faster plan
// Each returns 0 or an error, which ends the run.
//
// Both plans are timed on steps of one kind: the questions come before the
// first timed step and after the last, and nothing is captured between start
// and stop.
template <class Ops>
int run_group_steps(Ops& o, int nsteps, bool may_ask, bool tune) {
  SettleQuestions q;
  int done = 0, left = nsteps;
  auto ask = [&]() -> int {
    if (!may_ask || !q.due(done, left)) return 0;
    ++q.asked;
    return o.ask(q.settled);
  };
  auto step = [&]() -> int {
    const int rc = o.step(!q.settled);
    ++done;
    --left;
    return rc;
  };
  int rc = 0;
  if (tune) {
    for (int which = 1; which >= 0; --which) {
      if ((rc = o.plan(which))) return rc;
      for (int k = 0; k < 2; ++k) {
        if (which == 1 && (rc = ask())) return rc;
        if ((rc = step())) return rc;
      }
      if (which == 1 && (rc = ask())) return rc;
      if ((rc = o.ready(!q.settled))) return rc;
      if ((rc = o.start())) return rc;
      for (int k = 0; k < 2; ++k)
        if ((rc = step())) return rc;
      if ((rc = o.stop(which))) return rc;
    }
    if ((rc = o.choose())) return rc;
  }
  while (left > 0) {
    if ((rc = ask())) return rc;
    if ((rc = step())) return rc;
  }
  return 0;
}

}  // namespace lbmpsm
