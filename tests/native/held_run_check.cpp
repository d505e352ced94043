// Runs run_group_steps on a model of a group whose tables settle with a given
// map (0: never) and prints what breaks its rules (nothing: "ok").
#include <cstdio>
#include <cstdlib>

#include "held_run.h"

struct Model {
  int settles;         // the map that leaves the table as it is (and all after it)
  int fail_at = -1;    // the call that returns an error
  int calls = 0, steps = 0, maps = 0, asks = 0, which = -1;
  bool timing = false, answered = false;
  bool captured[2][2]{};      // [map][parity], of the plan
  int untimed = 0, timed[2]{0, 0}, kind[2]{-1, -1}, chosen = 0;
  const char* bad = nullptr;
  int call() { return calls++ == fail_at ? 7 : 0; }
  void check(bool ok, const char* what) {
    if (!ok && !bad) bad = what;
  }
  int ask(bool& settled) {
    check(!timing, "a question among the timed steps");
    check(steps > 0, "a question before the first step");
    ++asks;
    settled = settles > 0 && maps >= settles;
    answered = settled;
    return call();
  }
  int step(bool map) {
    check(map || answered, "a step without the map on a table not known to have settled");
    bool& c = captured[map][steps & 1];
    check(c || !timing, "a capture among the timed steps");
    c = true;
    ++steps;
    maps += map;
    if (timing) {
      ++timed[which];
      check(kind[which] < 0 || kind[which] == map, "timed steps of two kinds in one plan");
      kind[which] = map;
    } else {
      ++untimed;
    }
    return call();
  }
  int plan(int w) {
    check(!timing, "a change of plan among the timed steps");
    which = w;
    untimed = 0;
    for (auto& a : captured) a[0] = a[1] = false;
    return call();
  }
  int ready(bool map) {
    check(!timing, "a capture among the timed steps");
    captured[map][0] = captured[map][1] = true;
    return call();
  }
  int start() {
    check(untimed >= 2, "a plan timed without two steps before");
    timing = true;
    return call();
  }
  int stop(int w) {
    check(w == which, "the wrong plan");
    timing = false;
    return call();
  }
  int choose() {
    ++chosen;
    return call();
  }
};

int main() {
  long runs = 0;
  for (int settles = 0; settles <= 6; ++settles)
    for (int n = 0; n <= 20; ++n)
      for (int tune = 0; tune <= (n >= 8 ? 1 : 0); ++tune)
        for (int may_ask = 0; may_ask <= 1; ++may_ask) {
          Model m{settles};
          const int rc = lbmpsm::run_group_steps(m, n, may_ask, tune);
          m.check(rc == 0, "an error");
          m.check(m.steps == n, "not nsteps steps");
          m.check(m.asks <= (may_ask ? 3 : 0), "too many questions");
          m.check(m.chosen == tune, "the choice");
          if (tune) {
            m.check(m.timed[0] == 2 && m.timed[1] == 2, "two timed steps a plan");
            m.check(m.kind[0] == m.kind[1], "the plans timed on steps of two kinds");
            // a table that settles with the first or second map is timed without maps
            m.check(!may_ask || settles < 1 || settles > 2 || m.kind[0] == 0, "timed with maps");
          }
          // the maps end with the third question at the latest
          if (may_ask && settles >= 1 && settles <= 3 && n >= 8 && !tune) m.check(m.maps <= 3, "maps of a settled table");
          if (m.bad) {
            std::printf("settles %d steps %d tune %d ask %d: %s\n", settles, n, tune, may_ask, m.bad);
            return 1;
          }
          // an error of any call ends the run there
          for (int k = 0; k < m.calls; ++k) {
            Model e{settles, k};
            if (lbmpsm::run_group_steps(e, n, may_ask, tune) != 7 || e.calls != k + 1) {
              std::printf("error of call %d not returned\n", k);
              return 1;
            }
          }
          ++runs;
        }
  std::printf("ok %ld\n", runs);
}
