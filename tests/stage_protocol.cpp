// What the threads of a team do with the shared counters of a stage, between barriers, run in every
// order that the barriers allow. Built from the header the stage kernel is built from. A model stands for
// the part of the kernel named beside it; exit status 1 and a line of text when some order makes threads
// disagree: one waits at a barrier that another has left behind, or they hold different totals.
#include "../morello_b200/csrc/device_types.h"
#include <cstdio>
#include <cstring>
#include <set>
#include <string>
#include <vector>

enum { kThreads = 3 };
struct Thread {
  uint32_t pc, sweep, seen_early, seen_late, waiting, done;
};
struct World {
  StageCtl ctl;
  Thread t[kThreads];
};
// One step of a thread; `branch` 0 or 1 where the model has a choice. True: there is a second branch.
typedef bool (*Step)(World&, Thread&, uint32_t branch);

// The sweep loop: a sweep may change a cell, a barrier, and the decision to go on.
static bool sweeps(World& w, Thread& t, uint32_t branch) {
  switch (t.pc) {
    case 0: t.sweep++; t.pc = 1; return false;
    case 1:
      if (branch) w.ctl.any_changed = t.sweep;
      t.pc = 2;
      t.waiting = 1;
      return t.sweep < 4;   // the fourth changes nothing
    default:
      if (sweep_changed_a_cell(w.ctl.any_changed, t.sweep)) t.pc = 0;
      else t.done = 1;
      return false;
  }
}

// From the unordered phase to the working grids: its work items are counted, a barrier, every thread reads
// the count and takes part in solving them (and another barrier) if there are any; then items for the
// working grids are counted, a barrier, and that count is read. The small teams solve grids where they
// count them, so a stage may leave no items of the first kind.
static bool items(World& w, Thread& t, uint32_t branch) {
  switch (t.pc) {
    case 0:
      w.ctl.n_items_early += branch;
      t.pc = 1;
      t.waiting = 1;
      return true;
    case 1:
      t.seen_early = w.ctl.n_items_early;
      t.pc = t.seen_early ? 2 : 3;
      return false;
    case 2: t.pc = 3; t.waiting = 1; return false;
    case 3: w.ctl.n_items++; t.pc = 4; t.waiting = 1; return false;
    default: t.seen_late = w.ctl.n_items; t.done = 1; return false;
  }
}

static std::set<std::string> g_seen;
static long g_states = 0;

static bool explore(const World& w, Step step) {
  if (!g_seen.insert(std::string(reinterpret_cast<const char*>(&w), sizeof(w))).second) return true;
  g_states++;
  int waiting = 0, done = 0;
  for (const Thread& t : w.t) { waiting += t.waiting; done += t.done; }
  if (done == kThreads) {
    for (const Thread& t : w.t)
      if (t.seen_early != w.t[0].seen_early || t.seen_late != w.t[0].seen_late) { printf("threads hold different totals\n"); return false; }
    return true;
  }
  if (waiting == kThreads) {
    World n = w;
    for (Thread& t : n.t) t.waiting = 0;
    return explore(n, step);
  }
  if (waiting + done == kThreads) { printf("%d threads wait at a barrier that %d have left behind\n", waiting, done); return false; }
  for (int k = 0; k < kThreads; k++) {
    if (w.t[k].waiting || w.t[k].done) continue;
    for (uint32_t branch = 0; branch < 2; branch++) {
      World n = w;
      const bool two = step(n, n.t[k], branch);
      if (branch && !two) break;
      if (!explore(n, step)) return false;
    }
  }
  return true;
}

int main(int argc, char** argv) {
  World w;
  memset(&w, 0, sizeof(w));
  Step step = nullptr;
  if (argc == 2 && !strcmp(argv[1], "sweeps")) step = sweeps;
  if (argc == 2 && !strcmp(argv[1], "items")) step = items;
  if (!step) return 2;
  const bool ok = explore(w, step);
  printf("%ld states\n", g_states);
  return ok ? 0 : 1;
}
