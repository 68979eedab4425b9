// Every schedule of the column pipeline's copies and waits (PipeRing in ptx_pipering.h,
// cols_sweep_pipe in ptx_passes.cuh), the barriers modelled: a copy completes at any time after
// its issue, in any order, and with it a phase of its barrier; a wait for parity P holds while
// the barrier's open phase has parity P.  A group that has waited for its tile works on it and
// then issues the copy of the tile that takes the buffer next.  Prints, per tile count: the
// states reached, the waits that returned before their tile had come, the copies issued into a
// buffer or on a barrier still in use, the states from which nothing goes on before the end, and
// those in which both groups wait and left_open names other copies than the issued ones they
// have not waited for, or a wait for one of these would not hold just until it is done.
#include <cstdio>
#include <set>
#include <tuple>
#include <vector>

#include "ptx_pipering.h"

using Ring = ptx::PipeRing;

struct State {
  int next[2];            // the tile each group waits for or works on
  bool busy[2];           // it has passed the wait
  unsigned issued, done;  // copies, by tile
  bool operator<(const State& o) const { return key() < o.key(); }
  std::tuple<int, int, bool, bool, unsigned, unsigned> key() const {
    return {next[0], next[1], busy[0], busy[1], issued, done};
  }
  bool has(unsigned set, int i) const { return set >> i & 1; }
  bool waited(int i) const { return next[Ring::group(i)] > i || (next[Ring::group(i)] == i && busy[Ring::group(i)]); }
  bool finished(int i) const { return next[Ring::group(i)] > i; }
  int phases(int bar) const {  // completed phases of a barrier
    int count = 0;
    for (int i = 0; i < 32; ++i) count += Ring::barrier(i) == bar && has(done, i);
    return count;
  }
};
static_assert(Ring::kGroups == 2, "State holds two groups");

int main() {
  for (int n = 1; n <= 20; ++n) {
    State first{{0, 1}, {false, false}, 0, 0};
    for (int i = 0; i < Ring::kBufs && i < n; ++i) first.issued |= 1u << i;
    std::set<State> seen{first};
    std::vector<State> todo{first};
    int early = 0, in_use = 0, stuck = 0, wrong_open = 0;
    while (!todo.empty()) {
      const State a = todo.back();
      todo.pop_back();
      bool moved = false;
      for (int i = 0; i < n && !a.busy[0] && !a.busy[1]; ++i) {
        const bool open = a.has(a.issued, i) && !a.waited(i);
        const bool holds = (a.phases(Ring::barrier(i)) & 1u) == Ring::parity(i);
        wrong_open += Ring::left_open(i, a.next) != open || (open && holds == a.has(a.done, i));
      }
      auto go = [&](const State& b) {
        moved = true;
        if (seen.insert(b).second) todo.push_back(b);
      };
      for (int i = 0; i < n; ++i) {  // a copy arrives
        if (!a.has(a.issued, i) || a.has(a.done, i)) continue;
        State b = a;
        b.done |= 1u << i;
        go(b);
      }
      for (int g = 0; g < 2; ++g) {
        const int i = a.next[g];
        if (i >= n) continue;
        State b = a;
        if (!a.busy[g]) {
          if ((a.phases(Ring::barrier(i)) & 1u) == Ring::parity(i)) continue;  // the wait holds
          early += !a.has(a.done, i);
          b.busy[g] = true;
        } else {
          b.busy[g] = false;
          b.next[g] = i + Ring::kGroups;
          const int j = i + Ring::kBufs;
          if (j < n) {
            b.issued |= 1u << j;
            for (int k = 0; k < j; ++k) {
              const bool same_barrier = Ring::barrier(k) == Ring::barrier(j), same_buffer = Ring::buffer(k) == Ring::buffer(j);
              in_use += (same_barrier && !(a.has(a.done, k) && a.waited(k))) || (same_buffer && !b.finished(k));
            }
          }
        }
        go(b);
      }
      stuck += !moved && !(a.next[0] >= n && a.next[1] >= n && a.done == (1u << n) - 1);
    }
    std::printf("%d %zu %d %d %d %d\n", n, seen.size(), early, in_use, stuck, wrong_open);
  }
  return 0;
}
