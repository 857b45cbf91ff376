// Every interleaving of a producer, the threads that issue MMAs, the landing of loads (in any order) and the
// completion of MMAs over the operand ring: no block may be multiplied before its load has landed, no stage
// refilled before it has been read, and every block must be reached.  Exit status 0: holds for the rings below.
#include <stdio.h>

#include <set>
#include <vector>

#include "operand_ring.h"

// the ring with one full barrier per stage, whatever the number of issuing threads: must be found wrong
template <int S, int I>
struct OneBarrierPerStage : sd3::OperandRing<S, I> {
  static constexpr int FULL_BARS = S;
  void next() {
    sd3::OperandRing<S, I>::next();
    this->full = this->stage;
    this->full_parity = this->stage_parity;
  }
};

enum : signed char { NONE, LOADING, LANDED, ISSUED, DONE };

// An mbarrier's wait on parity p returns once the current phase's parity differs from p.
static bool passes(int completed_phases, unsigned parity) { return (completed_phases & 1u) != parity; }

template <typename Ring, int BUFS>
struct Model {
  static constexpr int BLOCKS = 4 * Ring::STAGES;
  std::vector<Ring> at;  // ring position of each block
  std::set<std::vector<signed char>> seen;
  const char* error = nullptr;

  Model() {
    Ring r;
    for (int b = 0; b < BLOCKS; ++b, r.next()) at.push_back(r);
  }
  // Completed phases of the barriers follow from the blocks' states.
  int full_phases(const std::vector<signed char>& s, int bar) const {
    int n = 0;
    for (int b = 0; b < BLOCKS; ++b) n += at[b].full == bar && s[b] >= LANDED;
    return n;
  }
  int empty_phases(const std::vector<signed char>& s, int stage) const {
    int n = 0;
    for (int b = 0; b < BLOCKS; ++b) n += at[b].stage == stage && s[b] == DONE;
    return n;
  }
  void run() {
    std::vector<std::vector<signed char>> todo{std::vector<signed char>(BLOCKS, NONE)};
    while (!todo.empty() && !error) {
      const std::vector<signed char> s = todo.back();
      todo.pop_back();
      if (!seen.insert(s).second) continue;
      bool moved = false;
      auto go = [&](int b, signed char to) {
        std::vector<signed char> t = s;
        t[b] = to;
        todo.push_back(t);
        moved = true;
      };
      int next_load = 0;
      while (next_load < BLOCKS && s[next_load] != NONE) ++next_load;
      if (next_load < BLOCKS && passes(empty_phases(s, at[next_load].stage), at[next_load].stage_parity ^ 1)) {
        if (next_load >= Ring::STAGES && s[next_load - Ring::STAGES] != DONE) error = "a stage was refilled before it was read";
        go(next_load, LOADING);
      }
      for (int t = 0; t < Ring::ISSUERS; ++t) {
        int b = t;  // the thread's next block
        while (b < BLOCKS && (s[b] == ISSUED || s[b] == DONE)) b += Ring::ISSUERS;
        if (b >= BLOCKS || (b >= BUFS && s[b - BUFS] != DONE)) continue;  // its accumulator is drained
        if (!passes(full_phases(s, at[b].full), at[b].full_parity)) continue;
        if (s[b] != LANDED) { error = "a block was multiplied before its load had landed"; break; }
        go(b, ISSUED);
      }
      for (int b = 0; b < BLOCKS; ++b) {
        if (s[b] == LOADING) go(b, LANDED);
        if (s[b] == ISSUED && (b < Ring::ISSUERS || s[b - Ring::ISSUERS] == DONE)) go(b, DONE);
      }
      if (!moved && !error)
        for (int b = 0; b < BLOCKS; ++b)
          if (s[b] != DONE) error = "stuck";
    }
  }
};

template <typename Ring>
static bool holds(const char* name) {
  Model<Ring, 4> m;
  m.run();
  printf("%s stages %d, threads %d: %zu states, %s\n", name, Ring::STAGES, Ring::ISSUERS, m.seen.size(),
         m.error ? m.error : "holds");
  return !m.error;
}

int main() {
  bool ok = holds<sd3::OperandRing<2, 2>>("ring") && holds<sd3::OperandRing<3, 2>>("ring") &&
            holds<sd3::OperandRing<4, 2>>("ring") && holds<sd3::OperandRing<3, 1>>("ring");
  ok = ok && holds<OneBarrierPerStage<2, 2>>("one barrier per stage") && !holds<OneBarrierPerStage<3, 2>>("one barrier per stage");
  return ok ? 0 : 1;
}
