// The operand ring of a GEMM whose MMAs are issued by several threads in turn: which stage, which barriers
// and which barrier phases a K block uses.  Plain C++, so that the schedule can be model-checked on the host.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define SD3_RING_FN __host__ __device__ __forceinline__
#else
#define SD3_RING_FN inline
#endif

namespace sd3 {

// Block b of the sequence lives in stage b % STAGES and is issued by thread b % ISSUERS.  A wait on an
// mbarrier tests one bit, the parity of the phase: it cannot tell the phase that is waited for from the one
// two before it, so a thread may only wait on a barrier of which it has seen every phase.  The producer sees
// every phase of a stage's "empty" barrier.  A thread that takes every second block of a ring with an odd
// number of stages sees every second use of a stage only: with one "full" barrier per stage it would take the
// barrier as complete for block b while the load of block b - STAGES, the other thread's, is still under way.  There are
// therefore as many "full" barriers as it takes for all uses of one to belong to the same thread: block b is
// announced on barrier b % FULL_BARS, whose previous use, b - FULL_BARS, the thread of block b has waited for itself.
template <int STAGES_, int ISSUERS_>
struct OperandRing {
  static constexpr int STAGES = STAGES_;
  static constexpr int ISSUERS = ISSUERS_;
  static constexpr int FULL_BARS = STAGES % ISSUERS == 0 ? STAGES : STAGES * ISSUERS;
  static_assert(FULL_BARS % STAGES == 0 && FULL_BARS % ISSUERS == 0, "a barrier belongs to one stage and one thread");

  int stage = 0, full = 0, turn = 0;  // of the current block: its stage, its full barrier, the thread that issues it
  uint32_t stage_parity = 0;          // parity of the current use of the stage (empty barrier)
  uint32_t full_parity = 0;           // parity of the phase its load completes on the full barrier

  SD3_RING_FN void next() {
    if (++stage == STAGES) { stage = 0; stage_parity ^= 1; }
    if (++full == FULL_BARS) { full = 0; full_parity ^= 1; }
    if (++turn == ISSUERS) turn = 0;
  }
};

}  // namespace sd3
