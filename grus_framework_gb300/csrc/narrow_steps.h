// narrow_steps.h -- the words by which the CTAs of narrow.cuh's cluster agree
// on what a step found.  Plain code without CUDA types, so that the host can
// run it too.
//
// Every thread of the cluster decides for itself from these words which
// barrier it goes to next, so a word must read the same to all of them, however
// late a thread comes to read it.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GRUS_HD __host__ __device__ __forceinline__
#else
#define GRUS_HD inline
#endif

namespace grus {
namespace narrow {

// What a step found, kept by step parity.  Before the cluster barrier that ends
// a step, CTAs write the step's number into its words; after the barrier every
// thread reads them.  A CTA that has read them may run ahead and write the next
// step's before another thread reads this step's -- which are others -- but not
// those of the step after that: its barrier in between waits for that thread.
// A word holds an older step's number until it is written, so nobody clears it.
struct alignas(16) StepWords {
  uint32_t work;     // some CTA has near work left
  uint32_t spilled;  // some list was full: vertices wait in the near bitmap
  uint32_t late;     // the step took longer than the time limit
  uint32_t many;     // it relaxed so many spilled vertices that the grid should
};

GRUS_HD bool found(uint32_t word, uint32_t step) { return word == step; }

GRUS_HD StepWords &words_of(StepWords (&w)[2], uint32_t step) { return w[step & 1u]; }

constexpr int kRounds = 4;  // rounds between cluster barriers

// A CTA's pushes to other CTAs, by step parity and by the round that makes them.
// Warps decide before a round, each when it gets there, whether the block goes
// on; faster warps may already push in that round, so the decision counts the
// rounds before it only, which a block barrier has ended.
struct AwayCounts {
  uint32_t n[2][kRounds];
};

GRUS_HD uint32_t &away_in(AwayCounts &a, uint32_t step, int round) { return a.n[step & 1u][round]; }

// Whether the block goes on to `round` over its `own` entries.
GRUS_HD bool goes_on(AwayCounts &a, uint32_t step, int round, uint32_t own) {
  uint32_t sum = 0;
  for (int r = 0; r < round; ++r) sum += away_in(a, step, r);
  return round == 0 || 4u * own > sum;
}

}  // namespace narrow
}  // namespace grus
