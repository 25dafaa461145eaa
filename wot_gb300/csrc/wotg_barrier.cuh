// wotg_barrier.cuh — the word of a cooperative kernel's grid barrier.
//
// Bits 0-23 count the CTAs' arrivals; bits 24-43 and 44-63 count two flags that an
// arrival may raise. All three only grow during a launch, and a CTA knows a flag was
// raised at a barrier by its count having moved since the CTA last took flags.
//
// A CTA may read the word late: when it sees barrier k complete, faster CTAs may
// already have arrived at k + 1 (and at no later one, which needs its own arrival). A
// barrier that carries no flags therefore leaves the counts last taken alone: taking
// what it happens to read would swallow a flag of k + 1, and this CTA alone would then
// find none there. Flags are taken where they are asked for; a barrier after one that
// takes flags carries none of the same kind, or its flags are or-ed with those before
// (a flag read one barrier early is then seen once, as by every other CTA).
#pragma once

#include <stdint.h>

namespace wotg {

constexpr int kBarrierArrivalBits = 24, kBarrierFlagBits = 20;

// What a CTA keeps between barriers: the arrivals that complete the next one, the flag
// counts last taken.
struct BarrierSeen {
  unsigned int target, flags, flags2;
};

__host__ __device__ inline unsigned long long barrier_arrival(bool flag, bool flag2) {
  return 1ull + ((unsigned long long)(flag ? 1 : 0) << kBarrierArrivalBits) +
         ((unsigned long long)(flag2 ? 1 : 0) << (kBarrierArrivalBits + kBarrierFlagBits));
}
__host__ __device__ inline bool barrier_complete(unsigned long long word, const BarrierSeen& s) {
  return ((unsigned int)word & ((1u << kBarrierArrivalBits) - 1)) >= s.target;
}
// Of a complete barrier of n CTAs: whether a flag was raised since flags were last taken.
__host__ __device__ inline void barrier_pass(unsigned long long word, int n, bool take, BarrierSeen& s, bool* raised,
                                             bool* raised2) {
  s.target += n;
  *raised = *raised2 = false;
  if (!take) return;
  const unsigned int f = (unsigned int)(word >> kBarrierArrivalBits) & ((1u << kBarrierFlagBits) - 1);
  const unsigned int f2 = (unsigned int)(word >> (kBarrierArrivalBits + kBarrierFlagBits));
  *raised = f != s.flags;
  *raised2 = f2 != s.flags2;
  s.flags = f;
  s.flags2 = f2;
}

}  // namespace wotg
