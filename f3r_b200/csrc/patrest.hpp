// patrest.hpp -- who works the rows off their block's pattern (pattern.cuh,
// patblock.cuh): rounds of `warps` groups of 32 rows, dealt to the CTAs of a
// persistent grid beside their tiles.
//
// The CTAs with a tile fewer than the others take up to kRestSpare rounds each,
// about what that tile costs; what is left is dealt round by round to all.  Left
// to those CTAs alone, whose number is anything from 1 to the grid, the rounds
// decide the time.  27-point, 32-row slices, us a product, those CTAs alone -> here:
// fp16 134^3 (9 of 592 CTAs) 67 -> 14.4, 160^3 (368) 22.6 -> 22.6, 192^3 (96) 36.9 ->
// 33.5; fp32 176^3 (2 of 444) 521 -> 33, 192^3 46 -> 42; fp64 192^3 106.5 -> 100.7.  Two
// right-hand sides at 88^3: 222 -> 18.8 ms a solve.  One round a CTA costs 10% in fp64
// at 100^3, four cost 9% at 192^3.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define F3R_HD __host__ __device__ __forceinline__
#else
#define F3R_HD inline
#endif

namespace f3r {

constexpr int kRestSpare = 2;

// Set up by the host, read by the kernels from their arguments.
struct PatRest {
  int32_t rounds, idle, first;  // of all; CTAs with a tile fewer (the last ones); rounds below first are theirs
  PatRest() : rounds(0), idle(1), first(0) {}
  PatRest(int ntiles, int ngroups, int warps, int grid) {
    rounds = (ngroups + warps - 1) / warps;
    idle = grid - ntiles % grid;
    first = rounds / kRestSpare < idle ? rounds : kRestSpare * idle;
  }
  // a CTA's first round and the one after round `at`; rounds and above: none
  F3R_HD int begin(int cta, int grid) const {
    const int at = cta >= grid - idle ? cta - (grid - idle) : first;
    return at < first ? at : first + cta;
  }
  F3R_HD int next(int at, int cta, int grid) const {
    if (at >= first) return at + grid;
    return at + idle < first ? at + idle : first + cta;
  }
};

}  // namespace f3r
