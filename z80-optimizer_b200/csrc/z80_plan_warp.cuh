// z80_plan_warp.cuh -- the pair plan of z80_plan.cuh by a warp, a lane per
// field.  Compiled for the host as well, where the including file supplies the
// warp's collectives (a test runs 32 lanes of it beside plan_pair).
#pragma once
#include <cstdint>

#include "z80_plan.cuh"

#if defined(__CUDACC__)
#define Z80B_WARP __device__ __forceinline__
#else
#define Z80B_WARP inline
#endif

namespace z80b {

// A pair's two programs, one instruction per lane: lanes 0..tl-1 the target,
// lanes tl..tl+cl-1 the candidate.
struct PairWords {
  uint32_t w;        // this lane's instruction (0 past the programs)
  uint32_t tl, cl;
  Z80B_WARP bool mine(unsigned lane) const { return lane < tl + cl; }
};

// plan_pair (z80_plan.cuh) by a warp, lane g on field g: the names of the
// fields are in the lanes, an instruction's dependency sets are met by ballots.
Z80B_WARP PairPlan plan_pair_warp(unsigned lane, const unsigned long long (*flow)[kFlowFields], const PairWords& p,
                                  uint32_t reads, uint32_t keepF, uint32_t keepR) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  const uint32_t n = p.tl + p.cl;
  unsigned long long row[kPlanMaxInsn];
  uint32_t word[kPlanMaxInsn], in[kPlanMaxInsn], out[kPlanMaxInsn];
#pragma unroll
  for (int i = 0; i < kPlanMaxInsn; i++) {
    word[i] = __shfl_sync(kFull, p.w, i);
    row[i] = 0;
    in[i] = out[i] = 0;
    if (uint32_t(i) < n && lane < kFlowFields) row[i] = flow[word[i] & 0xFFFFu][lane];
  }
  const uint32_t varying = plan_varying(reads), cmp = plan_compared(keepF, keepR);
  const uint32_t first = ((varying >> lane) & 1u) ? 256u + lane : 0u;
  uint32_t cur = first, end_t = 0;
#pragma unroll
  for (int i = 0; i < kPlanMaxInsn; i++) {
    if (uint32_t(i) >= n) break;
    if (uint32_t(i) == p.tl) {
      end_t = cur;
      cur = first;
    }
    in[i] = cur;
    const uint32_t dep = uint32_t(row[i]) & 0xFFFFFFu, src = uint32_t(row[i] >> 24) & 0xFFu;
    const uint32_t cst = uint32_t(row[i] >> 32) & 0xFFFFu;
    const uint32_t copy = __shfl_sync(kFull, cur, int(src & 31u));
    uint32_t id;
    if (!((row[i] >> 48) & 1u)) id = cur;
    else if (src != 0xFFu) id = copy;
    else if (cst < 256u) id = cst;
    else if (cst == kFlowImmLo) id = (word[i] >> 16) & 0xFFu;
    else if (cst == kFlowImmHi) id = word[i] >> 24;
    else id = 280u + 24u * i + lane;
    const bool computed = id == 280u + 24u * i + lane;
    bool found = false;
#pragma unroll
    for (int j = 0; j < i; j++) {
      if (word[j] != word[i]) continue;
      const unsigned same = __ballot_sync(kFull, in[j] == in[i]);
      if (computed && !found && (dep & ~same) == 0) {
        id = out[j];
        found = true;
      }
    }
    out[i] = id;
    cur = id;
  }
  if (p.cl == 0) end_t = cur;
  const uint32_t open = __ballot_sync(kFull, end_t != cur) & cmp;
  // what outputs can depend on, walked backwards over lanes [lo, hi)
  auto relevant = [&](uint32_t lo, uint32_t hi, uint32_t o) {
#pragma unroll
    for (int i = kPlanMaxInsn - 1; i >= 0; i--) {
      if (uint32_t(i) < lo || uint32_t(i) >= hi) continue;
      const bool on = (o >> lane) & 1u, changed = (row[i] >> 48) & 1u;
      o = __reduce_or_sync(kFull, !on ? 0u : (changed ? uint32_t(row[i]) & 0xFFFFFFu : 1u << lane));
    }
    return o;
  };
  bool keeps_t = true, keeps_c = true;
#pragma unroll
  for (int i = 0; i < kPlanMaxInsn; i++) {
    const bool ch = __shfl_sync(kFull, uint32_t(row[i] >> 48) & 1u, 0) != 0u;
    if (uint32_t(i) < p.tl) keeps_t = keeps_t && !ch;
    else if (uint32_t(i) < n) keeps_c = keeps_c && !ch;
  }
  const uint32_t rest = open & ~uint32_t(kRegA), a = open & kRegA;
  return plan_from(reads, open, relevant(0, p.tl, rest) | relevant(p.tl, n, rest), a ? relevant(0, p.tl, a) : 0u,
                   a ? relevant(p.tl, n, a) : 0u, keeps_t, keeps_c);
}

}  // namespace z80b
