// z80_plan.cuh -- what decides the ExhaustiveCheck of a (target, candidate)
// pair, worked out from its two programs before anything is swept.  plan_pair
// is the rule in plain C++ (checked against the oracle on the host); the
// kernel that plans pairs (plan_pair_warp in z80b_kernels.cu) is the same with
// a lane per field, and shares plan_from below.
//
// Value numbers.  Both programs run on names instead of values: a field (A,
// a register, SP, the memory byte, a flag bit) holds the name of an input
// field, a constant, or "output g of instruction w on inputs so named".  Two
// equal names are equal values for every state of the sweep, because an
// instruction's output depends on nothing but the fields of its dependency
// set (op_deps) and the immediate.  A compared output with the same name in
// both programs needs no sweep; only the others (`open`) do:
//  - none open: the pair is equivalent, nothing is swept;
//  - else only the inputs that an open output depends on are swept, A at two
//    values where that decides (see below), and the carry only if needed.
// Measured (1 B200): the length-2 enumeration of 9.4M targets evaluated
// 1.3e9 states where leaving out only what nothing compared depends on took
// 3.7e9 (ExhaustiveCheck 8.1 -> 3.1 ms); 100,003 targets with every flag dead
// 2.3e7 where it took 1.3e8 to 6.8e8.  With the probe of long sweeps
// (k_pair_plan) the enumeration evaluates 2.8e8.
// What the sweep would find is unchanged: the outputs left out agree in
// every state of it, and the inputs left out cannot change the others.
#pragma once
#include <cstdint>

#include "z80_isa.h"

#if defined(__CUDACC__)
#define Z80B_PLAN_HD __host__ __device__ __forceinline__
#else
#define Z80B_PLAN_HD inline
#endif

namespace z80b {

// Per-opcode flow of one instruction, in the field layout of op_deps (A bit
// 0, B..L bits 2..7, SP bit 8, the memory byte bit 9, flag bits 16..23).
constexpr int kFlowFields = 24;
struct OpFlow {
  uint32_t dep[kFlowFields];   // input fields output field g depends on
  uint32_t changed;            // output fields that are not simply their own input
  uint8_t src[kFlowFields];    // output g is an exact copy of this input field; 0xFF: computed
  uint16_t cst[kFlowFields];   // output g is this constant; kFlowImmLo / kFlowImmHi: a byte of the
                               // immediate; kFlowNoConst: not a constant
};
// One field of OpFlow in 64 bits, as the kernels read it: dep (24 bits), src
// (8), cst (16), changed (1).
inline uint64_t flow_word(const OpFlow& f, int g) {
  return uint64_t(f.dep[g]) | uint64_t(f.src[g]) << 24 | uint64_t(f.cst[g]) << 32 | uint64_t(f.changed >> g & 1u) << 48;
}
constexpr uint16_t kFlowImmLo = 0x100, kFlowImmHi = 0x101, kFlowNoConst = 0xFFFF;
constexpr uint32_t kFlowCarry = 1u << 16;

// The longest pair: targets of up to 4 instructions, candidates of up to 3.
constexpr int kPlanMaxInsn = 7;

Z80B_PLAN_HD int plan_ctz(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __ffs(int(x)) - 1;
#else
  return __builtin_ctz(x);
#endif
}
Z80B_PLAN_HD int plan_popc(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __popc(x);
#else
  return __builtin_popcount(x);
#endif
}

// Input fields that the outputs in `out` of a program can depend on.
Z80B_PLAN_HD uint32_t flow_relevant(const OpFlow* F, const uint32_t* w, uint32_t n, uint32_t out) {
  for (int i = int(n) - 1; i >= 0; i--) {
    const OpFlow& f = F[w[i] & 0xFFFFu];
    uint32_t in = out & ~f.changed;
    for (uint32_t o = out & f.changed; o; o &= o - 1) in |= f.dep[plan_ctz(o)];
    out = in;
  }
  return out;
}
// Whether a program leaves A exactly as it was.
Z80B_PLAN_HD bool flow_keeps_a(const OpFlow* F, const uint32_t* w, uint32_t n) {
  for (uint32_t i = 0; i < n; i++)
    if (F[w[i] & 0xFFFFu].changed & 1u) return false;
  return true;
}

// The compared outputs (cmp) of the two programs whose value numbers differ.
// `varying`: the input fields that the sweep moves; every other field is 0 in
// all of its states.
Z80B_PLAN_HD uint32_t open_outputs(const OpFlow* F, const uint32_t* tw, uint32_t tl, const uint32_t* cw, uint32_t cl,
                                   uint32_t varying, uint32_t cmp) {
  // names: 0..255 a constant, 256 + g the input field g, 280 + 24 i + g the
  // output g that instruction i was the first to compute
  uint16_t cur[kFlowFields], end_t[kFlowFields];
  uint16_t in[kPlanMaxInsn][kFlowFields], out[kPlanMaxInsn][kFlowFields];
  uint32_t word[kPlanMaxInsn];
  int n = 0;
  for (int p = 0; p < 2; p++) {
    const uint32_t* w = p ? cw : tw;
    const uint32_t len = p ? cl : tl;
    for (int g = 0; g < kFlowFields; g++) cur[g] = ((varying >> g) & 1u) ? uint16_t(256 + g) : uint16_t(0);
    for (uint32_t k = 0; k < len; k++, n++) {
      const uint32_t wk = w[k];
      const OpFlow& f = F[wk & 0xFFFFu];
      word[n] = wk;
      for (int g = 0; g < kFlowFields; g++) in[n][g] = cur[g];
      for (uint32_t o = f.changed; o; o &= o - 1) {
        const int g = plan_ctz(o);
        uint16_t id;
        if (f.src[g] != 0xFF) {
          id = in[n][f.src[g]];
        } else if (f.cst[g] < 256) {
          id = f.cst[g];
        } else if (f.cst[g] == kFlowImmLo) {
          id = uint16_t((wk >> 16) & 0xFFu);
        } else if (f.cst[g] == kFlowImmHi) {
          id = uint16_t(wk >> 24);
        } else {
          id = uint16_t(280 + 24 * n + g);
          for (int i = 0; i < n; i++) {
            if (word[i] != wk) continue;
            bool same = true;
            for (uint32_t d = f.dep[g]; d && same; d &= d - 1) {
              const int e = plan_ctz(d);
              same = in[i][e] == in[n][e];
            }
            if (same) {
              id = out[i][g];
              break;
            }
          }
        }
        out[n][g] = id;
        cur[g] = id;
      }
    }
    if (p == 0)
      for (int g = 0; g < kFlowFields; g++) end_t[g] = cur[g];
  }
  uint32_t open = 0;
  for (uint32_t o = cmp; o; o &= o - 1) {
    const int g = plan_ctz(o);
    if (end_t[g] != cur[g]) open |= 1u << g;
  }
  return open;
}

struct PairPlan {
  bool proven;          // every compared output has equal names: equivalent
  bool a_free;          // two values of A decide
  uint16_t reads;       // read mask of the fields that are swept
  uint8_t sweepf;       // PairRec::sweepf
  unsigned long long nblocks;  // A-blocks (256 states) of the sweep
};

// A-blocks of the reference's sweep for a read mask
// (pkg/search/verifier.go:159-171,428-476); reduced: the reference's sweep of
// the pair is a reduced one although these reads alone would not make it so
// (swept fields left out).
Z80B_PLAN_HD unsigned long long plan_blocks(uint32_t reads, bool reduced) {
  const int n = plan_popc(reads & (kRegB | kRegC | kRegD | kRegE | kRegH | kRegL | kRegM));
  const bool sp = (reads & kRegSP) != 0;
  if (n <= 2 && !sp && !reduced) return 2ull << (8 * n);
  return (2ull << (5 * n)) * (sp ? 16ull : 1ull);
}

// A sweep of `units` units in chunks of chunk_blocks units, at most max_chunks
// of them: their number, and the units of one.
Z80B_PLAN_HD uint32_t chunk_count(unsigned long long units, uint32_t chunk_blocks, uint32_t max_chunks) {
  const unsigned long long c = (units + chunk_blocks - 1) / chunk_blocks;
  return c > max_chunks ? max_chunks : uint32_t(c);
}
Z80B_PLAN_HD unsigned long long chunk_units(unsigned long long units, uint32_t chunks) {
  return (units + chunks - 1) / chunks;
}

// The plan from the open outputs: rest, what those other than A can depend on;
// at / ac, what A can (where it is open) in either program; keeps_t / keeps_c:
// the program leaves A as it was.
Z80B_PLAN_HD PairPlan plan_from(uint32_t reads, uint32_t open, uint32_t rest, uint32_t at, uint32_t ac, bool keeps_t,
                                bool keeps_c) {
  PairPlan r;
  const uint32_t ext = reads & (kRegB | kRegC | kRegD | kRegE | kRegH | kRegL | kRegM);
  const uint32_t sp = reads & kRegSP;
  r.proven = open == 0;
  const uint32_t rel = rest | at | ac;
  const uint32_t drop = (ext | sp) & ~rel;
  const bool red = sp != 0 || plan_popc(ext) > 2;
  r.reads = uint16_t(reads & ~drop);
  r.sweepf = 0;
  if (drop)
    r.sweepf = uint8_t((red ? 0x80u : 0u) | (uint32_t(plan_popc(drop & ext)) * (red ? 5u : 8u) + ((drop & sp) ? 4u : 0u)));
  r.nblocks = plan_blocks(r.reads, (r.sweepf & 0x80u) != 0);
  // the carry, the most significant field of the block index: when no open
  // output depends on it the first half of the blocks (carry 0) decides
  if (!(rel & kFlowCarry)) {
    r.nblocks >>= 1;
    r.sweepf += 1;
  }
  // Two values of A decide when no open output but A depends on the input A
  // and each program keeps A or computes its A from other inputs.
  r.a_free = !(rest & kRegA) && (!(at & kRegA) || keeps_t) && (!(ac & kRegA) || keeps_c);
  return r;
}
// Compared outputs and varying inputs of a pair.  reads: the union of the
// programs' read masks; keepF: compared flag bits; keepR: compared registers
// (bits 0..5 = B..L).  A, SP and the memory byte are always compared.
Z80B_PLAN_HD uint32_t plan_compared(uint32_t keepF, uint32_t keepR) {
  return kRegA | kRegSP | kRegM | ((keepR & 0x3Fu) << 2) | ((keepF & 0xFFu) << 16);
}
Z80B_PLAN_HD uint32_t plan_varying(uint32_t reads) {
  return (reads & (kRegB | kRegC | kRegD | kRegE | kRegH | kRegL | kRegM | kRegSP)) | kRegA | kFlowCarry;
}

Z80B_PLAN_HD PairPlan plan_pair(const OpFlow* F, const uint32_t* tw, uint32_t tl, const uint32_t* cw, uint32_t cl,
                                uint32_t reads, uint32_t keepF, uint32_t keepR) {
  const uint32_t open = open_outputs(F, tw, tl, cw, cl, plan_varying(reads), plan_compared(keepF, keepR));
  const uint32_t rest = flow_relevant(F, tw, tl, open & ~uint32_t(kRegA)) | flow_relevant(F, cw, cl, open & ~uint32_t(kRegA));
  return plan_from(reads, open, rest, flow_relevant(F, tw, tl, open & kRegA), flow_relevant(F, cw, cl, open & kRegA),
                   flow_keeps_a(F, tw, tl), flow_keeps_a(F, cw, cl));
}

}  // namespace z80b
