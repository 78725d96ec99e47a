// Host check of the pair planning (z80_plan.cuh) against the oracle.
// (1) op_flow: under the oracle's Exec no output changes with an input
// outside its dependency set, copies are exact copies, constants constant.
// (2) Random pairs, most with shared instructions, dead flags and dead
// registers: a pair said to be proven passes the oracle's ExhaustiveCheck,
// and for the others the planned sweep (fields left out at 0, the carry and
// A cut down where the plan says so, a reduced sweep staying reduced) gives
// the oracle's verdict.
#include <cstdio>
#include <random>

#include "../../oracle/z80_oracle.h"
#include "../../z80-optimizer_b200/csrc/z80_exec.cuh"
#include "../../z80-optimizer_b200/csrc/z80_tables.h"

using namespace z80b;

static const int kFields[] = {0, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 18, 19, 20, 21, 22, 23};
static uint32_t get_field(const orc::State& s, int g) {
  switch (g) {
    case 0: return s.A;
    case 2: return s.B;
    case 3: return s.C;
    case 4: return s.D;
    case 5: return s.E;
    case 6: return s.H;
    case 7: return s.L;
    case 8: return s.SP;
    case 9: return s.M;
    default: return (s.F >> (g - kDepF0)) & 1u;
  }
}
static void set_field(orc::State& s, int g, uint32_t v) {
  switch (g) {
    case 0: s.A = uint8_t(v); break;
    case 2: s.B = uint8_t(v); break;
    case 3: s.C = uint8_t(v); break;
    case 4: s.D = uint8_t(v); break;
    case 5: s.E = uint8_t(v); break;
    case 6: s.H = uint8_t(v); break;
    case 7: s.L = uint8_t(v); break;
    case 8: s.SP = uint16_t(v); break;
    case 9: s.M = uint8_t(v); break;
    default: s.F = uint8_t((s.F & ~(1u << (g - kDepF0))) | ((v & 1u) << (g - kDepF0))); break;
  }
}

// the planned sweep, block index fields fastest first: SP, the swept
// registers from the last to the first, the carry
static bool planned_sweep(const uint32_t* tw, int tn, const uint32_t* cw, int cn, const PairPlan& pl, uint32_t keepF,
                          uint32_t keepR) {
  const uint32_t bits[7] = {kRegB, kRegC, kRegD, kRegE, kRegH, kRegL, kRegM};
  int slot[7], nx = 0;
  for (int r = 0; r < 7; r++) slot[r] = (pl.reads & bits[r]) ? nx++ : -1;
  const bool spw = (pl.reads & kRegSP) != 0, reduced = spw || nx > 2 || (pl.sweepf & 0x80);
  for (uint64_t b = 0; b < pl.nblocks; b++) {
    uint64_t rest = b;
    Z80S x{};
    if (spw) {
      x.sp = rep_sp()[rest & 15];
      rest >>= 4;
    }
    uint32_t fv[7] = {};
    for (int f = nx - 1; f >= 0; f--) {
      fv[f] = reduced ? rep_values()[rest & 31] : uint32_t(rest & 255);
      rest >>= reduced ? 5 : 8;
    }
    uint32_t rv[7];
    for (int r = 0; r < 7; r++) rv[r] = slot[r] >= 0 ? fv[slot[r]] : 0;
    x.b = rv[0];
    x.c = rv[1];
    x.d = rv[2];
    x.e = rv[3];
    x.h = rv[4];
    x.l = rv[5];
    x.m = rv[6];
    x.f = uint32_t(rest & 1);
    for (uint32_t a = 0; a < (pl.a_free ? 2u : 256u); a++) {
      Z80S s = x, t = x;
      s.a = t.a = a;
      for (int i = 0; i < tn; i++) z_step(t, insn_op(tw[i]), insn_imm(tw[i]));
      for (int i = 0; i < cn; i++) z_step(s, insn_op(cw[i]), insn_imm(cw[i]));
      uint32_t d = (s.a ^ t.a) | (s.sp ^ t.sp) | (s.m ^ t.m) | ((s.f ^ t.f) & keepF);
      const uint32_t dr[6] = {s.b ^ t.b, s.c ^ t.c, s.d ^ t.d, s.e ^ t.e, s.h ^ t.h, s.l ^ t.l};
      for (int r = 0; r < 6; r++)
        if ((keepR >> r) & 1u) d |= dr[r];
      if (d) return false;
    }
  }
  return true;
}

int main() {
  orc::Init();
  std::mt19937_64 rng(71);
  const OpFlow* F = op_flow();
  long checks = 0;
  for (int op = 0; op < orc::OpCodeCount; op++) {
    for (int k = 0; k < 64; k++) {
      const uint64_t r = rng(), r2 = rng();
      const orc::State s{uint8_t(r), uint8_t(r >> 8), uint8_t(r >> 16), uint8_t(r >> 24), uint8_t(r >> 32),
                         uint8_t(r >> 40), uint8_t(r >> 48), uint8_t(r >> 56), uint16_t(r2), uint8_t(r2 >> 16)};
      const int kind = op_table()[op].imm;
      const uint16_t imm = kind == 0 ? uint16_t(0) : (kind == 1 ? uint16_t(rng() & 0xFF) : uint16_t(rng()));
      orc::State base = s;
      orc::Exec(base, uint16_t(op), imm);
      for (int g : kFields) {
        const uint32_t v = get_field(base, g);
        bool ok = true;
        if (!((F[op].changed >> g) & 1u)) ok = v == get_field(s, g);
        else if (F[op].src[g] != 0xFF) ok = v == get_field(s, F[op].src[g]);
        else if (F[op].cst[g] < 256) ok = v == F[op].cst[g];
        else if (F[op].cst[g] == kFlowImmLo) ok = v == (imm & 0xFFu);
        else if (F[op].cst[g] == kFlowImmHi) ok = v == (imm >> 8);
        if (!ok) {
          std::printf("op %d (%s): output field %d is not the copy or constant it is said to be\n", op,
                      op_mnemonic(uint16_t(op)), g);
          return 1;
        }
      }
      for (int f : kFields)
        for (int v = 0; v < 4; v++) {
          orc::State t = s;
          const uint32_t old = get_field(s, f);
          set_field(t, f, f >= kDepF0 ? (old ^ 1u) : (f == 8 ? uint32_t(rng() & 0xFFFF) : uint32_t(rng() & 0xFF)));
          orc::Exec(t, uint16_t(op), imm);
          for (int g : kFields) {
            if (F[op].dep[g] & (1u << f)) continue;
            if (!((F[op].changed >> g) & 1u) && f == g) continue;
            checks++;
            if (get_field(t, g) != get_field(base, g)) {
              std::printf("op %d (%s): output field %d changes with input field %d outside its set\n", op,
                          op_mnemonic(uint16_t(op)), g, f);
              return 1;
            }
          }
        }
    }
  }

  const auto& I = orc::Instructions8();
  int pairs = 0, proven = 0, equal = 0, sp_out = 0, cut = 0;
  for (int trial = 0; trial < 4000000 && (pairs < 6000 || proven < 1500 || sp_out < 150); trial++) {
    // the candidate, and a target made of it with instructions put in, taken
    // for others or left alone
    int cn = 1 + int(rng() % 2), tn = cn + 1 + int(rng() % 2);
    if (tn > 4) tn = 4;
    orc::Instruction ti[4], ci[3];
    auto pick = [&] {
      // one in four from the 16-bit and memory part of the list
      if (rng() % 4 == 0) {
        orc::Instruction in{};
        in.op = uint16_t(INC_BC + rng() % (kNumOps - INC_BC));
        if (op_table()[in.op].imm == 2) in.op = uint16_t(ADD_HL_DE);
        in.imm = op_table()[in.op].imm ? uint16_t(rng() & 0xFF) : uint16_t(0);
        return in;
      }
      return I[rng() % I.size()];
    };
    for (int i = 0; i < cn; i++) ci[i] = pick();
    for (int i = 0, m = 0; i < tn; i++) {
      const bool take = m < cn && (tn - i <= cn - m || rng() % 2);
      ti[i] = take ? ci[m++] : pick();
    }
    if (rng() % 4 == 0) ti[rng() % tn] = pick();
    uint32_t tw[4], cw[3];
    uint8_t named = 0;
    for (int i = 0; i < tn; i++) {
      tw[i] = uint32_t(ti[i].op) | uint32_t(ti[i].imm) << 16;
      if (rng() % 2) named |= uint8_t(op_regs(ti[i].op) & 0x3F);
    }
    for (int i = 0; i < cn; i++) cw[i] = uint32_t(ci[i].op) | uint32_t(ci[i].imm) << 16;
    const uint8_t dead = rng() % 3 == 0 ? uint8_t(0xFF) : (rng() % 3 == 0 ? uint8_t(0) : uint8_t(rng()));
    const uint8_t dregs = uint8_t(rng() % 2 ? named : rng() & 0x3F);
    const uint32_t keepF = uint8_t(~dead), keepR = ~uint32_t(dregs) & 0x3Fu;
    const uint16_t reads = uint16_t(seq_reads(tw, tn) | seq_reads(cw, cn));
    if (sweep_for(reads).states > (1ull << 22)) continue;
    const PairPlan pl = plan_pair(F, tw, uint32_t(tn), cw, uint32_t(cn), reads, keepF, keepR);
    if (!pl.proven && pl.nblocks > 4096) continue;
    const bool first_said = pl.proven || planned_sweep(tw, tn, cw, cn, pl, keepF, keepR);
    // pairs that fail are many: keep some of them
    if (!first_said && equal * 3 < pairs) continue;
    const bool want = orc::ExhaustiveCheckMaskedRegs(ti, tn, ci, cn, dead, dregs);
    if (want != first_said) {
      std::printf("verdict differs: %s -> %s dead %02x regs %02x: planned %d (proven %d), oracle %d\n",
                  disasm_seq(tw, tn).c_str(), disasm_seq(cw, cn).c_str(), dead, dregs, int(first_said),
                  int(pl.proven), int(want));
      return 1;
    }
    pairs++;
    equal += want;
    proven += pl.proven;
    sp_out += !pl.proven && (reads & ~pl.reads & kRegSP) != 0;
    cut += !pl.proven && pl.sweepf != 0;
  }
  if (proven < 1500 || pairs < 6000 || equal == proven || sp_out < 150 || cut < 1000) {
    std::printf("too few pairs (%d), proven (%d), equivalent (%d), without SP (%d), cut (%d)\n", pairs, proven, equal,
                sp_out, cut);
    return 1;
  }
  std::printf("OK plan: %ld independence checks; %d pairs, %d equivalent, %d of them proven, %d sweeps cut, %d "
              "without SP\n", checks, pairs, equal, proven, cut, sp_out);
  return 0;
}
