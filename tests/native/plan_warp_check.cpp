// Host check of the pair plan that the kernel runs (z80_plan_warp.cuh, a lane
// per field) against plan_pair (z80_plan.cuh), field by field.  The 32 lanes
// are 32 contexts of this program, switched at the warp's collectives; a lane
// that came to another collective than the rest would be caught.
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

static struct {
  ucontext_t host, lane[32];
  char stack[32][64 << 10];
  uint32_t slot[2][32];  // what the lanes gave to a collective; the next one uses the other row
  int kind[2][32];
  int phase[32], cur;
} W;
static const uint32_t* meet(int kind, uint32_t v) {
  const int me = W.cur, ph = W.phase[me]++;
  W.slot[ph & 1][me] = v;
  W.kind[ph & 1][me] = kind;
  swapcontext(&W.lane[me], &W.host);  // back when every lane has come
  for (int l = 0; l < 32; l++)
    if (W.phase[l] < ph + 1 || W.phase[l] > ph + 2 || W.kind[ph & 1][l] != kind) {
      std::printf("lanes %d and %d part at collective %d\n", me, l, ph);
      std::exit(1);
    }
  return W.slot[ph & 1];
}
static uint32_t __shfl_sync(unsigned, uint32_t v, int src) { return meet(1, v)[src & 31]; }
static unsigned __ballot_sync(unsigned, bool p) {
  const uint32_t* s = meet(2, p);
  unsigned r = 0;
  for (int l = 0; l < 32; l++) r |= s[l] << l;
  return r;
}
static uint32_t __reduce_or_sync(unsigned, uint32_t v) {
  const uint32_t* s = meet(3, v);
  uint32_t r = 0;
  for (int l = 0; l < 32; l++) r |= s[l];
  return r;
}

#include "../../z80-optimizer_b200/csrc/z80_plan_warp.cuh"
#include "../../z80-optimizer_b200/csrc/z80_tables.h"

using namespace z80b;

static unsigned long long g_flow[kNumOps][kFlowFields];
static struct {
  const uint32_t *t, *c;
  uint32_t tl, cl, reads, keepF, keepR;
} Q;
static PairPlan got[32];

static void lane_main(int lane) {
  PairWords p;
  p.tl = Q.tl;
  p.cl = Q.cl;
  p.w = uint32_t(lane) < p.tl ? Q.t[lane] : uint32_t(lane) < p.tl + p.cl ? Q.c[lane - int(p.tl)] : 0u;
  got[lane] = plan_pair_warp(unsigned(lane), g_flow, p, Q.reads, Q.keepF, Q.keepR);
}
static void run_warp() {
  for (int l = 0; l < 32; l++) {
    getcontext(&W.lane[l]);
    W.lane[l].uc_stack.ss_sp = W.stack[l];
    W.lane[l].uc_stack.ss_size = sizeof W.stack[l];
    W.lane[l].uc_link = &W.host;
    makecontext(&W.lane[l], (void (*)())lane_main, 1, l);
    W.phase[l] = 0;
  }
  // each turn runs every lane up to its next collective, or to its end
  for (bool more = true; more;) {
    const int before = W.phase[31];
    for (W.cur = 0; W.cur < 32; W.cur++) swapcontext(&W.host, &W.lane[W.cur]);
    more = W.phase[31] != before;
  }
  for (int l = 1; l < 32; l++)
    if (W.phase[l] != W.phase[0]) {
      std::printf("lane %d ends after %d collectives, lane 0 after %d\n", l, W.phase[l], W.phase[0]);
      std::exit(1);
    }
}

int main() {
  for (int op = 0; op < kNumOps; op++)
    for (int g = 0; g < kFlowFields; g++) g_flow[op][g] = flow_word(op_flow()[op], g);
  std::mt19937 rng(5);
  auto any = [&](int n) { return uint32_t(rng() % unsigned(n)); };
  // few registers, so that programs meet each other's outputs; and any opcode
  std::vector<uint32_t> few;
  const auto& p8 = pool8();
  for (int i = 0; i < 24; i++) few.push_back(p8[any(int(p8.size()))]);
  int proven = 0, total = 0, swept = 0;
  for (int it = 0; it < 6000; it++) {
    uint32_t t[4], c[3];
    Q.tl = 1 + any(4);
    Q.cl = 1 + any(3);
    if (it % 200 == 0)
      for (auto& w : few) w = p8[any(int(p8.size()))];
    auto word = [&] {
      const uint32_t k = any(8);
      if (k == 0) return uint32_t(any(kNumOps)) | any(65536) << 16;
      return k < 4 ? few[any(int(few.size()))] : few[any(5)];
    };
    for (auto& w : t) w = word();
    for (auto& w : c) w = any(3) ? t[any(int(Q.tl))] : word();
    if (it % 3 == 0)  // the candidate with instructions put in
      for (uint32_t i = 0, j = 0; i < Q.tl; i++)
        if (j < Q.cl && (any(2) || Q.tl - i <= Q.cl - j)) t[i] = c[j++];
    if (it < kNumOps) t[0] = uint32_t(it) | any(65536) << 16;
    Q.t = t;
    Q.c = c;
    Q.reads = seq_reads(t, int(Q.tl)) | seq_reads(c, int(Q.cl));
    Q.keepF = any(3) ? 0xFFu : any(256);
    Q.keepR = any(3) ? 0x3Fu : any(64);
    run_warp();
    const PairPlan want = plan_pair(op_flow(), t, Q.tl, c, Q.cl, Q.reads, Q.keepF, Q.keepR);
    for (int l = 0; l < 32; l++)
      if (got[l].proven != want.proven || got[l].a_free != want.a_free || got[l].reads != want.reads ||
          got[l].sweepf != want.sweepf || got[l].nblocks != want.nblocks) {
        std::printf("pair %d (%u + %u instructions), lane %d: proven %d/%d a_free %d/%d reads %x/%x sweepf %x/%x blocks "
                    "%llu/%llu\n", it, Q.tl, Q.cl, l, got[l].proven, want.proven, got[l].a_free, want.a_free,
                    got[l].reads, want.reads, got[l].sweepf, want.sweepf, got[l].nblocks, want.nblocks);
        return 1;
      }
    total++;
    proven += want.proven;
    swept += !want.proven && (want.sweepf || want.a_free);
  }
  if (proven < 200 || swept < 500) {
    std::printf("too few: %d proven, %d with less to sweep of %d\n", proven, swept, total);
    return 1;
  }
  std::printf("OK %d pairs, %d proven, %d with less to sweep\n", total, proven, swept);
  return 0;
}
