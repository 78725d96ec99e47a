// z80b_kernels.cu -- the CUDA kernels of the verification pipeline (sm_100a).
//
// Tier 1, QuickCheck (pkg/search/verifier.go:85-94,626-638): eight lanes per
// target run it on the eight test vectors (same opcode in every lane of a
// warp), hash the outputs and read the candidates filed under the same hash
// (k_qc_bucket, k_qc_long; k_pair_scan for the candidates of two
// instructions); pools without an index are scanned 32 candidates at a time
// (k_qc_scan).  Candidate outputs are precomputed once (k_pool_outputs).
// __ballot_sync turns the per-lane verdicts into ordered survivor slots.
//
// Tier 2, MidCheck (verifier.go:98-123): one warp per pair, lane v runs both
// sequences on MidCheck vector v, __all_sync decides.
//
// Tier 3, ExhaustiveCheck (verifier.go:159-612,642-853): k_pair_plan finds
// which inputs a pair's verdict depends on (z80_plan.cuh) and tries the pair
// on 512 states; the sweep of what is left is cut into chunks of "A-blocks"
// (the 256 values of A for one carry and one assignment of the swept
// registers).  A persistent grid pulls chunks from an atomic dispenser;
// within a chunk the 32 lanes take 32 consecutive A values or blocks, so
// every lane executes the same opcode.  A mismatch sets the pair's rejected
// flag, which the other chunks of the pair poll to stop early.  The
// reference's sweep order only matters for its early exit; the verdict (all
// states equal) does not depend on it.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "z80_bits.cuh"
#include "z80_plan_warp.cuh"
#include "z80_tables.h"
#include "z80b_kernels.cuh"

namespace z80b {

namespace {
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t kResolved = 0x80000000u;
constexpr int kBlock = 256;

// Tables that lanes index with different values live in global memory (L1
// cached; lane-indexed __constant__ loads would serialise); __constant__ is
// kept for the reduced-sweep values, whose index is the same in every lane
// of a warp.  Every kernel that runs z_step gives all lanes of a warp the
// same opcode (a per-lane 455-way switch serialises by opcode).  A flag that
// other warps write (the pair's rejection flag) is read by lane 0 and
// broadcast, never read per lane in front of a warp collective: lanes that
// read it at different times would leave the warp split at the next
// __shfl_sync / __any_sync, which is undefined.
__device__ OpInfo g_ops[kNumOps];
__device__ uint32_t g_vec[32][3];  // MidCheck vectors; the first 8 are the QuickCheck vectors
__constant__ uint8_t c_rep[32];
__constant__ uint16_t c_repsp[16];
// Lane-indexed copies of the sweep values and the A-dependence class per
// opcode (AClass of z80_tables.h).
__device__ uint8_t g_rep[32];
__device__ uint16_t g_repsp[16];
__device__ uint8_t g_aclass[kNumOps];
// compact sweep: renamed opcodes and register places per register set
// (compact_tables), the registers each opcode names
__device__ int16_t g_cren[kCompactSets][kNumOps];
__device__ int8_t g_corig[kCompactSets][2];
__device__ uint8_t g_cid[64];
__device__ uint8_t g_opregs[kNumOps];
// what each opcode's outputs are computed from (flow_word of z80_plan.cuh);
// 87 KB, a row of 192 bytes per instruction read
__device__ unsigned long long g_flow[kNumOps][kFlowFields];
// wide compact sweep: as for the compact one, per register set of at most four
// registers (wide_tables)
__device__ int16_t g_wren[kWideSets][kNumOps];
__device__ int8_t g_worig[kWideSets][4];
__device__ uint8_t g_wid[64];

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Runs n instructions held one per lane (lane first+i holds instruction i).
// Every lane of the warp must call this with the same n.
__device__ __forceinline__ void run_lanes(Z80S& s, uint32_t lane_word, int first, int n) {
#pragma unroll 1
  for (int i = 0; i < n; i++) {
    uint32_t w = __shfl_sync(kFull, lane_word, first + i);
    z_step(s, w & 0xFFFFu, w >> 16);
  }
}

__device__ __forceinline__ Z80S vec_state(int v) {
  return z_unpack(g_vec[v][0], g_vec[v][1], g_vec[v][2]);
}

// Byte masks of compared registers from keepR bits (B,C,D,E,H,L).
struct Keep {
  uint32_t f, b, c, d, e, h, l, sp, m;
};
__device__ __forceinline__ Keep make_keep(uint32_t keepF, uint32_t keepR, bool cmpM) {
  Keep k;
  k.f = keepF & 0xFFu;
  k.b = (keepR & 1u) ? 0xFFu : 0u;
  k.c = (keepR & 2u) ? 0xFFu : 0u;
  k.d = (keepR & 4u) ? 0xFFu : 0u;
  k.e = (keepR & 8u) ? 0xFFu : 0u;
  k.h = (keepR & 16u) ? 0xFFu : 0u;
  k.l = (keepR & 32u) ? 0xFFu : 0u;
  k.sp = 0xFFFFu;
  k.m = cmpM ? 0xFFu : 0u;
  return k;
}
__device__ __forceinline__ bool eq_keep(const Z80S& x, const Z80S& y, const Keep& k) {
  uint32_t d = (x.a ^ y.a) | ((x.f ^ y.f) & k.f) | ((x.b ^ y.b) & k.b) | ((x.c ^ y.c) & k.c) |
               ((x.d ^ y.d) & k.d) | ((x.e ^ y.e) & k.e) | ((x.h ^ y.h) & k.h) | ((x.l ^ y.l) & k.l) |
               ((x.sp ^ y.sp) & k.sp) | ((x.m ^ y.m) & k.m);
  return d == 0;
}
// Registers (B,C,D,E,H,L -> bit 0..5) differing between packed words.
__device__ __forceinline__ uint32_t reg_diff(uint32_t d0, uint32_t d1) {
  return ((d0 >> 16) & 0xFFu ? 1u : 0u) | ((d0 >> 24) ? 2u : 0u) | ((d1 & 0xFFu) ? 4u : 0u) |
         ((d1 >> 8) & 0xFFu ? 8u : 0u) | ((d1 >> 16) & 0xFFu ? 16u : 0u) | ((d1 >> 24) ? 32u : 0u);
}

// A-independent sweeps.  When no output of either sequence depends on the
// input A except A itself passing through (AClass folds of both sequences),
// every output but A is the same for all 256 values of A, and A_out is
// either A_in or a value independent of A_in in each sequence; two values of
// A then decide the verdict of all 256 (equal outputs at A = 0 and A = 1
// imply equal non-A outputs and either both pass A through or both write the
// same constant; a sequence passing A through against one writing a
// constant differs at one of the two).  Such a pair is swept as "units" of
// 128 A-blocks with A in {0, 1}: 256 states evaluated per unit instead of
// 32,768.  PairRec.keepR bit 6 marks it.
constexpr uint32_t kXIndep = 0x40u;
constexpr unsigned long long kUnitBlocks = 128;
__device__ __forceinline__ PairWords pair_words(const DevTargets& T, uint32_t t, const DevPool& P, uint32_t c) {
  PairWords p;
  p.tl = target_len(T, t);
  p.cl = pool_len(P, c);
  const unsigned lane = lane_id();
  p.w = 0;
  if (lane < p.tl) p.w = T.insn[(size_t)t * T.stride + lane];
  else if (lane < p.tl + p.cl) p.w = P.insn[(size_t)c * P.stride + (lane - p.tl)];
  return p;
}
// The fold of the AClass table over both programs: true when no output of
// either depends on the input A but A passing through (an A-dependent
// instruction only after one that overwrites A).
__device__ __forceinline__ bool pair_xindep(const PairWords& p) {
  const uint32_t k = p.mine(lane_id()) ? g_aclass[p.w & 0xFFFFu] : 1u;
  const unsigned dep = __ballot_sync(kFull, k == 0u), over = __ballot_sync(kFull, k == 2u);
  const unsigned tm = (1u << p.tl) - 1u, cm = ((1u << p.cl) - 1u) << p.tl;
  auto free_of = [&](unsigned m) {
    const unsigned d = dep & m, o = over & m;
    return d == 0u || (o != 0u && __ffs(int(o)) < __ffs(int(d)));
  };
  return free_of(tm) && free_of(cm);
}
// The sweep class of a pair (PairRec::cmap) by the registers its
// instructions name (fp, op_regs): 1 + the register-set entry when they name
// at most two of B..L, neither SP nor the memory byte, and all rename onto B
// and C (compact_map); kWideClass | (1 + the entry) for A-dependent pairs that
// name at most four and not SP and rename onto B, C, H and L (wide_map);
// kRegClass for the rest that name neither SP nor the memory byte; else 0.
constexpr uint8_t kWideClass = 0x80u;
constexpr uint8_t kRegClass = 0x40u;
__device__ __forceinline__ uint8_t pair_cmap(const PairWords& p, bool compact, bool wide, bool xindep) {
  const uint32_t op = p.w & 0xFFFFu;
  const uint32_t fp = __reduce_or_sync(kFull, p.mine(lane_id()) ? uint32_t(g_opregs[op]) : 0u);
  if (compact && !(fp & 0xC0u)) {
    const uint32_t id = g_cid[fp & 0x3Fu];
    if (id && __all_sync(kFull, !p.mine(lane_id()) || g_cren[id - 1][op] >= 0)) return uint8_t(id);
  }
  if (wide && !xindep && !(fp & 0x80u)) {
    const uint32_t id = g_wid[fp & 0x3Fu];
    if (id && __all_sync(kFull, !p.mine(lane_id()) || g_wren[id - 1][op] >= 0)) return uint8_t(kWideClass | id);
  }
  return wide && !(fp & 0xC0u) ? kRegClass : uint8_t(0);
}
// A-dependent pairs run bit-sliced (z80_bits.cuh): a unit is 4 A-blocks, a
// lane takes 32 consecutive values of A of one block.
constexpr unsigned long long kBitsBlocks = 4;
constexpr int kBitsWords = 88;  // planes of one ZB (A F B C D E H L M: 8 each, SP: 16)
__device__ __forceinline__ unsigned long long pair_units(unsigned long long nblocks, uint32_t keepR,
                                                         uint32_t xunit) {
  const unsigned long long xu = xunit ? xunit : kUnitBlocks;
  return (keepR & kXIndep) ? (nblocks + xu - 1) / xu : (nblocks + kBitsBlocks - 1) / kBitsBlocks;
}
constexpr int kChunksPerWarp = 16;
// The class of a pair (kClasses).
__device__ __forceinline__ int pair_class(const PairRec& pr) {
  if (pr.cmap & kWideClass) return 3;    // only set when R.wide
  if (pr.cmap == kRegClass) return 4;    // only set when R.wide
  if (pr.cmap != 0) return 2;            // only set when R.compact
  return (pr.keepR & kXIndep) ? 1 : 0;
}

// ------------------------------------------------------------------ kernels

// Warp per candidate, lane v runs the candidate on vector v (lanes 0..7
// QuickCheck, 0..31 MidCheck); the opcode is the same in every lane.
__global__ void k_pool_outputs(const uint32_t* __restrict__ insn, uint32_t n, uint32_t len,
                               uint4* __restrict__ qc, uint4* __restrict__ mid, bool by_pair) {
  const unsigned lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t c = gw; c < n; c += nw) {
    const uint32_t pw = lane < len ? insn[(size_t)c * len + lane] : 0u;
    Z80S s = vec_state(int(lane));
    run_lanes(s, pw, 0, int(len));
    uint32_t w[3];
    z_pack(s, w);
    const uint4 q = make_uint4(w[0], w[1], w[2], 0u);
    if (lane < 8) qc[by_pair ? (size_t)c * 8 + lane : (size_t)lane * n + c] = q;
    if (mid) mid[(size_t)lane * n + c] = q;
  }
}

// One warp per sequence; lane 0 runs it (arbitrary per-item opcodes would
// otherwise diverge inside the dispatch loop).
__global__ void k_exec(const uint32_t* __restrict__ in, const uint32_t* __restrict__ seqs,
                       const uint8_t* __restrict__ lens, uint32_t len, uint32_t stride, uint32_t n,
                       uint32_t* __restrict__ out) {
  const unsigned lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = gw; i < n; i += nw) {
    const uint32_t l = lens ? lens[i] : len;
    const uint32_t pw = lane < l ? seqs[(size_t)i * stride + lane] : 0u;
    Z80S s = z_unpack(in[3 * i], in[3 * i + 1], in[3 * i + 2]);
    run_lanes(s, pw, 0, int(l));
    if (lane == 0) {
      uint32_t w[3];
      z_pack(s, w);
      out[3 * i] = w[0];
      out[3 * i + 1] = w[1];
      out[3 * i + 2] = w[2];
    }
  }
}

// search.Fingerprint: 8 x {A,F,B,C,D,E,H,L,SP_hi,SP_lo}; warp per sequence,
// lane v (< 8) on test vector v.
__global__ void k_fingerprints(const uint32_t* __restrict__ seqs, uint32_t n, uint32_t len,
                               uint8_t* __restrict__ out) {
  const unsigned lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = gw; i < n; i += nw) {
    const uint32_t pw = lane < len ? seqs[(size_t)i * len + lane] : 0u;
    Z80S s = vec_state(int(lane & 7u));
    run_lanes(s, pw, 0, int(len));
    if (lane < 8) {
      uint8_t* p = out + (size_t)i * 80 + lane * 10;
      p[0] = uint8_t(s.a); p[1] = uint8_t(s.f); p[2] = uint8_t(s.b); p[3] = uint8_t(s.c);
      p[4] = uint8_t(s.d); p[5] = uint8_t(s.e); p[6] = uint8_t(s.h); p[7] = uint8_t(s.l);
      p[8] = uint8_t(s.sp >> 8); p[9] = uint8_t(s.sp);
    }
  }
}

// z80qc query semantics (cuda/z80_quickcheck.cu:666-681 over pkg/cpu
// outputs): candidate c matches when its fingerprint equals the query with
// the dead flag bits cleared in every F byte.  The query comes by value; the
// first kFpHere hits and the count go straight to page-locked host memory,
// written by the last block to end, which also clears the counters for the
// next query, so that a query is one launch and one wait.  Nearly every
// candidate is settled by its first vector (4.3 MB of the pool's 34 are read):
// bound by the launch and the wait; with the query copied in, the counter
// cleared and the results read by commands of their own it took 40 us, here
// 30 us.
__global__ void __launch_bounds__(256) k_fp_query(DevPool P, const __grid_constant__ FpQuery fp, uint32_t dead,
                                                  uint32_t* __restrict__ hits, FpCounters* __restrict__ ctr,
                                                  FpAnswer* __restrict__ answer) {
  const uint32_t keep0 = ~(dead << 8);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < P.n; base += stride) {
    const uint32_t c = base + lane_id();
    bool hit = c < P.n;
#pragma unroll 1
    for (int v = 0; v < 8 && hit; v++) {
      const uint4 q = P.qc[(size_t)v * P.n + c];
      hit = (((q.x ^ fp.w[3 * v]) & keep0) | (q.y ^ fp.w[3 * v + 1]) | ((q.z ^ fp.w[3 * v + 2]) & 0xFFFFu)) == 0;
    }
    const unsigned b = __ballot_sync(kFull, hit);
    if (!b) continue;
    uint32_t at = 0;
    if (lane_id() == 0) at = atomicAdd(&ctr->hits, (uint32_t)__popc(b));
    at = __shfl_sync(kFull, at, 0) + __popc(b & lanemask_lt());
    if (hit) {
      hits[at] = c;
      if (at < kFpHere) answer->hits[at] = c;
    }
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (atomicAdd(&ctr->done, 1u) == gridDim.x - 1u) {
    answer->count = atomicExch(&ctr->hits, 0u);
    ctr->done = 0;
  }
}

// Target side of a QuickCheck: encoded bytes, T-states and reads of the
// target (summed over its lanes), its outputs on the 8 vectors (warp-uniform
// copies) and the compared bytes of the packed words under its dead masks.
struct QCTarget {
  uint32_t tb, tts, trd, tl;
  uint32_t tw[8][3];
  uint32_t keep0, keep1;
};
__device__ __forceinline__ void qc_target(const DevTargets& T, uint32_t t, QCTarget& g) {
  const unsigned lane = lane_id();
  const uint32_t tl = target_len(T, t);
  const uint32_t pw = lane < tl ? T.insn[(size_t)t * T.stride + lane] : 0u;
  uint32_t sz = 0, ts = 0, rd = 0;
  if (lane < tl) {
    const OpInfo oi = g_ops[pw & 0xFFFFu];
    sz = oi.size;
    ts = oi.tstates;
    rd = oi.reads;
  }
#pragma unroll
  for (int off = 2; off >= 1; off >>= 1) {
    sz += __shfl_down_sync(kFull, sz, off);
    ts += __shfl_down_sync(kFull, ts, off);
    rd |= __shfl_down_sync(kFull, rd, off);
  }
  g.tl = tl;
  g.tb = __shfl_sync(kFull, sz, 0);
  g.tts = __shfl_sync(kFull, ts, 0);
  g.trd = __shfl_sync(kFull, rd, 0);
  Z80S s = vec_state(int(lane & 7u));
  run_lanes(s, pw, 0, int(tl));
  uint32_t w[3];
  z_pack(s, w);
#pragma unroll
  for (int v = 0; v < 8; v++) {
    g.tw[v][0] = __shfl_sync(kFull, w[0], v);
    g.tw[v][1] = __shfl_sync(kFull, w[1], v);
    g.tw[v][2] = __shfl_sync(kFull, w[2], v);
  }
  const uint32_t dead = target_dead(T, t) & 0xFFu;
  const uint32_t dregs = target_dead_regs(T, t) & 0x3Fu;
  g.keep0 = 0xFFu | ((~dead & 0xFFu) << 8) | ((dregs & 1u) ? 0u : 0xFF0000u) | ((dregs & 2u) ? 0u : 0xFF000000u);
  g.keep1 = ((dregs & 4u) ? 0u : 0xFFu) | ((dregs & 8u) ? 0u : 0xFF00u) | ((dregs & 16u) ? 0u : 0xFF0000u) |
            ((dregs & 32u) ? 0u : 0xFF000000u);
}

// QuickCheck of candidate c (vector-0 output q) against the target: fp
// (full equivalence; every pass in all-hits mode), mp (passes only under the
// dead masks), diff (FlagDiff | differing registers << 8 over the vectors).
__device__ __forceinline__ void qc_candidate(const DevPool& P, uint4 q, uint32_t c, const QCTarget& g,
                                             uint32_t keep2, bool all_hits, bool& fp, bool& mp, uint32_t& diff) {
  const uint32_t d0 = q.x ^ g.tw[0][0], d1 = q.y ^ g.tw[0][1], d2 = q.z ^ g.tw[0][2];
  if (((d0 & g.keep0) | (d1 & g.keep1) | (d2 & keep2)) != 0) return;
  bool full = (d0 | d1 | (d2 & keep2)) == 0;
  uint32_t fd = (d0 >> 8) & 0xFFu, rdf = reg_diff(d0, d1);
  bool ok = true;
#pragma unroll
  for (int v = 1; v < 8; v++) {
    const uint4 qv = P.qc[(size_t)v * P.n + c];
    const uint32_t e0 = qv.x ^ g.tw[v][0], e1 = qv.y ^ g.tw[v][1], e2 = qv.z ^ g.tw[v][2];
    ok = ok && (((e0 & g.keep0) | (e1 & g.keep1) | (e2 & keep2)) == 0);
    full = full && ((e0 | e1 | (e2 & keep2)) == 0);
    fd |= (e0 >> 8) & 0xFFu;
    rdf |= reg_diff(e0, e1);
  }
  if (!ok) return;
  if (all_hits) {
    fp = true;
  } else {
    fp = full;
    mp = !full;
  }
  diff = fd | (rdf << 8);
}

// Appends this warp's survivors of one 32-candidate step in enumeration
// order (collect pass) or tallies them per lane (count pass).
template <bool COLLECT>
__device__ __forceinline__ void qc_emit(const QCOut& o, bool fp, bool mp, uint32_t c, uint32_t diff, uint32_t obase,
                                        uint32_t nf_total, uint32_t& nf, uint32_t& nm, uint32_t& lf,
                                        uint32_t& lm) {
  if constexpr (!COLLECT) {
    lf += fp ? 1u : 0u;
    lm += mp ? 1u : 0u;
  } else {
    const unsigned bf = __ballot_sync(kFull, fp);
    const unsigned bm = __ballot_sync(kFull, mp);
    if (fp) {
      const uint32_t idx = obase + nf + __popc(bf & lanemask_lt());
      o.surv[idx] = c;
      o.sdiff[idx] = uint16_t(diff);
    }
    if (mp) {
      const uint32_t idx = obase + nf_total + nm + __popc(bm & lanemask_lt());
      o.surv[idx] = c;
      o.sdiff[idx] = uint16_t(diff);
    }
    nf += __popc(bf);
    nm += __popc(bm);
  }
}

// Count-pass epilogue: survivor counts and the target's metadata.
__device__ __forceinline__ void qc_count_out(const QCOut& o, uint32_t t, const QCTarget& g, uint32_t nf,
                                             uint32_t nm) {
  o.cnt_f[t] = nf;
  o.cnt_m[t] = nm;
  o.cnt_all[t] = nf + nm;
  TargetMeta m;
  m.tstates = uint16_t(g.tts);
  m.bytes = uint8_t(g.tb);
  m.len = uint8_t(g.tl);
  m.reads = uint16_t(g.trd);
  m.pad = 0;
  o.meta[t] = m;
}

template <bool COLLECT>
__global__ void __launch_bounds__(kBlock) k_qc_scan(DevTargets T, DevPool P, QCConfig cfg, QCOut o) {
  extern __shared__ uint4 smem[];
  uint4* s_q0 = smem;
  uint8_t* s_el = reinterpret_cast<uint8_t*>(smem + (cfg.use_smem ? P.n : 0));
  if (cfg.use_smem) {
    for (uint32_t i = threadIdx.x; i < P.n; i += blockDim.x) {
      s_q0[i] = P.qc[i];
      s_el[i] = uint8_t(P.size[i] | (P.prune[i] ? 0x80u : 0u));
    }
    __syncthreads();
  }
  const unsigned lane = lane_id();
  const uint32_t warps_per_block = blockDim.x >> 5;
  const uint32_t gw = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const uint32_t nw = gridDim.x * warps_per_block;
  unsigned long long my_checks = 0;

  for (uint32_t t = gw; t < T.n; t += nw) {
    uint32_t nf_total = 0, obase = 0;
    if (COLLECT) {
      nf_total = o.cnt_f[t];
      if (nf_total + o.cnt_m[t] == 0) continue;
      obase = o.base[t];
    }
    QCTarget g;
    qc_target(T, t, g);
    uint32_t nf = 0, nm = 0;
    uint32_t lf = 0, lm = 0, lc = 0;  // count pass: per-lane tallies, reduced once per target
    for (uint32_t base = 0; base < P.n; base += 32) {
      const uint32_t c = base + lane;
      bool el = false;
      if (c < P.n) {
        uint32_t e = cfg.use_smem ? s_el[c] : (P.size[c] | (P.prune[c] ? 0x80u : 0u));
        el = (e & 0x7Fu) < g.tb && !(e & 0x80u);
      }
      bool fp = false, mp = false;
      uint32_t diff = 0;
      if (el) qc_candidate(P, cfg.use_smem ? s_q0[c] : P.qc[c], c, g, cfg.w2mask, cfg.all_hits != 0, fp, mp, diff);
      if constexpr (!COLLECT) lc += el ? 1u : 0u;
      qc_emit<COLLECT>(o, fp, mp, c, diff, obase, nf_total, nf, nm, lf, lm);
    }
    if constexpr (!COLLECT) {
      nf = __reduce_add_sync(kFull, lf);
      nm = __reduce_add_sync(kFull, lm);
      const uint32_t nc = __reduce_add_sync(kFull, lc);
      if (lane == 0) {
        my_checks += nc;
        qc_count_out(o, t, g, nf, nm);
      }
    }
  }
  if (!COLLECT && lane == 0 && my_checks) atomicAdd(o.checks, my_checks);
}

// Allocates w consecutive pair slots for this thread (one atomic per warp;
// every lane of the warp takes part); returns the first slot.
__device__ __forceinline__ uint32_t alloc_pairs(uint32_t* counter, uint32_t w) {
  const unsigned lane = lane_id();
  uint32_t incl = w;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, off);
    if (lane >= unsigned(off)) incl += v;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  uint32_t base = 0;
  if (lane == 31 && total) base = atomicAdd(counter, total);
  base = __shfl_sync(kFull, base, 31);
  return base + incl - w;
}

// Puts the window of w survivors at sbase of lane (t, kind) into the pair
// slots from p0: who the pairs are.  What their sweeps take is worked out by
// k_pair_plan, a warp per pair (a window is up to 64 pairs and a plan some
// microseconds: planned here, one thread would plan a window's pairs one
// after the other).
__device__ __forceinline__ void put_window(const RoundBuf& R, uint32_t p0, uint32_t w, uint32_t t, uint32_t kind,
                                           const uint32_t* __restrict__ surv, unsigned long long sbase) {
  for (uint32_t j = 0; j < w; j++) {
    const uint32_t p = p0 + j;
    PairRec pr{};
    pr.target = t;
    pr.cand = surv[sbase + j];
    pr.keepR = kind ? 0x80u : 0u;
    R.pairs[p] = pr;
    R.pair_src[p] = uint32_t(sbase + j);
    R.rejected[p] = 0;
    R.wlen[p] = j == 0 ? uint8_t(w) : uint8_t(0);
    if (R.wend) {
      R.wend[p] = p0 + w;
      R.cdone[p] = 0;
    }
  }
}

// Lane 0, after a warp's chunk of pair p ran to its end without a mismatch:
// counts the chunk; the warp that counts the last one of a pair that still
// stands (its whole sweep passed) cancels the pairs after it in its survivor
// window (rejected 0 -> 2): the first passing pair of a window wins, so
// their sweeps cannot change the result.  A chunk with a mismatch rejects
// the pair and is not counted, so a rejected pair never reaches its count.
// nch = the pair's chunks.
__device__ __forceinline__ void chunk_passed(uint32_t* rejected, const uint32_t* wend, uint32_t* cdone, uint32_t p,
                                          uint32_t nch) {
  __threadfence();
  const uint32_t before = atomicAdd(&cdone[p], 1u);
  if (before + 1u != nch) return;
  __threadfence();
  if (atomicAdd(&rejected[p], 0u) != 0u) return;
  // windows hold at most 64 pairs; an unrolled, guarded run keeps a loop
  // out of the sweep kernels' loop nest (which made them spill)
  const uint32_t e = wend[p];
#pragma unroll
  for (uint32_t i = 1; i < 64; i++)
    if (p + i < e) atomicCAS(&rejected[p + i], 0u, 2u);
}

// One round's pairs: each unresolved (target, kind) lane puts its window of
// next survivors into the round (pairs past the buffer's capacity wait for
// the next round).  PAIR: the length-2 pass, whose survivors are in slots.
// A thread looks at four lanes (one 16-byte load of their progress; mostly
// they are resolved), a block takes the slots for all of its windows with one
// atomic.  With a lane per thread and an atomic per warp the first round of
// 9.8M targets was bound by some 460,000 atomics on one address, the later
// ones by 65 dependent loads in a row: 226 and 82 us, now 116 and
// 44.
constexpr uint32_t kBuildLanes = 4;
template <bool PAIR>
__global__ void __launch_bounds__(256) k_round_build(const RoundArgs* __restrict__ A) {
  __shared__ uint32_t sum[2][8];  // per warp; two sets, as a block without windows passes one barrier only
  __shared__ uint32_t at;
  const RoundBuf& R = A->R;
  const uint32_t lanes = 2u * A->T.n, warp = threadIdx.x >> 5;
  const unsigned lane = lane_id();
  const uint32_t step = kBuildLanes * blockDim.x;
  uint32_t set = 0;
  for (uint32_t base = blockIdx.x * step; base < lanes; base += gridDim.x * step, set ^= 1u) {
    const uint32_t i0 = base + kBuildLanes * threadIdx.x;
    uint32_t nx[kBuildLanes];
    if (i0 + kBuildLanes <= lanes) {
      const uint4 v = *reinterpret_cast<const uint4*>(A->L.next + i0);
      nx[0] = v.x, nx[1] = v.y, nx[2] = v.z, nx[3] = v.w;
    } else {
#pragma unroll
      for (uint32_t k = 0; k < kBuildLanes; k++) nx[k] = i0 + k < lanes ? A->L.next[i0 + k] : kResolved;
    }
    uint32_t w[kBuildLanes], all = 0;
    unsigned long long sbase[kBuildLanes];
#pragma unroll
    for (uint32_t k = 0; k < kBuildLanes; k++) {
      const uint32_t idx = i0 + k, t = idx >> 1, kind = idx & 1u;
      w[k] = 0;
      sbase[k] = 0;
      if (nx[k] & kResolved) continue;
      uint32_t cnt;
      if constexpr (PAIR) {
        cnt = A->ps.cnt[idx];
        sbase[k] = (unsigned long long)idx * kSlots2 + nx[k];
      } else {
        const uint32_t cf = A->q.cnt_f[t];
        cnt = kind ? A->q.cnt_m[t] : cf;
        sbase[k] = cnt ? A->q.base[t] + (kind ? cf : 0u) + nx[k] : 0u;
      }
      if (nx[k] < cnt) w[k] = min(1u << A->L.spec[idx], cnt - nx[k]);
      else A->L.next[idx] = nx[k] | kResolved;  // no survivor (left): resolved without a winner
      all += w[k];
    }
    uint32_t incl = all;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, incl, off);
      if (lane >= unsigned(off)) incl += v;
    }
    if (lane == 31) sum[set][warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; k++) {
      if (k < warp) before += sum[set][k];
      total += sum[set][k];
    }
    if (total == 0) continue;
    if (threadIdx.x == 0) at = atomicAdd(&R.ctl->npairs, total);
    __syncthreads();
    uint32_t p0 = at + before + incl - all;
#pragma unroll
    for (uint32_t k = 0; k < kBuildLanes; k++) {
      const uint32_t idx = i0 + k;
      if (!w[k]) continue;
      const uint32_t fit = p0 >= R.cap ? 0u : min(w[k], R.cap - p0);
      if (fit < w[k]) R.ctl->active = 1;
      put_window(R, p0, fit, idx >> 1, idx & 1u, PAIR ? A->ps.surv : A->q.surv, sbase[k]);
      p0 += w[k];
    }
  }
}

// pkg/gpu semantics: one pair per MidCheck survivor (all survivors when
// midpass is null) of [lo, hi).
__global__ void k_pairs_from_survivors(QCOut q, const uint8_t* __restrict__ midpass, uint32_t lo, uint32_t hi,
                                       const uint32_t* __restrict__ surv_target, RoundBuf R) {
  const uint32_t i = lo + blockIdx.x * blockDim.x + threadIdx.x;
  const bool have = i < hi && (!midpass || midpass[i]);
  if (!__any_sync(kFull, have)) return;
  const uint32_t p = alloc_pairs(&R.ctl->npairs, have ? 1u : 0u);
  if (!have || p >= R.cap) return;
  PairRec pr{};
  pr.target = surv_target[i];
  pr.cand = q.surv[i];
  pr.keepR = 0x80u;  // compared under the target's dead masks
  R.pairs[p] = pr;
  R.pair_src[p] = i;
  R.rejected[p] = 0;
}
// Independent pairs (i, i) of a target batch and a pool of as many.
__global__ void k_pairs_identity(uint32_t n, RoundBuf R) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) R.ctl->npairs = n;
  if (i >= n) return;
  PairRec pr{};
  pr.target = i;
  pr.cand = i;
  pr.keepR = 0x80u;
  R.pairs[i] = pr;
  R.rejected[i] = 0;
}

// K = states per lane per dispatch ("vectors per lane").  One warp
// iteration covers 32*K values of A; an A-block (256 states) takes 8/K
// iterations.
// Initial register values of A-block ab (everything but A and F's carry),
// decoded field by field from the sweep shape: the same values as
// bdec_state, in a form that keeps the bit-sliced A-independent unit within
// its registers.  Block index fields fastest first: SP (reduced sweeps), the
// swept registers from the last to the first, carry.  UNIFORM selects the
// __constant__ tables (the index is the same in every lane) or their global
// copies (lane-dependent index).
template <bool UNIFORM>
__device__ __forceinline__ void decode_block(unsigned long long ab, bool spw, bool reduced, int nx, int fw,
                                             const int (&slot)[7], Z80S& init) {
  unsigned long long rest = ab;
  uint32_t sp = 0;
  if (spw) {
    sp = UNIFORM ? c_repsp[uint32_t(rest & 15ull)] : g_repsp[uint32_t(rest & 15ull)];
    rest >>= 4;
  }
  uint32_t fieldv[7];
#pragma unroll
  for (int f = 6; f >= 0; f--) {
    fieldv[f] = 0;
    if (f < nx) {
      const uint32_t x = uint32_t(rest) & (reduced ? 31u : 255u);
      fieldv[f] = reduced ? (UNIFORM ? c_rep[x] : g_rep[x]) : x;
      rest >>= fw;
    }
  }
  uint32_t rv[7];
#pragma unroll
  for (int r = 0; r < 7; r++) {
    uint32_t v = 0;
#pragma unroll
    for (int f = 0; f < 7; f++)
      if (slot[r] == f) v = fieldv[f];
    rv[r] = v;
  }
  init.a = 0;
  init.f = uint32_t(rest & 1ull);
  init.b = rv[0]; init.c = rv[1]; init.d = rv[2]; init.e = rv[3];
  init.h = rv[4]; init.l = rv[5]; init.m = rv[6];
  init.sp = sp;
}

// Runs the candidate then the target from K initial states (init(q, x)
// writes state q) and reports whether any compared output differs (only
// states with valid[q]).
template <int K, class Init>
__device__ __forceinline__ bool run_compare(const Init& init, const bool (&valid)[K], uint32_t pw, int tl, int cl,
                                            uint32_t keep0, uint32_t keep1) {
  Z80S X[K];
  uint32_t P0[K], P1[K], P2[K];
  const int nsteps = tl + cl;
  // one dispatch site: the candidate runs first; its output is packed into
  // three words per state, the registers are re-initialised and the target
  // runs on them
#pragma unroll 1
  for (int st = -1; st < nsteps; st++) {
    if (st == -1 || st == cl) {
      if (st == cl) {
#pragma unroll
        for (int q = 0; q < K; q++) {
          P0[q] = X[q].a | (X[q].f << 8) | (X[q].b << 16) | (X[q].c << 24);
          P1[q] = X[q].d | (X[q].e << 8) | (X[q].h << 16) | (X[q].l << 24);
          P2[q] = X[q].sp | (X[q].m << 16);
        }
      }
#pragma unroll
      for (int q = 0; q < K; q++) init(q, X[q]);
      if (st == -1) continue;
    }
    // lanes tl.. hold the candidate, lanes 0.. the target
    const int src = st < cl ? tl + st : st - cl;
    const uint32_t w = __shfl_sync(kFull, pw, src);
    z_stepK<K>(X, w & 0xFFFFu, w >> 16);
  }
  bool bad = false;
#pragma unroll
  for (int q = 0; q < K; q++) {
    const uint32_t d0 = (X[q].a | (X[q].f << 8) | (X[q].b << 16) | (X[q].c << 24)) ^ P0[q];
    const uint32_t d1 = (X[q].d | (X[q].e << 8) | (X[q].h << 16) | (X[q].l << 24)) ^ P1[q];
    const uint32_t d2 = (X[q].sp | (X[q].m << 16)) ^ P2[q];
    bad = bad || (valid[q] && ((d0 & keep0) | (d1 & keep1) | d2) != 0);
  }
  return bad;
}

// Runs both programs of a pair on 512 states of its sweep -- every value of A
// twice, each with a block of its own spread over the sweep -- and tells
// whether one of them differs.  Warp-wide, the same pair in every lane.
__device__ __forceinline__ bool probe_pair(const PairWords& words, unsigned long long nblocks, uint32_t reads,
                                           uint32_t sweepf, uint32_t keepF, uint32_t keepR) {
  const unsigned lane = lane_id();
  const uint32_t ext = reads & (kRegB | kRegC | kRegD | kRegE | kRegH | kRegL | kRegM);
  const bool spw = (reads & kRegSP) != 0;
  const int nx = __popc(ext);
  const bool reduced = spw || nx > 2 || (sweepf & 0x80u) != 0;
  int slot[7];
  {
    int k = 0;
    const uint32_t bits[7] = {kRegB, kRegC, kRegD, kRegE, kRegH, kRegL, kRegM};
#pragma unroll
    for (int r = 0; r < 7; r++) slot[r] = (ext & bits[r]) ? k++ : -1;
  }
  const BDec bd = bdec_make(spw, reduced, nx, reduced ? 5 : 8, slot);
  const uint32_t keep0 = 0xFFu | (keepF << 8) | ((keepR & 1u) ? 0xFF0000u : 0u) | ((keepR & 2u) ? 0xFF000000u : 0u);
  const uint32_t keep1 = ((keepR & 4u) ? 0xFFu : 0u) | ((keepR & 8u) ? 0xFF00u : 0u) |
                         ((keepR & 16u) ? 0xFF0000u : 0u) | ((keepR & 32u) ? 0xFF000000u : 0u);
  bool bad = false;
#pragma unroll 1
  for (uint32_t i = 0; i < 8u && !__any_sync(kFull, bad); i++) {
    uint32_t W[2][3];
    const bool valid[2] = {true, true};
#pragma unroll
    for (uint32_t q = 0; q < 2; q++) {
      const uint32_t n = (i * 2u + q) * 32u + lane;  // 0..511
      unsigned long long h = (n + 1ull) * 0x9E3779B97F4A7C15ull;
      h ^= h >> 29;
      h *= 0xBF58476D1CE4E5B9ull;
      h ^= h >> 32;
      Z80S x = bdec_state(bd, h & (nblocks - 1ull), g_rep, g_repsp);  // nblocks is a power of two
      x.a = (n * 37u) & 0xFFu;
      z_pack(x, W[q]);
    }
    auto init = [&](int q, Z80S& x) { x = z_unpack(W[q][0], W[q][1], W[q][2]); };
    bad = run_compare<2>(init, valid, words.w, int(words.tl), int(words.cl), keep0, keep1);
  }
  return __any_sync(kFull, bad);
}

// Plans the round's pairs (z80_plan.cuh), a warp each: compared outputs,
// swept fields, class and chunks.  A pair that its programs prove equivalent
// gets no chunk and keeps its zero flag; the pairs after it in its window
// cannot win and are cancelled.  A pair whose sweep takes more than one chunk
// is probed first: nearly all long sweeps belong to pairs that passed the
// eight QuickCheck vectors and are no equivalences, and such a sweep draws
// every resident warp into one pair before its first mismatch is seen, one
// pair after the other.  The chunks of a pair go to its class's list
// (RoundCtl::alloc), one atomic each.
// Bound by latency (some ten dependent loads and a few hundred instructions a
// pair).  A lane per pair, each running plan_pair on arrays in local memory,
// took 26 us a round however few its pairs (200 uneven targets: 1.75 ms a
// search, 0.95 ms with this and k_qc_long; the 851,000 pairs of the 9.8M
// length-2 targets' rounds pay for it: 0.98 ms of a 5.1 ms step under ncu, and
// at 64 registers a thread it spills, 370 bytes stored and 516 loaded, most of
// them in the probe that few pairs run); in the round build, a
// window's up to 64 pairs in one thread, 0.3 ms a round.  The probe and the polls between units:
// 40,009 uneven targets evaluate 4.5e8 states where it was 1.6e10 (84 -> 43 ms
// of sweeps), the 9.4M length-2 targets 2.7e8 where it was 1.3e9 (3.2 ->
// 2.05 ms).
__global__ void __launch_bounds__(128, 8) k_pair_plan(const RoundArgs* __restrict__ A) {
  const RoundBuf& R = A->R;
  const DevTargets& T = A->T;
  const DevPool& P = A->P;
  const uint32_t np = min(R.ctl->npairs, R.cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) R.ctl->nscan = 0;  // the rescan before this round has read it
  const unsigned lane = lane_id();
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  unsigned long long covered = 0;  // reference states that proofs and probes answer for
  uint32_t probes = 0;
  for (uint32_t p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); p < np; p += nw) {
    PairRec pr = R.pairs[p];
    const uint32_t t = pr.target, c = pr.cand;
    const bool masked = (pr.keepR & 0x80u) != 0;
    const PairWords words = pair_words(T, t, P, c);
    uint32_t reads;
    if (P.reads) reads = A->q.meta[t].reads | P.reads[c];
    else reads = __reduce_or_sync(kFull, words.mine(lane) ? uint32_t(g_ops[words.w & 0xFFFFu].reads) : 0u);
    pr.keepF = masked ? uint8_t(~target_dead(T, t)) : uint8_t(0xFFu);
    pr.keepR = masked ? uint8_t((~target_dead_regs(T, t) & 0x3Fu) | 0x80u) : uint8_t(0x3Fu);
    const PairPlan pl = plan_pair_warp(lane, g_flow, words, reads, pr.keepF, pr.keepR);
    pr.reads = pl.reads;
    pr.sweepf = pl.sweepf;
    pr.nblocks = pl.nblocks;
    pr.cmap = 0;
    if (pl.proven) {
      pr.nblocks = 0;  // no chunk in any class
      covered += 256ull * plan_blocks(reads, false);
      if (R.wend)
        for (uint32_t i = p + 1 + lane; i < R.wend[p]; i += 32) R.rejected[i] = 2;
    } else {
      if (pl.a_free || pair_xindep(words)) pr.keepR |= uint8_t(kXIndep);
      // compact classes: A-dependent pairs, and A-independent ones when
      // those are swept bit-sliced (units of kXBitsBlocks)
      const bool xind = (pr.keepR & kXIndep) != 0;
      if (!xind || R.xunit == kXBitsBlocks) pr.cmap = pair_cmap(words, R.compact != 0, R.wide != 0, xind);
      if (pair_units(pr.nblocks, pr.keepR, R.xunit) > R.chunk_blocks) {
        probes++;
        if (probe_pair(words, pr.nblocks, pr.reads, pr.sweepf, pr.keepF, pr.keepR)) {
          pr.nblocks = 0;
          if (lane == 0) R.rejected[p] = 1;
        }
      }
    }
    if (lane == 0) {
      R.pairs[p] = pr;
      const uint32_t ch =
          pr.nblocks ? chunk_count(pair_units(pr.nblocks, pr.keepR, R.xunit), R.chunk_blocks, R.max_chunks) : 0u;
      if (ch) {
        const int cls = pair_class(pr);
        const unsigned long long at = atomicAdd(&R.ctl->alloc[cls], 1ull << kChunkBits | ch);
        R.cbase[cls][at >> kChunkBits] = at & kChunkMask;
        R.cpair[cls][at >> kChunkBits] = p;
      }
    }
  }
  if (lane == 0 && (covered || probes)) {
    atomicAdd(R.states, covered + 512ull * probes);
    if (probes) atomicAdd(R.states + 1, 512ull * probes);
  }
}

// Planes of the 32 states A = a0 .. a0+31 (a0 a multiple of 32) with the
// other registers of x.
__device__ __forceinline__ void zb_init(ZB& z, const Z80S& x, uint32_t a0) {
  z.a[0] = 0xAAAAAAAAu;
  z.a[1] = 0xCCCCCCCCu;
  z.a[2] = 0xF0F0F0F0u;
  z.a[3] = 0xFF00FF00u;
  z.a[4] = 0xFFFF0000u;
  z.a[5] = (a0 & 32u) ? kZBOnes : 0u;
  z.a[6] = (a0 & 64u) ? kZBOnes : 0u;
  z.a[7] = (a0 & 128u) ? kZBOnes : 0u;
  zb_set8(z.f, x.f);
  zb_set8(z.b, x.b);
  zb_set8(z.c, x.c);
  zb_set8(z.d, x.d);
  zb_set8(z.e, x.e);
  zb_set8(z.h, x.h);
  zb_set8(z.l, x.l);
  zb_set8(z.m, x.m);
#pragma unroll
  for (int i = 0; i < 16; i++) z.sp[i] = ((x.sp >> i) & 1u) ? kZBOnes : 0u;
}
// Saves / compares the planes (s: this lane's column, stride 32 words).
__device__ __forceinline__ void zb_save(const ZB& z, uint32_t* s) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s[(0 + i) * 32] = z.a[i];
    s[(8 + i) * 32] = z.f[i];
    s[(16 + i) * 32] = z.b[i];
    s[(24 + i) * 32] = z.c[i];
    s[(32 + i) * 32] = z.d[i];
    s[(40 + i) * 32] = z.e[i];
    s[(48 + i) * 32] = z.h[i];
    s[(56 + i) * 32] = z.l[i];
    s[(64 + i) * 32] = z.m[i];
  }
#pragma unroll
  for (int i = 0; i < 16; i++) s[(72 + i) * 32] = z.sp[i];
}
__device__ __forceinline__ uint32_t zb_diff(const ZB& z, const uint32_t* s, uint32_t keepF, uint32_t keepR) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    d |= z.a[i] ^ s[(0 + i) * 32];
    if ((keepF >> i) & 1u) d |= z.f[i] ^ s[(8 + i) * 32];
    if (keepR & 1u) d |= z.b[i] ^ s[(16 + i) * 32];
    if (keepR & 2u) d |= z.c[i] ^ s[(24 + i) * 32];
    if (keepR & 4u) d |= z.d[i] ^ s[(32 + i) * 32];
    if (keepR & 8u) d |= z.e[i] ^ s[(40 + i) * 32];
    if (keepR & 16u) d |= z.h[i] ^ s[(48 + i) * 32];
    if (keepR & 32u) d |= z.l[i] ^ s[(56 + i) * 32];
    d |= z.m[i] ^ s[(64 + i) * 32];
  }
#pragma unroll
  for (int i = 0; i < 16; i++) d |= z.sp[i] ^ s[(72 + i) * 32];
  return d;
}
// One unit (4 A-blocks) of an A-dependent sweep, bit-sliced: lane l takes
// block unit*4 + l/8 and A = (l%8)*32 .. +31; the candidate's outputs wait in
// shared memory while the target runs.  One dispatch site for both programs.
__device__ __forceinline__ bool bits_unit(unsigned long long u, unsigned long long nblocks, const BDec& bd,
                                          uint32_t pw, int tl, int cl, uint32_t keepF, uint32_t keepR, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long blk = u * kBitsBlocks + (lane >> 3);
  const bool valid = blk < nblocks;
  const Z80S x = bdec_state(bd, valid ? blk : u * kBitsBlocks, g_rep, g_repsp);
  const uint32_t a0 = (lane & 7u) * 32u;
  ZB z;
#pragma unroll 1
  for (int st = -1; st < tl + cl; st++) {
    if (st == -1 || st == cl) {
      if (st == cl) zb_save(z, sm);
      zb_init(z, x, a0);
      if (st == -1) continue;
    }
    const int src = st < cl ? tl + st : st - cl;
    const uint32_t w = __shfl_sync(kFull, pw, src);
    zb_step(z, w & 0xFFFFu, w >> 16);
  }
  return valid && zb_diff(z, sm, keepF, keepR) != 0u;
}

// One unit of a compact sweep: the layout of bits_unit (lane l: block 4u +
// l/8, A = 32(l % 8) .. +31) on the compact state (A, F, B, C; ZB4).  The
// pair's programs arrive renamed onto B and C; o0 / o1 are the original
// registers (0..5 = B..L) that B and C stand for, or -1 where none does.
// Only A, F (under keepF) and those registers (under keepR) can differ.
constexpr int kCompactWords = 32;  // planes saved per lane: A, F, B, C
__device__ __forceinline__ bool cbits_unit(unsigned long long u, unsigned long long nblocks, const CDec& dec,
                                           uint32_t pw, int tl, int cl, uint32_t keepF, uint32_t keepR, int o0, int o1,
                                           uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long blk = u * kBitsBlocks + (lane >> 3);
  const bool valid = blk < nblocks;
  uint32_t vb, vc, carry;
  cdec_vals(dec, valid ? blk : u * kBitsBlocks, vb, vc, carry);
  const uint32_t a0 = (lane & 7u) * 32u;
  ZB4 z;
  auto init = [&]() {
    z.a[0] = 0xAAAAAAAAu;
    z.a[1] = 0xCCCCCCCCu;
    z.a[2] = 0xF0F0F0F0u;
    z.a[3] = 0xFF00FF00u;
    z.a[4] = 0xFFFF0000u;
    z.a[5] = (a0 & 32u) ? kZBOnes : 0u;
    z.a[6] = (a0 & 64u) ? kZBOnes : 0u;
    z.a[7] = (a0 & 128u) ? kZBOnes : 0u;
    zb_set8(z.f, carry);
    zb_set8(z.b, vb);
    zb_set8(z.c, vc);
  };
  init();
#pragma unroll 1
  for (int st = 0; st < tl + cl; st++) {
    if (st == cl) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        sm[(0 + i) * 32] = z.a[i];
        sm[(8 + i) * 32] = z.f[i];
        sm[(16 + i) * 32] = z.b[i];
        sm[(24 + i) * 32] = z.c[i];
      }
      init();
    }
    const int src = st < cl ? tl + st : st - cl;
    const uint32_t w = __shfl_sync(kFull, pw, src);
    zb4_step(z, w & 0xFFFFu, w >> 16);
  }
  const bool cmp_b = o0 >= 0 && ((keepR >> o0) & 1u), cmp_c = o1 >= 0 && ((keepR >> o1) & 1u);
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    d |= z.a[i] ^ sm[(0 + i) * 32];
    if ((keepF >> i) & 1u) d |= z.f[i] ^ sm[(8 + i) * 32];
    if (cmp_b) d |= z.b[i] ^ sm[(16 + i) * 32];
    if (cmp_c) d |= z.c[i] ^ sm[(24 + i) * 32];
  }
  return valid && d != 0u;
}

// A-independent sweeps, bit-sliced: lane l of a unit takes the 32 A-blocks
// u*1024 + 32l .. +31 as one state word (block j in bit j), first at A = 0,
// then at A = 1 (two values decide these pairs).  In an aligned group of 32
// blocks only the low 5 bits of the block index change, and they move one
// thing: the last swept register's low 5 bits (full sweep), its 32
// representative values (reduced sweep), SP's 16 representatives and one bit
// of the next field (SP sweep), or the carry (no extra register).
__device__ __forceinline__ void zb_set_reg(ZB& z, int r, const uint32_t (&pl)[8]) {
  switch (r) {
    case 0: zb_copy8(z.b, pl); break;
    case 1: zb_copy8(z.c, pl); break;
    case 2: zb_copy8(z.d, pl); break;
    case 3: zb_copy8(z.e, pl); break;
    case 4: zb_copy8(z.h, pl); break;
    case 5: zb_copy8(z.l, pl); break;
    case 6: zb_copy8(z.m, pl); break;
    default: break;
  }
}
__device__ __forceinline__ bool xbits_unit(unsigned long long u, unsigned long long nblocks, bool spw, bool reduced,
                                           int nx, int fw, const int (&slot)[7], int rlast, uint32_t pw, int tl,
                                           int cl, uint32_t keepF, uint32_t keepR, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long g0 = u * kXBitsBlocks + (unsigned long long)lane * 32ull;
  const uint32_t valid = g0 >= nblocks ? 0u
                         : (nblocks - g0 >= 32ull ? 0xFFFFFFFFu : ((1u << uint32_t(nblocks - g0)) - 1u));
  Z80S x;
  decode_block<false>(g0 < nblocks ? g0 : 0ull, spw, reduced, nx, fw, slot, x);
  // planes of what the low 5 bits of the block index move
  uint32_t vp[8], spp[16];
  uint32_t fp0 = 0u;
#pragma unroll
  for (int i = 0; i < 16; i++) spp[i] = 0u;
  if (spw) {
    // SP: state j takes representative j mod 16; bit 4: the last field's x
    // (even x0 in states 0-15, x0 + 1 in 16-31) or, with no field, the carry
#pragma unroll
    for (int i = 0; i < 16; i++) spp[i] = __ballot_sync(kFull, (g_repsp[lane & 15u] >> i) & 1u);
    const uint32_t x0 = uint32_t(g0 >> 4) & 31u;
    const uint32_t lo = g_rep[x0], hi = g_rep[(x0 + 1u) & 31u];
#pragma unroll
    for (int i = 0; i < 8; i++)
      vp[i] = (((lo >> i) & 1u) ? 0x0000FFFFu : 0u) | (((hi >> i) & 1u) ? 0xFFFF0000u : 0u);
    fp0 = 0xFFFF0000u;
  } else if (reduced) {
    // the last field's 32 representatives, state j = representative j
#pragma unroll
    for (int i = 0; i < 8; i++) vp[i] = __ballot_sync(kFull, (g_rep[lane] >> i) & 1u);
    fp0 = 0xAAAAAAAAu;  // every swept field left out: the carry is bit 0
  } else {
    // full sweep: the last field's low 5 bits count the states, the rest is
    // the group's value; with no extra register the carry is bit 0
    uint32_t v = 0u;
    switch (rlast) {
      case 0: v = x.b; break;
      case 1: v = x.c; break;
      case 2: v = x.d; break;
      case 3: v = x.e; break;
      case 4: v = x.h; break;
      case 5: v = x.l; break;
      case 6: v = x.m; break;
      default: break;
    }
    vp[0] = 0xAAAAAAAAu;
    vp[1] = 0xCCCCCCCCu;
    vp[2] = 0xF0F0F0F0u;
    vp[3] = 0xFF00FF00u;
    vp[4] = 0xFFFF0000u;
#pragma unroll
    for (int i = 5; i < 8; i++) vp[i] = ((v >> i) & 1u) ? kZBOnes : 0u;
    fp0 = 0xAAAAAAAAu;
  }
  ZB z;
  bool bad = false;
#pragma unroll 1
  for (uint32_t abit = 0; abit < 2u; abit++) {
    auto init = [&]() {
      zb_set8(z.a, abit);
      zb_set8(z.f, x.f);
      zb_set8(z.b, x.b);
      zb_set8(z.c, x.c);
      zb_set8(z.d, x.d);
      zb_set8(z.e, x.e);
      zb_set8(z.h, x.h);
      zb_set8(z.l, x.l);
      zb_set8(z.m, x.m);
#pragma unroll
      for (int i = 0; i < 16; i++) z.sp[i] = spw ? spp[i] : (((x.sp >> i) & 1u) ? kZBOnes : 0u);
      if (nx >= 1) zb_set_reg(z, rlast, vp);
      else z.f[0] = fp0;
    };
    init();
#pragma unroll 1
    for (int st = 0; st < tl + cl; st++) {
      if (st == cl) {
        zb_save(z, sm);
        init();
      }
      const int src = st < cl ? tl + st : st - cl;
      const uint32_t w = __shfl_sync(kFull, pw, src);
      zb_step(z, w & 0xFFFFu, w >> 16);
    }
    bad = bad || (zb_diff(z, sm, keepF, keepR) & valid) != 0u;
  }
  return bad;
}

// One unit of a compact A-independent sweep: xbits_unit's layout (lane l:
// the 32 A-blocks u*1024 + 32l .. +31 as one state word, at A = 0 then
// A = 1) on the A/F/B/C state with renamed programs.  A compact pair reads
// neither SP nor more than two registers, so its sweep is a full one over
// at most two fields, and the field the low 5 block bits move is the last
// swept register, now B (o0) or C (o1), or with no swept register the carry.
__device__ __forceinline__ bool cxbits_unit(unsigned long long u, unsigned long long nblocks, int nx, const CDec& dec,
                                            int rlast, uint32_t pw, int tl, int cl, uint32_t keepF, uint32_t keepR,
                                            int o0, int o1, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long g0 = u * kXBitsBlocks + (unsigned long long)lane * 32ull;
  const uint32_t valid = g0 >= nblocks ? 0u
                         : (nblocks - g0 >= 32ull ? 0xFFFFFFFFu : ((1u << uint32_t(nblocks - g0)) - 1u));
  uint32_t vb, vc, carry;
  cdec_vals(dec, g0 < nblocks ? g0 : 0ull, vb, vc, carry);
  // the moving field's planes: state j has j in its low 5 bits, the group's
  // value above them
  const uint32_t v = rlast == o0 ? vb : vc;
  uint32_t vp[8];
  vp[0] = 0xAAAAAAAAu;
  vp[1] = 0xCCCCCCCCu;
  vp[2] = 0xF0F0F0F0u;
  vp[3] = 0xFF00FF00u;
  vp[4] = 0xFFFF0000u;
#pragma unroll
  for (int i = 5; i < 8; i++) vp[i] = ((v >> i) & 1u) ? kZBOnes : 0u;
  ZB4 z;
  bool bad = false;
#pragma unroll 1
  for (uint32_t abit = 0; abit < 2u; abit++) {
    auto init = [&]() {
      zb_set8(z.a, abit);
      zb_set8(z.f, carry);
      zb_set8(z.b, vb);
      zb_set8(z.c, vc);
      if (nx == 0) z.f[0] = 0xAAAAAAAAu;
      else if (rlast == o0) zb_copy8(z.b, vp);
      else zb_copy8(z.c, vp);
    };
    init();
#pragma unroll 1
    for (int st = 0; st < tl + cl; st++) {
      if (st == cl) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          sm[(0 + i) * 32] = z.a[i];
          sm[(8 + i) * 32] = z.f[i];
          sm[(16 + i) * 32] = z.b[i];
          sm[(24 + i) * 32] = z.c[i];
        }
        init();
      }
      const int src = st < cl ? tl + st : st - cl;
      const uint32_t w = __shfl_sync(kFull, pw, src);
      zb4_step(z, w & 0xFFFFu, w >> 16);
    }
    const bool cmp_b = o0 >= 0 && ((keepR >> o0) & 1u), cmp_c = o1 >= 0 && ((keepR >> o1) & 1u);
    uint32_t d = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      d |= z.a[i] ^ sm[(0 + i) * 32];
      if ((keepF >> i) & 1u) d |= z.f[i] ^ sm[(8 + i) * 32];
      if (cmp_b) d |= z.b[i] ^ sm[(16 + i) * 32];
      if (cmp_c) d |= z.c[i] ^ sm[(24 + i) * 32];
    }
    bad = bad || (d & valid) != 0u;
  }
  return bad;
}

// Wide compact sweeps (A-dependent pairs): the layout of bits_unit on the
// wide state (A, F, B, C, H, L, M; ZBW) with renamed programs.  Fields 0..3 are
// B, C, H, L (standing for the registers the pair's set puts there), field
// 4 is M; cmp bit s: field s is compared (it stands for a register under
// keepR).  A and M are always compared, F under keepF.
constexpr int kWideWords = 56;  // planes saved per lane
__device__ __forceinline__ void zbw_init(ZBW& z, const uint32_t (&v)[5], uint32_t carry) {
  zb_set8(z.f, carry);
  zb_set8(z.b, v[0]);
  zb_set8(z.c, v[1]);
  zb_set8(z.h, v[2]);
  zb_set8(z.l, v[3]);
  zb_set8(z.m, v[4]);
}
__device__ __forceinline__ void zbw_save(const ZBW& z, uint32_t* s) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s[(0 + i) * 32] = z.a[i];
    s[(8 + i) * 32] = z.f[i];
    s[(16 + i) * 32] = z.b[i];
    s[(24 + i) * 32] = z.c[i];
    s[(32 + i) * 32] = z.h[i];
    s[(40 + i) * 32] = z.l[i];
    s[(48 + i) * 32] = z.m[i];
  }
}
__device__ __forceinline__ uint32_t zbw_diff(const ZBW& z, const uint32_t* s, uint32_t keepF, uint32_t cmp) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    d |= z.a[i] ^ s[(0 + i) * 32];
    if ((keepF >> i) & 1u) d |= z.f[i] ^ s[(8 + i) * 32];
    if (cmp & 1u) d |= z.b[i] ^ s[(16 + i) * 32];
    if (cmp & 2u) d |= z.c[i] ^ s[(24 + i) * 32];
    if (cmp & 4u) d |= z.h[i] ^ s[(32 + i) * 32];
    if (cmp & 8u) d |= z.l[i] ^ s[(40 + i) * 32];
    d |= z.m[i] ^ s[(48 + i) * 32];
  }
  return d;
}
// A-dependent: lane l takes block 4u + l/8 and A = 32(l % 8) .. +31.
__device__ __forceinline__ bool wbits_unit(unsigned long long u, unsigned long long nblocks, const WDec& dec,
                                           uint32_t pw, int tl, int cl, uint32_t keepF, uint32_t cmp, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long blk = u * kBitsBlocks + (lane >> 3);
  const bool valid = blk < nblocks;
  uint32_t v[5], carry;
  wdec_vals(dec, uint32_t(valid ? blk : u * kBitsBlocks), g_rep, v, carry);
  const uint32_t a0 = (lane & 7u) * 32u;
  ZBW z;
  auto init = [&]() {
    z.a[0] = 0xAAAAAAAAu;
    z.a[1] = 0xCCCCCCCCu;
    z.a[2] = 0xF0F0F0F0u;
    z.a[3] = 0xFF00FF00u;
    z.a[4] = 0xFFFF0000u;
    z.a[5] = (a0 & 32u) ? kZBOnes : 0u;
    z.a[6] = (a0 & 64u) ? kZBOnes : 0u;
    z.a[7] = (a0 & 128u) ? kZBOnes : 0u;
    zbw_init(z, v, carry);
  };
  init();
#pragma unroll 1
  for (int st = 0; st < tl + cl; st++) {
    if (st == cl) {
      zbw_save(z, sm);
      init();
    }
    const int src = st < cl ? tl + st : st - cl;
    const uint32_t w = __shfl_sync(kFull, pw, src);
    zbw_step(z, w & 0xFFFFu, w >> 16);
  }
  return valid && zbw_diff(z, sm, keepF, cmp) != 0u;
}
// Register-state sweeps (pairs naming neither SP nor the memory byte that
// no compact state takes): the layouts of bits_unit (A-dependent pairs) and
// xbits_unit (A-independent ones) on ZB6 (A, F, B..L), no renaming.
constexpr int kRegWords = 64;  // planes saved per lane
__device__ __forceinline__ void zb6_init(ZB6& z, const Z80S& x) {
  zb_set8(z.f, x.f);
  zb_set8(z.b, x.b);
  zb_set8(z.c, x.c);
  zb_set8(z.d, x.d);
  zb_set8(z.e, x.e);
  zb_set8(z.h, x.h);
  zb_set8(z.l, x.l);
}
__device__ __forceinline__ void zb6_save(const ZB6& z, uint32_t* s) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s[(0 + i) * 32] = z.a[i];
    s[(8 + i) * 32] = z.f[i];
    s[(16 + i) * 32] = z.b[i];
    s[(24 + i) * 32] = z.c[i];
    s[(32 + i) * 32] = z.d[i];
    s[(40 + i) * 32] = z.e[i];
    s[(48 + i) * 32] = z.h[i];
    s[(56 + i) * 32] = z.l[i];
  }
}
__device__ __forceinline__ uint32_t zb6_diff(const ZB6& z, const uint32_t* s, uint32_t keepF, uint32_t keepR) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    d |= z.a[i] ^ s[(0 + i) * 32];
    if ((keepF >> i) & 1u) d |= z.f[i] ^ s[(8 + i) * 32];
    if (keepR & 1u) d |= z.b[i] ^ s[(16 + i) * 32];
    if (keepR & 2u) d |= z.c[i] ^ s[(24 + i) * 32];
    if (keepR & 4u) d |= z.d[i] ^ s[(32 + i) * 32];
    if (keepR & 8u) d |= z.e[i] ^ s[(40 + i) * 32];
    if (keepR & 16u) d |= z.h[i] ^ s[(48 + i) * 32];
    if (keepR & 32u) d |= z.l[i] ^ s[(56 + i) * 32];
  }
  return d;
}
// A-dependent: lane l takes block 4u + l/8 and A = 32(l % 8) .. +31.
__device__ __forceinline__ bool rbits_unit(unsigned long long u, unsigned long long nblocks, const BDec& bd,
                                           uint32_t pw, int tl, int cl, uint32_t keepF, uint32_t keepR, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long blk = u * kBitsBlocks + (lane >> 3);
  const bool valid = blk < nblocks;
  const Z80S x = bdec_state(bd, valid ? blk : u * kBitsBlocks, g_rep, g_repsp);
  const uint32_t a0 = (lane & 7u) * 32u;
  ZB6 z;
  auto init = [&]() {
    z.a[0] = 0xAAAAAAAAu;
    z.a[1] = 0xCCCCCCCCu;
    z.a[2] = 0xF0F0F0F0u;
    z.a[3] = 0xFF00FF00u;
    z.a[4] = 0xFFFF0000u;
    z.a[5] = (a0 & 32u) ? kZBOnes : 0u;
    z.a[6] = (a0 & 64u) ? kZBOnes : 0u;
    z.a[7] = (a0 & 128u) ? kZBOnes : 0u;
    zb6_init(z, x);
  };
  init();
#pragma unroll 1
  for (int st = 0; st < tl + cl; st++) {
    if (st == cl) {
      zb6_save(z, sm);
      init();
    }
    const int src = st < cl ? tl + st : st - cl;
    const uint32_t w = __shfl_sync(kFull, pw, src);
    zb6_step(z, w & 0xFFFFu, w >> 16);
  }
  return valid && zb6_diff(z, sm, keepF, keepR) != 0u;
}
// A-independent: lane l takes the 32 A-blocks u*1024 + 32l .. +31 as one
// state word, at A = 0 and then A = 1; the low 5 bits of the block index
// move the last swept register rlast (its low 5 bits in a full sweep, its
// 32 representative values in a reduced one) or, with none, the carry.
__device__ __forceinline__ void zb6_set_reg(ZB6& z, int r, const uint32_t (&pl)[8]) {
  switch (r) {
    case 0: zb_copy8(z.b, pl); break;
    case 1: zb_copy8(z.c, pl); break;
    case 2: zb_copy8(z.d, pl); break;
    case 3: zb_copy8(z.e, pl); break;
    case 4: zb_copy8(z.h, pl); break;
    case 5: zb_copy8(z.l, pl); break;
    default: break;
  }
}
__device__ __forceinline__ bool rxbits_unit(unsigned long long u, unsigned long long nblocks, bool reduced, int nx,
                                            int rlast, const BDec& bd, uint32_t pw, int tl, int cl, uint32_t keepF,
                                            uint32_t keepR, uint32_t* sm) {
  const unsigned lane = lane_id();
  const unsigned long long g0 = u * kXBitsBlocks + (unsigned long long)lane * 32ull;
  const uint32_t valid = g0 >= nblocks ? 0u
                         : (nblocks - g0 >= 32ull ? 0xFFFFFFFFu : ((1u << uint32_t(nblocks - g0)) - 1u));
  const Z80S x = bdec_state(bd, g0 < nblocks ? g0 : 0ull, g_rep, g_repsp);
  uint32_t vp[8];
  if (reduced) {
#pragma unroll
    for (int i = 0; i < 8; i++) vp[i] = __ballot_sync(kFull, (g_rep[lane] >> i) & 1u);
  } else {
    uint32_t v = 0u;
    switch (rlast) {
      case 0: v = x.b; break;
      case 1: v = x.c; break;
      case 2: v = x.d; break;
      case 3: v = x.e; break;
      case 4: v = x.h; break;
      case 5: v = x.l; break;
      default: break;
    }
    vp[0] = 0xAAAAAAAAu;
    vp[1] = 0xCCCCCCCCu;
    vp[2] = 0xF0F0F0F0u;
    vp[3] = 0xFF00FF00u;
    vp[4] = 0xFFFF0000u;
#pragma unroll
    for (int i = 5; i < 8; i++) vp[i] = ((v >> i) & 1u) ? kZBOnes : 0u;
  }
  ZB6 z;
  bool bad = false;
#pragma unroll 1
  for (uint32_t abit = 0; abit < 2u; abit++) {
    auto init = [&]() {
      zb_set8(z.a, abit);
      zb6_init(z, x);
      if (nx >= 1) zb6_set_reg(z, rlast, vp);
      else z.f[0] = 0xAAAAAAAAu;
    };
    init();
#pragma unroll 1
    for (int st = 0; st < tl + cl; st++) {
      if (st == cl) {
        zb6_save(z, sm);
        init();
      }
      const int src = st < cl ? tl + st : st - cl;
      const uint32_t w = __shfl_sync(kFull, pw, src);
      zb6_step(z, w & 0xFFFFu, w >> 16);
    }
    bad = bad || (zb6_diff(z, sm, keepF, keepR) & valid) != 0u;
  }
  return bad;
}

// One unit (128 A-blocks at A = 0, 1) of an A-independent sweep, for the
// A-independent sweep kernel; kept out of line (that kernel compiles without
// register spills at every K this way).
template <int K>
__device__ __noinline__ bool xindep_unit(unsigned long long first, unsigned long long nb, const BDec bd, uint32_t pw,
                                         int tl, int cl, uint32_t keep0, uint32_t keep1) {
  const unsigned lane = lane_id();
  bool bad = false;
#pragma unroll 1
  for (uint32_t i = 0; i < 8u / K; i++) {
    uint32_t W[K][3];  // initial states, packed
    bool valid[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
      const uint32_t sl = (i * K + q) * 32u + lane;
      valid[q] = (sl >> 1) < nb;
      Z80S x = bdec_state(bd, valid[q] ? first + (sl >> 1) : first, g_rep, g_repsp);
      x.a = sl & 1u;
      z_pack(x, W[q]);
    }
    auto init = [&](int q, Z80S& x) { x = z_unpack(W[q][0], W[q][1], W[q][2]); };
    bad = run_compare<K>(init, valid, pw, tl, cl, keep0, keep1) || bad;
  }
  return bad;
}

// One kernel per pair class: CLS 0 runs the bit-sliced pairs (outputs
// depend on A), CLS 1 the A-independent ones (K states per lane per
// dispatch), CLS 2 the A-independent ones bit-sliced, CLS 3 the pairs whose
// registers fit the compact state (three blocks per SM), CLS 4 the
// A-dependent ones that fit the wide compact state (two blocks per SM), CLS
// 5 the rest that name neither SP nor the memory byte, on A, F and B..L; each class
// draws chunks from its own numbering and dispenser.  Kept apart so that
// neither path's registers weigh on the other.
// chunks_per_warp: chunks a warp takes before its block retires.
#ifndef Z80B_REG_BLOCKS
#define Z80B_REG_BLOCKS 2
#endif
// The entry of a class's chunk list whose range holds chunk k: the last e
// with cbase[e] <= k (cbase ascending from cbase[0] = 0).  Warp-wide, k the
// same in every lane: each step the 32 lanes probe 32 evenly spaced entries
// of the range left and a ballot keeps the span after the last probe that is
// <= k, so a list of n entries takes ceil(log32 n) dependent loads instead
// of log2 n.
__device__ __forceinline__ uint32_t chunk_entry(const unsigned long long* __restrict__ cbase, uint32_t n,
                                                unsigned long long k, unsigned lane) {
  uint32_t lo = 0;  // the answer lies in [lo, lo + n); cbase[lo] <= k
  while (n > 1) {
    const uint32_t step = (n + 31u) / 32u;
    const uint32_t off = lane * step;
    const bool le = off < n && cbase[lo + off] <= k;
    const unsigned b = __ballot_sync(kFull, le);  // a prefix of the lanes, lane 0 always
    const uint32_t last = 31u - uint32_t(__clz(b));
    lo += last * step;
    n = min(step, n - last * step);
  }
  return lo;
}
template <int K, int CLS>
__global__ void __launch_bounds__(kBlock, CLS == 3 ? 3 : (CLS == 4 ? 2 : (CLS == 5 ? Z80B_REG_BLOCKS : 1)))
    k_exhaustive(const __grid_constant__ SweepArgs A, int chunks_per_warp) {
  static_assert(K == 1 || K == 2 || K == 4 || K == 8, "K divides 8");
  constexpr bool XI = CLS != 0;
  constexpr int kList = CLS >= 3 ? CLS - 1 : (XI ? 1 : 0);
  const unsigned long long alloc = A.ctl->alloc[kList], total = alloc & kChunkMask;
  const uint32_t entries = uint32_t(alloc >> kChunkBits);
  const unsigned lane = lane_id();
  __shared__ unsigned long long tally[kBlock / 32][2];  // per warp: reference states covered, states evaluated
  if (lane < 2) tally[threadIdx.x >> 5][lane] = 0;
  __syncwarp();
  // At most kChunksPerWarp chunks per warp, then the block retires: the grid
  // covers all chunks, and blocks of kernels on other streams (with a higher
  // priority) get SMs as soon as blocks of a long sweep retire.
  for (int taken = 0; taken < chunks_per_warp; taken++) {
    unsigned long long k = 0;
    if (lane == 0) k = atomicAdd(&A.ctl->counter[kList], 1ull);
    k = __shfl_sync(kFull, k, 0);
    if (k >= total) break;
    const uint32_t e = chunk_entry(A.cbase[kList], entries, k, lane);
    const uint32_t p = A.cpair[kList] ? A.cpair[kList][e] : e;
    const unsigned long long c0 = A.cbase[kList][e];
    const uint32_t nch = uint32_t((e + 1 < entries ? A.cbase[kList][e + 1] : total) - c0);
    volatile uint32_t* const flag = A.rejected + p;
    // lane 0 reads the flag and the warp acts on one value, so the
    // shuffles below always see all 32 lanes
    if (__shfl_sync(kFull, lane == 0 ? *flag : 0u, 0)) {
      // The pair is settled: the dispenser jumps over what is left of its
      // chunks.  A pair of 2^20 chunks that fails in its first ones had them
      // all drawn one by one (1 ns each: 2 ms a round for two such pairs;
      // 40,009 uneven targets, 243 rounds: 196 ms of sweeps, with the jump
      // 84 ms).
      if (lane == 0) atomicMax(&A.ctl->counter[kList], c0 + nch);
      continue;
    }
    const PairRec pr = A.pairs[p];
    unsigned long long u0;
    uint32_t units;
    {
      const unsigned long long nunits = pair_units(pr.nblocks, pr.keepR, A.xunit);
      const unsigned long long upc = chunk_units(nunits, nch);
      u0 = (k - c0) * upc;
      units = u0 < nunits ? uint32_t(min(upc, nunits - u0)) : 0u;
    }

    // programs: lanes 0..tl-1 target, tl..tl+cl-1 candidate
    const uint32_t tl = A.tlens ? A.tlens[pr.target] : A.tlen, cl = A.plens ? A.plens[pr.cand] : A.plen;
    uint32_t pw = 0;
    if (lane < tl) pw = A.tinsn[(size_t)pr.target * A.tstride + lane];
    else if (lane < tl + cl) pw = A.pinsn[(size_t)pr.cand * A.pstride + (lane - tl)];

    // sweep shape (verifier.go:428-476): extra registers in B,C,D,E,H,L,M order
    const uint32_t ext = pr.reads & (kRegB | kRegC | kRegD | kRegE | kRegH | kRegL | kRegM);
    const int nx = __popc(ext);
    const bool spw = (pr.reads & kRegSP) != 0;
    const bool reduced = spw || nx > 2 || (pr.sweepf & 0x80u) != 0;
    const int fw = reduced ? 5 : 8;  // bits per swept register in the block index
    int slot[7];
    {
      int k2 = 0;
      const uint32_t bits[7] = {kRegB, kRegC, kRegD, kRegE, kRegH, kRegL, kRegM};
#pragma unroll
      for (int r = 0; r < 7; r++) slot[r] = (ext & bits[r]) ? k2++ : -1;
    }
    const BDec bd = bdec_make(spw, reduced, nx, fw, slot);
    // compared bytes of the packed words (A F B C / D E H L / SP M)
    [[maybe_unused]] const uint32_t keep0 = 0xFFu | (uint32_t(pr.keepF) << 8) | ((pr.keepR & 1u) ? 0xFF0000u : 0u) |
                           ((pr.keepR & 2u) ? 0xFF000000u : 0u);
    [[maybe_unused]] const uint32_t keep1 =
        ((pr.keepR & 4u) ? 0xFFu : 0u) | ((pr.keepR & 8u) ? 0xFF00u : 0u) | ((pr.keepR & 16u) ? 0xFF0000u : 0u) |
        ((pr.keepR & 32u) ? 0xFF000000u : 0u);

    bool bad = false;      // a unit of this chunk has a mismatch
    bool stopped = false;  // left the chunk on the pair's flag (rejected or cancelled elsewhere)
    uint32_t done = 0;     // units swept
    // The pair's flag is asked for before a unit and looked at after it, so
    // that the read's latency passes behind the unit: a rejected pair costs
    // each warp one unit, not a batch of them between two polls.
    auto sweep = [&](auto unit) {
      while (done < units) {
        const uint32_t settled = lane == 0 ? *flag : 0u;
        bad = __any_sync(kFull, unit(u0 + done));
        done++;
        if (bad) break;
        if (__shfl_sync(kFull, settled, 0)) {
          stopped = true;
          break;
        }
      }
    };
    extern __shared__ uint32_t zsm[];  // the candidate's output planes, a column per lane
    const bool xind = (pr.keepR & kXIndep) != 0;
    if constexpr (CLS == 5) {
      // the register state (A, F, B..L), programs as they are
      uint32_t* sm = zsm + (threadIdx.x >> 5) * (kRegWords * 32) + lane;
      if (xind) {
        int rlast = -1;  // the register of the last swept field (the fastest)
#pragma unroll
        for (int r = 0; r < 6; r++)
          if (slot[r] == nx - 1) rlast = r;
        sweep([&](unsigned long long u) {
          return rxbits_unit(u, pr.nblocks, reduced, nx, rlast, bd, pw, int(tl), int(cl), pr.keepF, pr.keepR, sm);
        });
      } else {
        sweep([&](unsigned long long u) {
          return rbits_unit(u, pr.nblocks, bd, pw, int(tl), int(cl), pr.keepF, pr.keepR, sm);
        });
      }
    } else if constexpr (CLS == 4) {
      // the wide compact state, the programs renamed onto B, C, H and L
      const uint32_t set = (pr.cmap & ~uint32_t(kWideClass)) - 1u;
      if (lane < tl + cl) pw = (uint32_t(uint16_t(g_wren[set][pw & 0xFFFFu]))) | (pw & 0xFFFF0000u);
      int o[4];
      uint32_t cmp = 0;
#pragma unroll
      for (int f = 0; f < 4; f++) {
        o[f] = g_worig[set][f];
        if (o[f] >= 0 && ((pr.keepR >> o[f]) & 1u)) cmp |= 1u << f;
      }
      uint32_t* sm = zsm + (threadIdx.x >> 5) * (kWideWords * 32) + lane;
      const WDec dec = wdec_make(nx, reduced, slot, o);
      sweep([&](unsigned long long u) {
        return wbits_unit(u, pr.nblocks, dec, pw, int(tl), int(cl), pr.keepF, cmp, sm);
      });
    } else if constexpr (CLS == 3) {
      // the compact state, the programs renamed onto B and C
      const uint32_t set = pr.cmap - 1u;
      if (lane < tl + cl) pw = (uint32_t(uint16_t(g_cren[set][pw & 0xFFFFu]))) | (pw & 0xFFFF0000u);
      const int o0 = g_corig[set][0], o1 = g_corig[set][1];
      uint32_t* sm = zsm + (threadIdx.x >> 5) * (kCompactWords * 32) + lane;
      const CDec dec = cdec_make(nx, slot, o0, o1);
      if (xind) {
        // A-independent: units of 1,024 A-blocks, each at A = 0 and 1
        int rlast = -1;
#pragma unroll
        for (int r = 0; r < 7; r++)
          if (slot[r] == nx - 1) rlast = r;
        sweep([&](unsigned long long u) {
          return cxbits_unit(u, pr.nblocks, nx, dec, rlast, pw, int(tl), int(cl), pr.keepF, pr.keepR, o0, o1, sm);
        });
      } else {
        sweep([&](unsigned long long u) {
          return cbits_unit(u, pr.nblocks, dec, pw, int(tl), int(cl), pr.keepF, pr.keepR, o0, o1, sm);
        });
      }
    } else if constexpr (!XI) {
      // Unit = 4 A-blocks, bit-sliced (256 states of each block in 8 lanes).
      // The reference nests its loops as A, carry, first register, ...,
      // last register, SP (verifier.go:498-531,578-610); the block index
      // varies SP and the last register fastest, so a sweep the reference
      // abandons early is abandoned early here too.
      uint32_t* sm = zsm + (threadIdx.x >> 5) * (kBitsWords * 32) + lane;
      sweep([&](unsigned long long u) {
        return bits_unit(u, pr.nblocks, bd, pw, int(tl), int(cl), pr.keepF, pr.keepR, sm);
      });
    } else if constexpr (CLS == 2) {
      // Unit = 1,024 A-blocks, 32 per lane, each at A = 0 and A = 1.
      uint32_t* sm = zsm + (threadIdx.x >> 5) * (kBitsWords * 32) + lane;
      int rlast = -1;  // the register of the last swept field (the fastest)
#pragma unroll
      for (int r = 0; r < 7; r++)
        if (slot[r] == nx - 1) rlast = r;
      sweep([&](unsigned long long u) {
        return xbits_unit(u, pr.nblocks, spw, reduced, nx, fw, slot, rlast, pw, int(tl), int(cl), pr.keepF, pr.keepR,
                          sm);
      });
    } else {
      // Unit = 128 A-blocks, each evaluated at A = 0 and A = 1: state slot s
      // of the warp (s = (i*K + q)*32 + lane) takes block unit*128 + s/2 with
      // A = s & 1.
      sweep([&](unsigned long long u) {
        const unsigned long long first = u * kUnitBlocks;
        const unsigned long long nb = (pr.nblocks - first < kUnitBlocks) ? pr.nblocks - first : kUnitBlocks;
        return xindep_unit<K>(first, nb, bd, pw, int(tl), int(cl), keep0, keep1);
      });
    }
    if (lane == 0) {
      const unsigned long long per = xind ? (A.xunit ? A.xunit : kUnitBlocks) : kBitsBlocks;
      const unsigned long long lo = u0 * per, hi = min(pr.nblocks, (u0 + done) * per);
      tally[threadIdx.x >> 5][0] += ((hi - lo) * 256ull) << (pr.sweepf & 0x3Fu);
      tally[threadIdx.x >> 5][1] += (hi - lo) * (xind ? 2ull : 256ull);
      if (bad) *flag = 1u;
      else if (!stopped && A.wend) chunk_passed(A.rejected, A.wend, A.cdone, p, nch);
    }
  }
  if (lane == 0 && tally[threadIdx.x >> 5][0]) {
    atomicAdd(A.states, tally[threadIdx.x >> 5][0]);
    atomicAdd(A.states + 1, tally[threadIdx.x >> 5][1]);
  }
}
// Window heads settle their lane: the first pair of the window that passed
// wins; if none did, the lane moves past the window, the next window doubles
// (up to 2^max_spec), and a lane with nothing left is resolved without a
// winner.  PAIR: a lane whose slots are used up but not its pairs waits for a
// rescan.
template <bool PAIR>
__global__ void __launch_bounds__(256) k_round_resolve(const RoundArgs* __restrict__ A) {
  const RoundBuf& R = A->R;
  const Lanes& L = A->L;
  const uint32_t np = min(R.ctl->npairs, R.cap);
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    const uint32_t w = R.wlen[p];
    if (w == 0) continue;
    const PairRec pr = R.pairs[p];
    const uint32_t kind = (pr.keepR & 0x80u) ? 1u : 0u;
    const uint32_t idx = 2 * pr.target + kind;
    uint32_t j = 0;
    while (j < w && R.rejected[p + j] != 0) j++;
    if (j < w) {
      L.win[idx] = R.pairs[p + j].cand;
      L.windiff[idx] = A->sdiff[R.pair_src[p + j]];
      L.next[idx] = (L.next[idx] + j) | kResolved;
      continue;
    }
    const uint32_t nx = L.next[idx] + w;
    if (L.spec[idx] < A->max_spec) L.spec[idx] += 1;
    bool left;
    if constexpr (PAIR) {
      left = nx < A->ps.cnt[idx];
      if (!left && A->ps.resume[idx] != kNone) {
        left = true;
        A->ps.scan[atomicAdd(&R.ctl->nscan, 1u)] = idx;
      }
    } else {
      left = nx < (kind ? A->q.cnt_m[pr.target] : A->q.cnt_f[pr.target]);
    }
    L.next[idx] = left ? nx : nx | kResolved;
    if (left) R.ctl->active = 1;
  }
}
// The counters of the round that ended and a clean slate for the next one;
// in a loop, its condition.
template <bool LOOP>
__global__ void k_round_end(const RoundArgs* __restrict__ A, cudaGraphConditionalHandle loop) {
  RoundCtl& c = *A->R.ctl;
  const unsigned lane = lane_id();
  if (lane < kClasses) {
    c.alloc[lane] = 0;
    c.counter[lane] = 0;
  }
  if (lane != 0) return;
  const uint32_t np = min(c.npairs, A->R.cap);
  c.iters += 1;
  c.np = np;
  if (np) {
    c.rounds += 1;
    c.pairs += np;
  }
  uint32_t more = c.active;
  if (more && c.iters >= kMaxRoundIters) {
    // the loop has run far past any legitimate number of rounds: end it and
    // let the host report the error
    c.overrun = 1;
    more = 0;
  }
  c.more = more;
  c.npairs = 0;
  c.active = 0;
  if (LOOP && !more) cudaGraphSetConditional(loop, 0);
}
__global__ void k_round_args(RoundArgs a, RoundArgs* __restrict__ dst) {
  const uint32_t* s = reinterpret_cast<const uint32_t*>(&a);
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  for (uint32_t i = threadIdx.x; i < sizeof(RoundArgs) / 4; i += blockDim.x) d[i] = s[i];
  uint32_t* c = reinterpret_cast<uint32_t*>(a.R.ctl);
  for (uint32_t i = threadIdx.x; i < sizeof(RoundCtl) / 4; i += blockDim.x) c[i] = 0u;
}
static_assert(sizeof(RoundArgs) % 4 == 0 && sizeof(RoundCtl) % 4 == 0, "copied by words");

// Lane i copies word i of the counters and the passes' controls; lane 0 adds
// the totals.
__global__ void k_report(const Tally* __restrict__ t, QCOut q, uint32_t n, const uint32_t* __restrict__ rbase,
                         const uint32_t* __restrict__ rcnt, uint32_t nr, const RoundCtl* __restrict__ ctl, Report* out) {
  static_assert(sizeof(Tally) % 4 == 0 && sizeof(RoundCtl) % 4 == 0, "copied by words");
  for (uint32_t i = threadIdx.x; i < sizeof(Tally) / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(&out->tally)[i] = reinterpret_cast<const uint32_t*>(t)[i];
  if (ctl)
    for (uint32_t i = threadIdx.x; i < 2 * sizeof(RoundCtl) / 4; i += blockDim.x)
      reinterpret_cast<uint32_t*>(out->pass)[i] = reinterpret_cast<const uint32_t*>(ctl)[i];
  if (threadIdx.x != 0) return;
  out->nsurv = (unsigned long long)q.base[n - 1] + q.cnt_f[n - 1] + q.cnt_m[n - 1];
  out->nrules = nr ? (unsigned long long)rbase[nr - 1] + rcnt[nr - 1] : 0ull;
}
__global__ void k_lanes_init(Lanes L, uint32_t lanes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= lanes) return;
  L.next[i] = 0;
  L.win[i] = kNone;
  L.spec[i] = 0;
}
// Thread i takes the i-th run of the items; the runs' sums are scanned by
// warps, then the warps' totals by the first.
__global__ void __launch_bounds__(1024) k_scan_small(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                     uint32_t n) {
  __shared__ uint32_t totals[32];
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t lo = min(threadIdx.x * per, n), hi = min(lo + per, n);
  uint32_t sum = 0;
  for (uint32_t i = lo; i < hi; i++) sum += in[i];
  uint32_t x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane_id() >= unsigned(o)) x += y;
  }
  if (lane_id() == 31) totals[threadIdx.x >> 5] = x;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t w = 0; w < (threadIdx.x >> 5); w++) before += totals[w];
  uint32_t at = before + x - sum;
  for (uint32_t i = lo; i < hi; i++) {
    const uint32_t v = in[i];  // in may be out
    out[i] = at;
    at += v;
  }
}

__global__ void k_midcheck(DevTargets T, DevPool P, const uint32_t* __restrict__ surv,
                           const uint32_t* __restrict__ surv_target, uint32_t nsurv, uint8_t* __restrict__ pass) {
  const unsigned lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = gw; i < nsurv; i += nw) {
    const uint32_t t = surv_target[i], c = surv[i];
    const uint32_t tl = target_len(T, t), cl = pool_len(P, c);
    uint32_t pw = 0;
    if (lane < tl) pw = T.insn[(size_t)t * T.stride + lane];
    else if (lane < tl + cl) pw = P.insn[(size_t)c * P.stride + (lane - tl)];
    Z80S x = vec_state(int(lane)), y = x;
    run_lanes(x, pw, 0, int(tl));
    run_lanes(y, pw, int(tl), int(cl));
    const Keep keep = make_keep(~target_dead(T, t), ~target_dead_regs(T, t) & 0x3Fu, true);
    bool ok = __all_sync(kFull, eq_keep(x, y, keep));
    if (lane == 0) pass[i] = ok ? 1 : 0;
  }
}

__global__ void k_surv_targets(QCOut q, uint32_t n, uint32_t* __restrict__ st) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  uint32_t b = q.base[t], c = q.cnt_f[t] + q.cnt_m[t];
  for (uint32_t j = 0; j < c; j++) st[b + j] = t;
}

__global__ void k_rule_count_first(Lanes L, Lanes L2, uint32_t n, uint32_t* __restrict__ cnt, DevTargets T,
                                   unsigned long long* checked, uint32_t pool_enum,
                                   unsigned long long pool2_enum) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long ch = 0;
  if (t < n) {
    uint32_t c = 0;
    const bool masked = target_dead(T, t) != 0 || target_dead_regs(T, t) != 0;
    for (int kind = 0; kind < 2; kind++) {
      const uint32_t w1 = L.win[2 * t + kind];
      const uint32_t w2 = L2.win ? L2.win[2 * t + kind] : kNone;
      c += (w1 != kNone || w2 != kNone) ? 1u : 0u;
      // worker.go:134 counts every enumerated candidate up to and including
      // the winner (the pool index is the enumeration ordinal): all of the
      // shorter lengths, then the winner's own length
      if (kind == 0 || masked) {
        if (w1 != kNone) ch += (unsigned long long)w1 + 1ull;
        else if (L2.win) ch += pool_enum + ((w2 != kNone) ? (unsigned long long)w2 + 1ull : pool2_enum);
        else ch += pool_enum;
      }
    }
    cnt[t] = c;
  }
  // one atomic per block: one per warp, all on the same address, took 267 us
  // for 9.8M targets (45 us so)
  __shared__ unsigned long long part[8];
  for (int off = 16; off; off >>= 1) ch += __shfl_down_sync(kFull, ch, off);
  if (lane_id() == 0) part[threadIdx.x >> 5] = ch;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t k = 1; k < blockDim.x >> 5; k++) ch += part[k];
    if (ch) atomicAdd(checked, ch);
  }
}
// What candidate c saves on a target.
__device__ __forceinline__ void rule_savings(DevRule& r, const TargetMeta& m, const DevPool& P, uint32_t c) {
  int ts = 0;
  const uint32_t cl = pool_len(P, c);
  for (uint32_t i = 0; i < cl; i++) ts += g_ops[P.insn[(size_t)c * P.stride + i] & 0xFFFFu].tstates;
  r.bytes_saved = int16_t(int(m.bytes) - int(P.size[c]));
  r.cycles_saved = int16_t(int(m.tstates) - ts);
}
__global__ void k_rule_write_first(Lanes L, Lanes L2, uint32_t n, const uint32_t* __restrict__ base,
                                   const TargetMeta* __restrict__ meta, DevPool P, DevPool P2,
                                   DevRule* __restrict__ out) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  uint32_t b = base[t];
  for (int kind = 0; kind < 2; kind++) {
    const uint32_t idx = 2 * t + kind;
    const uint32_t w1 = L.win[idx];
    const uint32_t w2 = L2.win ? L2.win[idx] : kNone;
    if (w1 == kNone && w2 == kNone) continue;
    DevRule r;
    r.target = t;
    r.cand = w1 != kNone ? w1 : w2;
    r.diff = kind ? (w1 != kNone ? L.windiff[idx] : L2.windiff[idx]) : uint16_t(0);
    r.kind = uint8_t(kind);
    r.clen = w1 != kNone ? 1 : 2;
    rule_savings(r, meta[t], w1 != kNone ? P : P2, r.cand);
    out[b++] = r;
  }
}

// All-hits: flag[i] = 1 when survivor i passed MidCheck and ExhaustiveCheck.
__global__ void k_rule_count_all(RoundBuf R, uint32_t npairs, uint32_t* __restrict__ flag) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npairs) return;
  if (R.rejected[p] == 0) flag[R.pair_src[p]] = 1u;
}

__global__ void k_rule_write_all(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ base,
                                 uint32_t nsurv, const uint32_t* __restrict__ surv,
                                 const uint16_t* __restrict__ sdiff, const uint32_t* __restrict__ surv_target,
                                 const TargetMeta* __restrict__ meta, DevPool P, DevRule* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nsurv || !flag[i]) return;
  DevRule r;
  r.target = surv_target[i];
  r.cand = surv[i];
  r.diff = sdiff[i];
  r.kind = 2;
  r.clen = 1;
  rule_savings(r, meta[r.target], P, r.cand);
  out[base[i]] = r;
}

// Verifier tiers for explicit pairs (QuickCheck, MidCheck, FlagDiff); warp
// per pair, lane v = vector v.
__global__ void k_verify_small(const uint32_t* __restrict__ tgt, const uint8_t* __restrict__ tlens,
                               const uint32_t* __restrict__ cand, const uint8_t* __restrict__ clens,
                               uint32_t stride, uint32_t n, const uint8_t* __restrict__ dead,
                               uint32_t tiers, uint8_t* __restrict__ out, uint8_t* __restrict__ flagdiff) {
  const unsigned lane = lane_id();
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = gw; i < n; i += nw) {
    const uint32_t tl = tlens[i], cl = clens[i];
    uint32_t pw = 0;
    if (lane < tl) pw = tgt[(size_t)i * stride + lane];
    else if (lane < tl + cl) pw = cand[(size_t)i * stride + (lane - tl)];
    Z80S x = vec_state(int(lane)), y = x;
    run_lanes(x, pw, 0, int(tl));
    run_lanes(y, pw, int(tl), int(cl));
    const uint32_t dm = dead ? dead[i] : 0u;
    const Keep keep = make_keep(~dm, 0x3Fu, true);
    const bool eq = eq_keep(x, y, keep);
    // FlagDiff (verifier.go:658-673) over the 8 QuickCheck vectors
    const bool regs_eq = (x.a == y.a) && (x.b == y.b) && (x.c == y.c) && (x.d == y.d) &&
                         (x.e == y.e) && (x.h == y.h) && (x.l == y.l) && (x.sp == y.sp) && (x.m == y.m);
    const unsigned q8 = __ballot_sync(kFull, eq) & 0xFFu;
    const unsigned all32 = __ballot_sync(kFull, eq);
    const unsigned r8 = __ballot_sync(kFull, regs_eq) & 0xFFu;
    uint32_t fx = lane < 8 ? (x.f ^ y.f) : 0u;
    for (int off = 16; off; off >>= 1) fx |= __shfl_down_sync(kFull, fx, off);
    if (lane == 0) {
      uint8_t r = 0;
      if ((tiers & 1u) && q8 == 0xFFu) r |= 1;
      if ((tiers & 2u) && all32 == kFull) r |= 2;
      out[i] = r;
      if (flagdiff) flagdiff[i] = (r8 == 0xFFu) ? uint8_t(fx) : uint8_t(0);
    }
  }
}

// ------------------------------------------------- length-2 candidates
//
// The candidates of length 2 are the 4,531^2 odometer pairs of the 8-bit
// list (pair index = first * 4531 + second, the EnumerateSequences8 order),
// held as a pool whose QuickCheck outputs are precomputed like the length-1
// pool, the eight outputs of a pair in one 128-byte line.  Instead of
// comparing every target with all 20.5M pairs, an index per dead-register
// mask in use (PairIndex) sorts the unpruned pairs into groups with the same
// outputs; a target finds the groups with its own outputs by hash, compares
// their F bytes under its dead flags, and takes the smallest pair indices of
// the groups that pass.  Survivors go to fixed slots per (target, kind)
// lane; a lane whose slots are used up without a winner goes on from the
// pair after the last one it took.

// Bytes of an output's packed words 0 and 1 that count under a dead-register
// mask whatever the dead flags are (A and the live registers; not F).
__device__ __forceinline__ uint32_t key_keep0(uint32_t dregs) {
  return 0xFFu | ((dregs & 1u) ? 0u : 0xFF0000u) | ((dregs & 2u) ? 0u : 0xFF000000u);
}
__device__ __forceinline__ uint32_t key_keep1(uint32_t dregs) {
  return ((dregs & 4u) ? 0u : 0xFFu) | ((dregs & 8u) ? 0u : 0xFF00u) | ((dregs & 16u) ? 0u : 0xFF0000u) |
         ((dregs & 32u) ? 0u : 0xFF000000u);
}
// Hash of one vector's output (A, live registers, SP, M); the hash of a
// sequence is the sum over the eight vectors, so that the lanes of a warp can
// each hash one.  (The finalising multipliers are the published ones of
// splitmix64, and in qc_mix below those of MurmurHash3.)
__device__ __forceinline__ unsigned long long vector_hash(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t v) {
  unsigned long long h = ((unsigned long long)w0 << 32) | w1;
  h ^= (unsigned long long)(w2 + (v << 24)) * 0x9E3779B97F4A7C15ull;
  h ^= h >> 30;
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 27;
  h *= 0x94D049BB133111EBull;
  return h ^ (h >> 31);
}
__device__ __forceinline__ uint32_t pair_group_key(uint32_t size, unsigned long long h) {
  return ((size - 2u) << 30) | uint32_t(h >> 34);
}
// Thread per unpruned pair (one 128-byte line each).
__global__ void __launch_bounds__(256) k_pair_keys(DevPool P, const uint4* __restrict__ out,
                                                   const uint32_t* __restrict__ valid, uint32_t n, uint32_t dregs,
                                                   unsigned long long* __restrict__ keys) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t q = valid[i];
  const uint32_t k0 = key_keep0(dregs), k1 = key_keep1(dregs);
  unsigned long long h = 0;
  uint32_t flo = 0, fhi = 0;
#pragma unroll
  for (uint32_t v = 0; v < 8; v++) {
    const uint4 o = out[(size_t)q * 8 + v];
    h += vector_hash(o.x & k0, o.y & k1, o.z, v);
    const uint32_t f = (o.x >> 8) & 0xFFu;
    if (v < 4) flo |= f << (8 * v);
    else fhi |= f << (8 * (v - 4));
  }
  const uint32_t fh = uint32_t(vector_hash(flo, fhi, 0u, 0u) >> 32);
  keys[i] = ((unsigned long long)pair_group_key(P.size[q], h) << 32) | fh;
}
// A position begins a group where its pair's outputs (live registers, A, SP,
// M, F) differ from the position before it; equal keys are compared in full,
// so a group never mixes two outputs whose hashes collide.
__global__ void __launch_bounds__(256) k_pair_heads(const uint4* __restrict__ out,
                                                    const unsigned long long* __restrict__ keys,
                                                    const uint32_t* __restrict__ members, uint32_t n, uint32_t dregs,
                                                    uint32_t* __restrict__ head) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool h = i == 0 || keys[i] != keys[i - 1];
  if (!h) {
    const uint32_t k0 = key_keep0(dregs) | 0xFF00u, k1 = key_keep1(dregs);
    const uint4* a = out + (size_t)members[i] * 8;
    const uint4* b = out + (size_t)members[i - 1] * 8;
    uint32_t d = 0;
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const uint4 x = a[v], y = b[v];
      d |= ((x.x ^ y.x) & k0) | ((x.y ^ y.y) & k1) | (x.z ^ y.z);
    }
    h = d != 0;
  }
  head[i] = h ? 1u : 0u;
}
// gid: inclusive sum of the head flags.
__global__ void __launch_bounds__(256) k_pair_groups(const uint4* __restrict__ out,
                                                     const unsigned long long* __restrict__ keys,
                                                     const uint32_t* __restrict__ members, uint32_t n,
                                                     const uint32_t* __restrict__ gid, uint4* __restrict__ groups) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (i == n - 1) groups[gid[i]] = make_uint4(0xFFFFFFFFu, n, 0u, 0u);
  if (i != 0 && gid[i] == gid[i - 1]) return;
  const uint4* o = out + (size_t)members[i] * 8;
  uint32_t f[2] = {0u, 0u};
#pragma unroll
  for (int v = 0; v < 8; v++) f[v >> 2] |= ((o[v].x >> 8) & 0xFFu) << (8 * (v & 3));
  groups[gid[i] - 1] = make_uint4(uint32_t(keys[i] >> 32), i, f[0], f[1]);
}
__global__ void k_pair_top(const uint4* __restrict__ groups, uint32_t n_groups, uint32_t* __restrict__ top) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > kPairTop) return;
  uint32_t lo = 0, hi = n_groups;
  if (t == kPairTop) lo = n_groups;
  else
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (groups[mid].x < (t << (32 - kPairTopBits))) lo = mid + 1;
      else hi = mid;
    }
  top[t] = lo;
}

// Lanes of the length-2 pass: a (target, kind) lane takes part when the
// length-1 pass found no candidate for it, the target is long enough in
// bytes for a 2-instruction replacement, and (masked kind) the target has
// dead flags or registers.
__global__ void k_pair_lanes_init(DevTargets T, Lanes L1, QCOut q1, Lanes L2, PairScan ps) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long chk = 0;
  if (t < T.n) {
    const uint32_t tb = q1.meta[t].bytes;
    const bool masked = target_dead(T, t) != 0 || target_dead_regs(T, t) != 0;
    bool any = false;
    for (int kind = 0; kind < 2; kind++) {
      const uint32_t idx = 2 * t + kind;
      const bool need = L1.win[idx] == kNone && tb >= 3 && (kind == 0 || masked);
      L2.next[idx] = need ? 0u : kResolved;
      L2.spec[idx] = 0;
      L2.win[idx] = kNone;
      L2.windiff[idx] = 0;
      ps.cnt[idx] = 0;
      ps.resume[idx] = need ? 0u : kNone;
      any = any || need;
    }
    if (any) chk = ps.eligible[tb < 16 ? tb : 15];
  }
  for (int off = 16; off; off >>= 1) chk += __shfl_down_sync(kFull, chk, off);
  if (lane_id() == 0 && chk) atomicAdd(ps.checks, chk);
}

__device__ __forceinline__ uint32_t lower_bound_u64(const unsigned long long* a, uint32_t n, unsigned long long v) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (a[mid] < v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The two hashes of one vector's compared output; an output's hash is the sum
// over the eight vectors, so that lanes can each hash one.
__device__ __forceinline__ uint32_t qc_mix(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t h = a * 0x9E3779B1u;
  h = (h ^ (h >> 15)) + b;
  h *= 0x85EBCA6Bu;
  h = (h ^ (h >> 13)) + c;
  h *= 0xC2B2AE35u;
  return h ^ (h >> 16);
}
__device__ __forceinline__ uint32_t qc_hash(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t v) {
  return qc_mix(w0, w1, w2 + (v << 27));
}
__device__ __forceinline__ uint32_t qc_hash2(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t v) {
  return qc_mix(w1 ^ 0x5BD1E995u, w2 + (v << 24), w0 + 0x27D4EB2Fu);
}
// Index build (QCIndex): pruned candidates' keys sort past every real one.
__global__ void k_qc_keys(DevPool P, uint32_t w2mask, uint32_t m0, uint32_t nm, unsigned long long* __restrict__ keys) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nm * P.n) return;
  const uint32_t m = m0 + i / P.n, q = i % P.n;
  if (P.prune[q]) {
    keys[i] = ~0ull;
    return;
  }
  uint32_t h = 0;
#pragma unroll
  for (uint32_t v = 0; v < 8; v++) {
    const uint4 o = P.qc[(size_t)v * P.n + q];
    h += qc_hash(o.x & key_keep0(m), o.y & key_keep1(m), o.z & w2mask, v);
  }
  keys[i] = ((unsigned long long)m << 58) | ((unsigned long long)h << kQCIndexBits) | q;
}
__global__ void k_qc_entries(DevPool P, uint32_t w2mask, const unsigned long long* __restrict__ keys, uint32_t n,
                             uint4* __restrict__ entries, uint32_t* __restrict__ hash2) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long key = keys[i];
  const uint32_t m = uint32_t(key >> 58), c = uint32_t(key) & ((1u << kQCIndexBits) - 1u);
  uint32_t h2 = 0, f[2] = {0u, 0u};
#pragma unroll
  for (uint32_t v = 0; v < 8; v++) {
    const uint4 o = P.qc[(size_t)v * P.n + c];
    h2 += qc_hash2(o.x & key_keep0(m), o.y & key_keep1(m), o.z & w2mask, v);
    f[v >> 2] |= ((o.x >> 8) & 0xFFu) << (8 * (v & 3u));
  }
  entries[i] = make_uint4(uint32_t(key >> kQCIndexBits), c | uint32_t(P.size[c]) << kQCIndexBits, f[0], f[1]);
  hash2[i] = h2;
}
// Every entry against the nearest one before it with both hashes equal:
// flags[0] is set where their outputs differ, flags[1] where entries of one
// first hash have two second ones.
__global__ void k_qc_check(DevPool P, uint32_t w2mask, const unsigned long long* __restrict__ keys,
                           const uint32_t* __restrict__ hash2, uint32_t n, uint32_t* __restrict__ flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned long long run = keys[i] >> kQCIndexBits;
  const uint32_t m = uint32_t(keys[i] >> 58), c = uint32_t(keys[i]) & ((1u << kQCIndexBits) - 1u);
  uint32_t j = i;
  do {
    if (j == 0 || (keys[j - 1] >> kQCIndexBits) != run) return;
    j--;
    if (hash2[j] != hash2[i]) flags[1] = 1;
  } while (hash2[j] != hash2[i]);
  const uint32_t e = uint32_t(keys[j]) & ((1u << kQCIndexBits) - 1u);
  uint32_t d = 0;
#pragma unroll
  for (uint32_t v = 0; v < 8; v++) {
    const uint4 x = P.qc[(size_t)v * P.n + c], y = P.qc[(size_t)v * P.n + e];
    d |= ((x.x ^ y.x) & key_keep0(m)) | ((x.y ^ y.y) & key_keep1(m)) | ((x.z ^ y.z) & w2mask);
  }
  if (d) flags[0] = 1;
}
__global__ void k_qc_top(const unsigned long long* __restrict__ keys, uint32_t nv, uint32_t first, uint32_t m0,
                         uint32_t nm, uint32_t top_bits, uint32_t* __restrict__ top) {
  const uint32_t per = (1u << top_bits) + 1u;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nm * per) return;
  const uint32_t j = i / per, b = i - j * per, m = m0 + j;
  const uint32_t seg = j * nv;
  const unsigned long long lo =
      ((unsigned long long)m << 58) | ((unsigned long long)b << (32u - top_bits + kQCIndexBits));
  top[m * per + b] = first + (b == per - 1u ? seg + nv : seg + lower_bound_u64(keys + seg, nv, lo));
}

// What a target's lanes know of it when they read its range of entries.
struct QCQuery {
  uint32_t t;                  // the target
  uint32_t base;               // lane that ran vector 0 (the others follow it)
  uint32_t h, h2, flo, fhi;    // hashes, F bytes
  uint32_t live;               // live flag bits, in every byte
  uint32_t size, m, k0, k1;    // encoded bytes, dead registers, live bytes of words 0 and 1
  uint32_t nf_total, obase;    // collect pass: full survivors, first slot
};
// Survivors of one target found so far: tallies per lane (count pass), places
// (collect pass: full, masked), all of them (single pass).
struct QCFound {
  uint32_t lf = 0, lm = 0, nf = 0, nm = 0, nk = 0;
};
// Reads entries [r0, r1) of a target's range, W at a time (W lanes per target:
// 8, each group its own target, or 32, the whole warp one), `steps` times.
// w: this lane's vector's outputs (of its own target).
// late: fills in what the query does not need before its first hit.
template <int W, bool COLLECT, bool KEEP, class Late>
__device__ __forceinline__ void qc_range(QCQuery& q, QCFound& f, uint32_t r0, uint32_t r1, uint32_t steps,
                                         const uint32_t (&w)[3], const DevPool& P, const QCConfig& cfg,
                                         const QCIndex& ix, const QCOut& o, Late late) {
  const unsigned lane = lane_id(), sub = lane & 7u;
  const unsigned pos = W == 8 ? sub : lane;
  const unsigned gshift = W == 8 ? (lane & ~7u) : 0u, gmask = W == 8 ? 0xFFu : kFull;
  const unsigned before = lanemask_lt() & (gmask << gshift);
  uint32_t same = 2;  // the target's outputs against an entry's: 2 not compared yet
  for (uint32_t k = 0; k < steps; k++) {
    const uint32_t i = r0 + uint32_t(W) * k + pos;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    bool hit = i < r1;
    if (hit) {
      e = ix.entries[i];
      hit = e.x == q.h;
    }
    if (!__any_sync(kFull, hit)) continue;  // most steps find nothing
    late();
    if (ix.check_h2 && hit) hit = ix.hash2[i] == q.h2;
    const uint32_t c = e.y & ((1u << kQCIndexBits) - 1u);
    // the outputs themselves, once per target: entries of equal hashes have
    // equal outputs
    const unsigned ghit = (__ballot_sync(kFull, hit) >> gshift) & gmask;
    const uint32_t c0 = __shfl_sync(kFull, c, int(gshift) + (ghit ? __ffs(int(ghit)) - 1 : 0));
    const uint32_t x = __shfl_sync(kFull, w[0], int(q.base + sub)), y = __shfl_sync(kFull, w[1], int(q.base + sub));
    const uint32_t z = __shfl_sync(kFull, w[2], int(q.base + sub));
    bool differs = false;
    if (same == 2 && ghit) {
      const uint4 v = P.qc[(size_t)sub * P.n + c0];
      differs = (((v.x ^ x) & q.k0) | ((v.y ^ y) & q.k1) | ((v.z ^ z) & cfg.w2mask)) != 0;
    }
    const unsigned gdiff = (__ballot_sync(kFull, differs) >> gshift) & gmask;
    if (same == 2 && ghit) same = gdiff ? 0u : 1u;
    const bool pass = hit && same == 1u && (e.y >> kQCIndexBits) < q.size &&
                      (((e.z ^ q.flo) | (e.w ^ q.fhi)) & q.live) == 0;
    uint32_t fd = (e.z ^ q.flo) | (e.w ^ q.fhi);
    fd |= fd >> 16;
    fd = (fd | (fd >> 8)) & 0xFFu;
    // dead registers that differ, on the candidate itself: to tell full from
    // masked, and for the survivors that are stored
    uint32_t rdf = 0;
    const bool need = pass && q.m != 0 && (COLLECT || fd == 0 || (KEEP && f.nk < kQCSlots));
    if (__any_sync(kFull, need)) {
      constexpr int kAhead = W == 8 ? 2 : 8;  // loads in flight
#pragma unroll 1
      for (int j0 = 0; j0 < 8; j0 += kAhead) {
        uint2 v[kAhead];
#pragma unroll
        for (int j = 0; j < kAhead; j++)
          if (need) v[j] = *reinterpret_cast<const uint2*>(&P.qc[(size_t)(j0 + j) * P.n + c]);
#pragma unroll
        for (int j = 0; j < kAhead; j++) {
          const uint32_t a = __shfl_sync(kFull, w[0], int(q.base) + j0 + j);
          const uint32_t b = __shfl_sync(kFull, w[1], int(q.base) + j0 + j);
          if (need) rdf |= reg_diff(v[j].x ^ a, v[j].y ^ b);
        }
      }
    }
    const uint32_t diff = fd | (rdf << 8);
    const bool fp = pass && (cfg.all_hits != 0 || diff == 0), mp = pass && !fp;
    if constexpr (!COLLECT) {
      f.lf += fp ? 1u : 0u;
      f.lm += mp ? 1u : 0u;
      if constexpr (KEEP) {
        const unsigned bs = __ballot_sync(kFull, pass);
        const uint32_t rank = f.nk + __popc(bs & before);
        if (pass && rank < kQCSlots)
          o.tmp[(size_t)q.t * kQCSlots + rank] = c | (diff << 16) | (mp ? 0x80000000u : 0u);
        f.nk += __popc((bs >> gshift) & gmask);
      }
    } else {
      // this target's survivors of the step, in enumeration order
      const unsigned bf = __ballot_sync(kFull, fp), bm = __ballot_sync(kFull, mp);
      if (fp) {
        const uint32_t idx = q.obase + f.nf + __popc(bf & before);
        o.surv[idx] = c;
        o.sdiff[idx] = uint16_t(diff);
      }
      if (mp) {
        const uint32_t idx = q.obase + q.nf_total + f.nm + __popc(bm & before);
        o.surv[idx] = c;
        o.sdiff[idx] = uint16_t(diff);
      }
      f.nf += __popc((bf >> gshift) & gmask);
      f.nm += __popc((bm >> gshift) & gmask);
    }
  }
}

// The query of the target in lanes base.. (w: its outputs by vector) short of
// the second hash and the F bytes.
__device__ __forceinline__ QCQuery qc_query(const DevTargets& T, const QCConfig& cfg, uint32_t t, bool valid,
                                            const uint32_t (&w)[3]) {
  QCQuery q{};
  q.t = t;
  q.base = lane_id() & ~7u;
  q.live = valid ? (~target_dead(T, t) & 0xFFu) * 0x01010101u : 0u;
  q.m = valid ? target_dead_regs(T, t) & 0x3Fu : 0u;
  q.k0 = key_keep0(q.m);
  q.k1 = key_keep1(q.m);
  q.h = qc_hash(w[0] & q.k0, w[1] & q.k1, w[2] & cfg.w2mask, lane_id() & 7u);
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) q.h += __shfl_xor_sync(kFull, q.h, off);
  return q;
}
__device__ __forceinline__ void qc_late(QCQuery& q, const QCConfig& cfg, const uint32_t (&w)[3]) {
  const unsigned sub = lane_id() & 7u;
  const uint32_t fb = ((w[0] >> 8) & 0xFFu) << (8u * (sub & 3u));
  q.h2 = qc_hash2(w[0] & q.k0, w[1] & q.k1, w[2] & cfg.w2mask, sub);
  q.flo = sub < 4u ? fb : 0u;
  q.fhi = sub < 4u ? 0u : fb;
#pragma unroll
  for (int off = 4; off >= 1; off >>= 1) {
    q.h2 += __shfl_xor_sync(kFull, q.h2, off);
    q.flo |= __shfl_xor_sync(kFull, q.flo, off);
    q.fhi |= __shfl_xor_sync(kFull, q.fhi, off);
  }
}
__device__ __forceinline__ void qc_bounds(const QCIndex& ix, const QCQuery& q, uint32_t& r0, uint32_t& r1) {
  const uint32_t* top = ix.top + q.m * ((1u << ix.top_bits) + 1u) + (q.h >> (32u - ix.top_bits));
  r0 = top[0];
  r1 = top[1];
}

// QuickCheck through the index: a target only meets the candidates whose
// compared outputs hash like its own.  Eight lanes per target, four targets
// per warp: lane 8g + v runs target t0 + g on vector v and hashes its output;
// the hash's range is read eight entries at a time.  A target with an entry
// of its hash (one in fourteen of the length-2 enumeration) goes on: its
// outputs against the first such entry's, and F under the dead flags entry by
// entry, from the entries themselves.  Entries of a hash are in pool order, so
// survivors come out in enumeration order as in the full scan.  Targets with
// long ranges are left to k_qc_long.  Lanes of a group that has no target
// (past the end) take part in the warp's collectives with nothing to do.
// Bound by issue and by the chain program - table - entry (more registers
// than 64 and it slows with the blocks that go).  Hashing the first vector
// alone, gathering all eight outputs of every candidate that agreed on it and
// broadcasting the target's eight outputs to every lane took 5.1 ms for 9.4M
// length-2 targets and 1.0 ms for 100,003 targets with every flag dead, this
// 1.9 and 0.13 ms (the 1.9 are hardly more than the wait for the targets: 75 MB
// take 2.3 ms to arrive, of which the last three chunks' 1.7 pass in here).
// COLLECT: the collect pass; else the count pass, which with KEEP also keeps
// the survivors of targets with at most kQCSlots (single pass).
constexpr uint32_t kQCLong = 64;  // entries: eight steps of a group, two of a warp
template <bool COLLECT, bool KEEP>
__global__ void __launch_bounds__(kBlock, 4) k_qc_bucket(DevTargets T, DevPool P, QCConfig cfg, QCIndex ix, QCOut o) {
  const unsigned lane = lane_id();
  const unsigned sub = lane & 7u;
  const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  unsigned long long my_checks = 0;
  for (uint32_t t0 = gw * 4u; t0 < T.n; t0 += nw * 4u) {
    const uint32_t t = t0 + (lane >> 3);
    const bool valid = t < T.n;
    bool work = valid;
    if (COLLECT) {
      // single pass: the count pass kept the survivors of targets with at
      // most kQCSlots of them
      if (valid) work = o.cnt_f[t] + o.cnt_m[t] > (o.tmp ? kQCSlots : 0u);
      if (!__any_sync(kFull, work)) continue;
    }
    // the target on vector `sub`; every lane reads the program itself
    const uint32_t tl = valid ? target_len(T, t) : 0u;
    const uint32_t* prog = T.insn + (size_t)t * T.stride;
    uint32_t size = 0, tstates = 0, reads = 0;
    Z80S st = vec_state(int(sub));
    const uint32_t steps = __reduce_max_sync(kFull, tl);
#pragma unroll 1
    for (uint32_t i = 0; i < steps; i++) {
      if (i < tl) {
        const uint32_t w = prog[i];
        if ((w & 0xFFFFu) >= uint32_t(kNumOps)) {
          // (only where the host leaves the check to this kernel) reported,
          // and nothing more of this target
          if (cfg.bad) atomicMax(cfg.bad, ~(cfg.first + t));
          work = false;
          continue;
        }
        const OpInfo oi = g_ops[w & 0xFFFFu];
        size += oi.size;
        tstates += oi.tstates;
        reads |= oi.reads;
        z_step(st, w & 0xFFFFu, w >> 16);
      }
    }
    uint32_t w[3];
    z_pack(st, w);
    QCQuery q = qc_query(T, cfg, t, valid, w);
    q.size = size;
    if (COLLECT && valid) {
      q.nf_total = o.cnt_f[t];
      q.obase = o.base[t];
    }
    uint32_t r0 = 0, r1 = 0;
    if (work) qc_bounds(ix, q, r0, r1);
    const bool is_long = r1 - r0 > kQCLong;
    if (is_long) {
      if (sub == 0) o.longs[atomicAdd(o.nlong, 1u)] = t;
      r1 = r0;
    }
    QCFound f;
    bool hashed = false;
    qc_range<8, COLLECT, KEEP>(q, f, r0, r1, (__reduce_max_sync(kFull, r1 - r0) + 7u) / 8u, w, P, cfg, ix, o, [&] {
      if (!hashed) qc_late(q, cfg, w);
      hashed = true;
    });
    if constexpr (!COLLECT) {
      if (hashed) {
#pragma unroll
        for (int off = 4; off >= 1; off >>= 1) {
          f.lf += __shfl_xor_sync(kFull, f.lf, off);
          f.lm += __shfl_xor_sync(kFull, f.lm, off);
        }
      }
      if (sub == 0 && valid) {
        my_checks += ix.elig_lt[size < 255u ? size : 255u];
        QCTarget g;
        g.tb = size;
        g.tts = tstates;
        g.trd = reads;
        g.tl = tl;
        qc_count_out(o, t, g, f.lf, f.lm);
        if (KEEP && f.lf + f.lm > kQCSlots) atomicAdd(o.over, 1u);
      }
    }
  }
  if constexpr (!COLLECT) {
    for (int off = 16; off; off >>= 1) my_checks += __shfl_down_sync(kFull, my_checks, off);
    if (lane == 0 && my_checks) atomicAdd(o.checks, my_checks);
  }
}
// The targets whose range is long (they leave little to compare: A kept,
// registers dead; up to 3,900 of the 4,523 candidates), a warp each: every
// eight lanes run the target, the range is read 32 entries at a time.  A
// kernel of its own, so that its registers do not weigh on the others' warps.
// Eight entries at a time such targets took 0.5 ms of a search of 200 uneven
// targets, here 0.15 ms.
template <bool COLLECT, bool KEEP>
__global__ void __launch_bounds__(128) k_qc_long(DevTargets T, DevPool P, QCConfig cfg, QCIndex ix, QCOut o) {
  const unsigned lane = lane_id();
  const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  const uint32_t n = *o.nlong;
  for (uint32_t i = gw; i < n; i += nw) {
    const uint32_t t = o.longs[i], tl = target_len(T, t);
    const uint32_t pw = lane < tl ? T.insn[(size_t)t * T.stride + lane] : 0u;
    const uint32_t size = __reduce_add_sync(kFull, lane < tl ? uint32_t(g_ops[pw & 0xFFFFu].size) : 0u);
    Z80S st = vec_state(int(lane & 7u));
    run_lanes(st, pw, 0, int(tl));
    uint32_t w[3];
    z_pack(st, w);
    QCQuery q = qc_query(T, cfg, t, true, w);
    qc_late(q, cfg, w);
    q.size = size;
    q.base = 0;
    if (COLLECT) {
      q.nf_total = o.cnt_f[t];
      q.obase = o.base[t];
    }
    uint32_t r0, r1;
    qc_bounds(ix, q, r0, r1);
    QCFound f;
    qc_range<32, COLLECT, KEEP>(q, f, r0, r1, (r1 - r0 + 31u) / 32u, w, P, cfg, ix, o, [] {});
    if constexpr (!COLLECT) {
      const uint32_t lf = __reduce_add_sync(kFull, f.lf), lm = __reduce_add_sync(kFull, f.lm);
      if (lane == 0) {
        o.cnt_f[t] = lf;
        o.cnt_m[t] = lm;
        o.cnt_all[t] = lf + lm;
        if (KEEP && lf + lm > kQCSlots) atomicAdd(o.over, 1u);
      }
    }
  }
}

// Thread per target: the survivors the single-pass count kept go to
// base[t] + (full ones in order, then masked ones in order), as the collect
// pass would have placed them.
__global__ void __launch_bounds__(256) k_qc_compact(QCOut o, uint32_t n) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const uint32_t nf = o.cnt_f[t], tot = nf + o.cnt_m[t];
  if (tot == 0 || tot > kQCSlots) return;
  const uint32_t* __restrict__ kept = o.tmp + (size_t)t * kQCSlots;
  uint32_t jf = o.base[t], jm = jf + nf;
  for (uint32_t j = 0; j < tot; j++) {
    const uint32_t e = kept[j];
    const uint32_t idx = (e >> 31) ? jm++ : jf++;
    o.surv[idx] = e & 0xFFFFu;
    o.sdiff[idx] = uint16_t((e >> 16) & 0x7FFFu);
  }
}

// The first position in [lo, hi) that `below` is false at (true, then false,
// over the range), hi if none.  Warp-wide, the same in every lane: each step
// probes the ends of 32 spans.
template <class Below>
__device__ __forceinline__ uint32_t warp_first(uint32_t lo, uint32_t hi, Below below) {
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31u) / 32u;
    const uint32_t i = lo + lane_id() * step + (step - 1u);
    const unsigned m = __ballot_sync(kFull, i < hi && below(i));  // spans that lie below as a whole
    lo += uint32_t(__popc(m)) * step;
    if (lo >= hi) return hi;
    hi = min(hi, lo + (step - 1u));
  }
  return lo;
}
// Ascending over the lanes: a bitonic merge of a bitonic sequence, and a sort.
__device__ __forceinline__ uint32_t warp_merge(uint32_t x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const uint32_t y = __shfl_xor_sync(kFull, x, o);
    x = (lane_id() & unsigned(o)) ? max(x, y) : min(x, y);
  }
  return x;
}
__device__ __forceinline__ uint32_t warp_sort(uint32_t x) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int o = k >> 1; o; o >>= 1) {
      const uint32_t y = __shfl_xor_sync(kFull, x, o);
      const bool up = (lane_id() & unsigned(k)) == 0 || k == 32;
      x = (((lane_id() & unsigned(o)) == 0) == up) ? min(x, y) : max(x, y);
    }
  return x;
}

// Warp per (target, kind) lane whose slots are used up and whose pairs are
// not: the kSlots2 smallest survivors from ps.resume on.  The lane's target
// runs on the eight vectors, one per thread; the groups of its hash are read
// 128 at a time and their F bytes compared under the dead flags; the members
// of a group that passes are merged, 32 at a time, into the smallest pair
// indices so far, which the threads hold in order.  Groups whose first
// member cannot enter are passed over.
// Bound by latency: a chain of some ten dependent loads per lane, and for
// targets that leave little to compare (A kept, registers dead) a walk over
// the groups of one large bucket.  A walk over the bucket's pairs instead
// (20.5M pairs, one output compared at a time, one warp per target) took
// 147 ms for 10,007 uneven targets.
// W warps per lane.  One suits many lanes; where few lanes are looked at (small
// jobs, and the lanes that wait for a rescan) a block of 16 shares the groups
// and merges what its warps found: a rescan of the large bucket that a late
// round's lanes share took 137 us of one warp, 46 of a block (40,009 uneven
// targets, 228 rescans: 33 -> 20 ms).  32 warps are no faster (the search for
// where to go on within each group that passes is a chain of loads), and a
// bound shared by the warps while they scan gave nothing.
constexpr int kScanWarps = 16;
template <int W>
__global__ void __launch_bounds__(W == 1 ? kBlock : 32 * W) k_pair_scan(const RoundArgs* __restrict__ A, bool all) {
  __shared__ uint32_t found_by[W][32];
  const DevTargets& T = A->T;
  const PairScan& ps = A->ps;
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t gw = W == 1 ? blockIdx.x * (blockDim.x >> 5) + warp : blockIdx.x;
  const uint32_t nw = W == 1 ? gridDim.x * (blockDim.x >> 5) : gridDim.x;
  const uint32_t part = W == 1 ? 0u : warp;  // this warp's share of the groups
  const uint32_t lanes = all ? 2u * T.n : A->R.ctl->nscan;
  for (uint32_t i = gw; i < lanes; i += nw) {
    const uint32_t idx = all ? i : ps.scan[i];
    const uint32_t resume = ps.resume[idx];
    int skip = (A->L.next[idx] & kResolved) || resume == kNone;
    if constexpr (W > 1) skip = __syncthreads_or(skip);  // one answer for all the warps
    if (skip) continue;
    const uint32_t t = idx >> 1, kind = idx & 1u;
    const uint32_t tl = target_len(T, t);
    const uint32_t pw = lane < tl ? T.insn[(size_t)t * T.stride + lane] : 0u;
    Z80S st = vec_state(int(lane & 7u));
    run_lanes(st, pw, 0, int(tl));
    uint32_t w[3];  // the target's output on vector lane & 7
    z_pack(st, w);
    const uint32_t tb = A->q.meta[t].bytes;
    const uint32_t dead = kind ? target_dead(T, t) & 0xFFu : 0u;
    const uint32_t dregs = kind ? target_dead_regs(T, t) & 0x3Fu : 0u;
    const uint32_t k0 = key_keep0(dregs), k1 = key_keep1(dregs);
    const uint32_t keepf = (~dead & 0xFFu) * 0x01010101u;
    const uint32_t keep0 = k0 | ((~dead & 0xFFu) << 8);
    unsigned long long h = vector_hash(w[0] & k0, w[1] & k1, w[2], lane & 7u);
    uint32_t flo = 0, fhi = 0;
    {
      const uint32_t f = (w[0] >> 8) & 0xFFu, v = lane & 7u;
      if (v < 4) flo = f << (8 * v);
      else fhi = f << (8 * (v - 4));
    }
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      h += __shfl_xor_sync(kFull, h, o);
      flo |= __shfl_xor_sync(kFull, flo, o);
      fhi |= __shfl_xor_sync(kFull, fhi, o);
    }
    const PairIndex ix = ps.idx[dregs];
    uint32_t best = kNone, worst = kNone;  // this thread's survivor; the last thread's
    for (uint32_t size = 2; size < min(tb, 2u + kPairSizes); size++) {
      const uint32_t key = pair_group_key(size, h);
      const uint32_t* top = ix.top + (key >> (32 - kPairTopBits));
      const uint32_t hi = top[1];
      const uint32_t g0 = warp_first(top[0], hi, [&](uint32_t i) { return ix.groups[i].x < key; });
      for (uint32_t base = g0 + 128u * part; base < hi; base += 128u * W) {
        uint4 r[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const uint32_t i = base + 32u * u + lane;
          in[u] = i < hi;
          r[u] = in[u] ? ix.groups[i] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          in[u] = in[u] && r[u].x == key;
          const bool fm = in[u] && (((r[u].z ^ flo) | (r[u].w ^ fhi)) & keepf) == 0;
          if (!__any_sync(kFull, fm)) continue;
          const uint32_t first = fm ? ix.members[r[u].y] : kNone;
          for (unsigned b = __ballot_sync(kFull, first < worst); b; b &= b - 1) {
            const int j = __ffs(b) - 1;
            const uint32_t c0 = __shfl_sync(kFull, first, j);
            if (c0 >= worst) continue;
            // the group's outputs themselves, on the first member
            uint32_t d = 0;
            if (lane < 8) {
              const uint4 o = ps.out[(size_t)c0 * 8 + lane];
              d = ((o.x ^ w[0]) & keep0) | ((o.y ^ w[1]) & k1) | (o.z ^ w[2]);
            }
            if (__any_sync(kFull, d != 0)) continue;
            uint32_t pos = __shfl_sync(kFull, r[u].y, j);
            const uint32_t end = ix.groups[base + 32u * u + j + 1].y;
            // only members that agree on every flag can agree on everything
            // (masked lanes leave those to the full lane)
            const bool maybe_full =
                kind && __shfl_sync(kFull, r[u].z, j) == flo && __shfl_sync(kFull, r[u].w, j) == fhi;
            if (c0 < resume)
              pos = warp_first(pos, end, [&](uint32_t i) { return ix.members[i] < resume; });
            while (pos < end) {
              uint32_t c = pos + lane < end ? ix.members[pos + lane] : kNone;
              if (__shfl_sync(kFull, c, 0) >= worst) break;
              if (maybe_full) {
                uint32_t fd = 0;
                for (int v = 0; v < 8; v++) {
                  const uint32_t x = __shfl_sync(kFull, w[0], v), y = __shfl_sync(kFull, w[1], v);
                  const uint32_t z = __shfl_sync(kFull, w[2], v);
                  if (c != kNone) {
                    const uint4 o = ps.out[(size_t)c * 8 + v];
                    fd |= (o.x ^ x) | (o.y ^ y) | (o.z ^ z);
                  }
                }
                if (fd == 0) c = kNone;
                c = warp_sort(c);
              }
              best = warp_merge(min(best, __shfl_sync(kFull, c, 31 - int(lane))));
              worst = __shfl_sync(kFull, best, 31);
              pos += 32;
            }
          }
        }
        if (!__all_sync(kFull, in[3])) break;
      }
    }
    if constexpr (W > 1) {
      // the smallest of all warps' (the whole block comes here or none of it does)
      found_by[warp][lane] = best;
      __syncthreads();
      if (warp == 0) {
        for (int k = 1; k < W; k++) best = warp_merge(min(best, found_by[k][31 - lane]));
        worst = __shfl_sync(kFull, best, 31);
      }
      __syncthreads();
      if (warp != 0) continue;
    }
    // slots, and the outputs in which each survivor differs
    uint32_t fd = 0, rdf = 0;
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const uint32_t x = __shfl_sync(kFull, w[0], v), y = __shfl_sync(kFull, w[1], v);
      if (best != kNone) {
        const uint4 o = ps.out[(size_t)best * 8 + v];
        fd |= ((o.x ^ x) >> 8) & 0xFFu;
        rdf |= reg_diff(o.x ^ x, o.y ^ y);
      }
    }
    if (best != kNone) {
      ps.surv[(size_t)idx * kSlots2 + lane] = best;
      ps.sdiff[(size_t)idx * kSlots2 + lane] = uint16_t(fd | (rdf << 8));
    }
    const uint32_t found = __popc(__ballot_sync(kFull, best != kNone));
    if (lane == 0) {
      ps.cnt[idx] = found;
      A->L.next[idx] = 0;
      ps.resume[idx] = worst == kNone ? kNone : worst + 1u;
    }
  }
}
static_assert(kSlots2 == 32, "one slot per thread of the warp");

unsigned grid_for(uint32_t n, unsigned block) { return (n + block - 1) / block; }

// Launch facts are properties of a device: its SM count, and per kernel the
// dynamic shared-memory limit (cudaFuncSetAttribute acts on the current
// device) and the resident blocks per SM.  They are cached per device, for
// the device current at the launch; devices past kMaxCachedDevices are
// queried on every launch.
constexpr int kMaxCachedDevices = 64;
std::atomic<int> g_num_sms[kMaxCachedDevices];

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  return dev;
}

// Resident blocks per SM of kernel f on the current device with `smem`
// bytes of dynamic shared memory, raising the kernel's shared-memory limit
// to smem first when it is above the default; cache[] keeps one answer per
// device.
template <class F>
int blocks_per_sm(std::atomic<int>* cache, F f, int block, size_t smem, size_t smem_limit) {
  const int dev = current_device();
  if (dev >= 0 && dev < kMaxCachedDevices) {
    const int c = cache[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  if (smem_limit) cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_limit));
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, block, smem);
  if (per_sm < 1) per_sm = 1;
  if (dev >= 0 && dev < kMaxCachedDevices) cache[dev].store(per_sm, std::memory_order_relaxed);
  return per_sm;
}

}  // namespace

int dev_num_sms() {
  const int dev = current_device();
  if (dev >= 0 && dev < kMaxCachedDevices) {
    const int c = g_num_sms[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (n <= 0) n = 1;
  if (dev >= 0 && dev < kMaxCachedDevices) g_num_sms[dev].store(n, std::memory_order_relaxed);
  return n;
}

}  // namespace z80b

// Host helpers that need the tables (kept out of the anonymous namespace).
#include "z80_tables.h"

namespace z80b {

void dev_upload_tables(cudaStream_t s) {
  cudaMemcpyToSymbolAsync(g_ops, op_table(), sizeof(OpInfo) * kNumOps, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(g_vec, mid_vectors(), sizeof(uint32_t) * 32 * 3, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_rep, rep_values(), 32, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_repsp, rep_sp(), 32, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(g_rep, rep_values(), 32, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(g_repsp, rep_sp(), 32, 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(g_aclass, op_aclass(), kNumOps, 0, cudaMemcpyHostToDevice, s);
  {
    static uint64_t flow[kNumOps][kFlowFields];
    static std::once_flag once;
    std::call_once(once, [] {
      for (int op = 0; op < kNumOps; op++)
        for (int g = 0; g < kFlowFields; g++) flow[op][g] = flow_word(op_flow()[op], g);
    });
    cudaMemcpyToSymbolAsync(g_flow, flow, sizeof flow, 0, cudaMemcpyHostToDevice, s);
    const CompactTables& C = compact_tables();
    cudaMemcpyToSymbolAsync(g_cren, C.ren, sizeof C.ren, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(g_corig, C.orig, sizeof C.orig, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(g_cid, C.id_of_set, sizeof C.id_of_set, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(g_opregs, C.opregs, sizeof C.opregs, 0, cudaMemcpyHostToDevice, s);
    const WideTables& W = wide_tables();
    cudaMemcpyToSymbolAsync(g_wren, W.ren, sizeof W.ren, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(g_worig, W.orig, sizeof W.orig, 0, cudaMemcpyHostToDevice, s);
    cudaMemcpyToSymbolAsync(g_wid, W.id_of_set, sizeof W.id_of_set, 0, cudaMemcpyHostToDevice, s);
  }
}

void launch_pool_outputs(const uint32_t* insn, uint32_t n, uint32_t len, uint4* qc, uint4* mid, bool by_pair,
                         cudaStream_t s) {
  if (!n) return;
  unsigned grid = std::min<unsigned>(grid_for(n, 4), unsigned(dev_num_sms() * 16));
  k_pool_outputs<<<grid, 128, 0, s>>>(insn, n, len, qc, mid, by_pair);
}
void launch_exec(const uint32_t* in, const uint32_t* seqs, const uint8_t* lens, uint32_t len,
                 uint32_t stride, uint32_t n, uint32_t* out, cudaStream_t s) {
  if (!n) return;
  unsigned grid = std::min<unsigned>(grid_for(n, 4), unsigned(dev_num_sms() * 16));
  k_exec<<<grid, 128, 0, s>>>(in, seqs, lens, len, stride, n, out);
}
void launch_fingerprints(const uint32_t* seqs, uint32_t n, uint32_t len, uint8_t* out, cudaStream_t s) {
  if (!n) return;
  unsigned grid = std::min<unsigned>(grid_for(n, 4), unsigned(dev_num_sms() * 16));
  k_fingerprints<<<grid, 128, 0, s>>>(seqs, n, len, out);
}
void launch_fp_query(const DevPool& P, const FpQuery& fp, uint32_t dead, uint32_t* hits, FpCounters* ctr,
                     FpAnswer* answer, cudaStream_t s) {
  const unsigned grid = std::min<unsigned>(grid_for(P.n, 256), unsigned(dev_num_sms() * 8));
  k_fp_query<<<grid ? grid : 1u, 256, 0, s>>>(P, fp, dead, hits, ctr, answer);
}
void launch_qc_scan(const DevTargets& T, const DevPool& P, const QCConfig& cfg, const QCOut& o,
                    bool collect, cudaStream_t s) {
  if (!T.n) return;
  size_t smem = cfg.use_smem ? (size_t)P.n * 17 + 16 : 0;
  // occupancy depends on smem (the pool's size), so it is cached per device
  // only for the limit; the answer for this launch is computed each time
  static std::atomic<int> limit_set[2][kMaxCachedDevices];
  const int dev = current_device();
  const bool cache_ok = dev >= 0 && dev < kMaxCachedDevices;
  if (!cache_ok || !limit_set[collect][dev].load(std::memory_order_relaxed)) {
    if (collect) cudaFuncSetAttribute(k_qc_scan<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    else cudaFuncSetAttribute(k_qc_scan<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (cache_ok) limit_set[collect][dev].store(1, std::memory_order_relaxed);
  }
  int per_sm = 0;
  if (collect)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qc_scan<true>, kBlock, smem);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_qc_scan<false>, kBlock, smem);
  if (per_sm < 1) per_sm = 1;
  unsigned need = grid_for(T.n, kBlock / 32);
  unsigned grid = unsigned(dev_num_sms() * per_sm);
  if (grid > need) grid = need;
  if (collect) k_qc_scan<true><<<grid, kBlock, smem, s>>>(T, P, cfg, o);
  else k_qc_scan<false><<<grid, kBlock, smem, s>>>(T, P, cfg, o);
}
void launch_qc_keys(const DevPool& P, uint32_t w2mask, uint32_t m0, uint32_t nm, unsigned long long* keys,
                    cudaStream_t s) {
  const uint32_t n = nm * P.n;
  if (n) k_qc_keys<<<grid_for(n, 256), 256, 0, s>>>(P, w2mask, m0, nm, keys);
}
void launch_qc_entries(const DevPool& P, uint32_t w2mask, const unsigned long long* keys, uint32_t nv, uint32_t first,
                       uint32_t m0, uint32_t nm, uint32_t top_bits, uint4* entries, uint32_t* hash2, uint32_t* top,
                       uint32_t* flags, cudaStream_t s) {
  const uint32_t n = nm * nv;
  if (n) {
    k_qc_entries<<<grid_for(n, 256), 256, 0, s>>>(P, w2mask, keys, n, entries + first, hash2 + first);
    k_qc_check<<<grid_for(n, 256), 256, 0, s>>>(P, w2mask, keys, hash2 + first, n, flags);
  }
  const uint32_t nt = nm * ((1u << top_bits) + 1u);
  k_qc_top<<<grid_for(nt, 256), 256, 0, s>>>(keys, nv, first, m0, nm, top_bits, top);
}
void launch_qc_compact(const QCOut& q, uint32_t n, cudaStream_t s) {
  if (!n) return;
  k_qc_compact<<<grid_for(n, 256), 256, 0, s>>>(q, n);
}

void launch_qc_bucket(const DevTargets& T, const DevPool& P, const QCConfig& cfg, const QCIndex& ix,
                      const QCOut& o, bool collect, cudaStream_t s) {
  if (!T.n) return;
  static std::atomic<int> occ[3][kMaxCachedDevices];
  const bool keep = !collect && o.tmp;
  const int per_sm = collect ? blocks_per_sm(occ[1], k_qc_bucket<true, false>, kBlock, 0, 0)
                             : (keep ? blocks_per_sm(occ[2], k_qc_bucket<false, true>, kBlock, 0, 0)
                                     : blocks_per_sm(occ[0], k_qc_bucket<false, false>, kBlock, 0, 0));
  unsigned need = grid_for((T.n + 3u) / 4u, kBlock / 32);  // four targets per warp
  unsigned grid = unsigned(dev_num_sms() * per_sm);
  if (grid > need) grid = need;
  const unsigned lgrid = std::min<unsigned>(grid_for(T.n, 4), unsigned(dev_num_sms() * 4));
  if (collect) {
    k_qc_bucket<true, false><<<grid, kBlock, 0, s>>>(T, P, cfg, ix, o);
    k_qc_long<true, false><<<lgrid, 128, 0, s>>>(T, P, cfg, ix, o);
  } else if (keep) {
    k_qc_bucket<false, true><<<grid, kBlock, 0, s>>>(T, P, cfg, ix, o);
    k_qc_long<false, true><<<lgrid, 128, 0, s>>>(T, P, cfg, ix, o);
  } else {
    k_qc_bucket<false, false><<<grid, kBlock, 0, s>>>(T, P, cfg, ix, o);
    k_qc_long<false, false><<<lgrid, 128, 0, s>>>(T, P, cfg, ix, o);
  }
}
SweepArgs sweep_args(const RoundArgs& a) {
  SweepArgs w{};
  w.tinsn = a.T.insn;
  w.tlens = a.T.len;
  w.tlen = a.T.len ? 0u : a.T.fixed_len;
  w.tstride = a.T.stride;
  w.pinsn = a.P.insn;
  w.plens = a.P.lens;
  w.plen = a.P.lens ? 0u : a.P.len;
  w.pstride = a.P.stride;
  w.pairs = a.R.pairs;
  w.rejected = a.R.rejected;
  w.wend = a.R.wend;
  w.cdone = a.R.cdone;
  for (int c = 0; c < kClasses; c++) {
    w.cbase[c] = a.R.cbase[c];
    w.cpair[c] = a.R.cpair[c];
  }
  w.states = a.R.states;
  w.ctl = a.R.ctl;
  w.xunit = a.R.xunit;
  return w;
}
void launch_round_args(const RoundArgs& a, RoundArgs* dst, cudaStream_t s) { k_round_args<<<1, 256, 0, s>>>(a, dst); }
// The work of a round's kernels is known on the device only: grid-stride
// launches, of a few blocks for small jobs (whose rounds are launch latency)
// and of every SM's blocks for the others.
void launch_round_build(const RoundArgs* a, bool pair, bool small, cudaStream_t s) {
  const unsigned grid = small ? 32u : unsigned(dev_num_sms() * 8);
  if (pair) k_round_build<true><<<grid, 256, 0, s>>>(a);
  else k_round_build<false><<<grid, 256, 0, s>>>(a);
}
void launch_pair_plan(const RoundArgs* a, bool small, cudaStream_t s) {
  k_pair_plan<<<unsigned(dev_num_sms() * (small ? 4 : 16)), 128, 0, s>>>(a);
}
void launch_round_resolve(const RoundArgs* a, bool pair, bool small, cudaStream_t s) {
  const unsigned grid = small ? 32u : unsigned(dev_num_sms() * 8);
  if (pair) k_round_resolve<true><<<grid, 256, 0, s>>>(a);
  else k_round_resolve<false><<<grid, 256, 0, s>>>(a);
}
void launch_round_end(const RoundArgs* a, bool in_loop, cudaGraphConditionalHandle loop, cudaStream_t s) {
  if (in_loop) k_round_end<true><<<1, 32, 0, s>>>(a, loop);
  else k_round_end<false><<<1, 32, 0, s>>>(a, loop);
}
void launch_pairs_identity(uint32_t n, const RoundBuf& R, cudaStream_t s) {
  if (n) k_pairs_identity<<<grid_for(n, 256), 256, 0, s>>>(n, R);
}
void launch_pairs_from_survivors(const QCOut& q, const uint8_t* midpass, uint32_t lo, uint32_t hi,
                                 const uint32_t* surv_target, const RoundBuf& R, cudaStream_t s) {
  if (hi <= lo) return;
  k_pairs_from_survivors<<<grid_for(hi - lo, 256), 256, 0, s>>>(q, midpass, lo, hi, surv_target, R);
}
// Shared memory of a sweep kernel (bit-sliced classes): the candidate's
// output planes, one column of words per lane.
constexpr int exhaustive_smem(int cls) {
  return cls == 1 ? 0
                  : kBlock * (cls == 3 ? kCompactWords : (cls == 4 ? kWideWords : (cls == 5 ? kRegWords : kBitsWords))) * 4;
}
// Resident blocks per SM of a sweep kernel on the current device (its
// shared-memory limit raised first), cached per device.
template <int K, int CLS>
int exhaustive_blocks_per_sm() {
  constexpr int smem = exhaustive_smem(CLS);
  static std::atomic<int> occ[kMaxCachedDevices];
  return blocks_per_sm(occ, k_exhaustive<K, CLS>, kBlock, smem, smem);
}
template <int K, int CLS>
void launch_exhaustive_k(const SweepArgs& a, unsigned long long total, cudaStream_t s) {
  constexpr int smem = exhaustive_smem(CLS);
  const int per_sm = exhaustive_blocks_per_sm<K, CLS>();
  // resident blocks, or more when the chunks exceed kChunksPerWarp per warp
  const unsigned long long wpb = kBlock / 32;
  unsigned long long need = (total + wpb - 1) / wpb;
  unsigned long long grid = (unsigned long long)dev_num_sms() * per_sm;
  if (grid > need) grid = need;
  const unsigned long long cover = (total + wpb * kChunksPerWarp - 1) / (wpb * kChunksPerWarp);
  if (grid < cover) grid = cover;
  if (grid > 0x7FFFFFFFull) grid = 0x7FFFFFFFull;
  k_exhaustive<K, CLS><<<unsigned(grid), kBlock, smem, s>>>(a, kChunksPerWarp);
}

// The same kernel on a persistent grid (resident blocks on every SM) whose
// blocks take chunks until the class's total is spent.
template <int K, int CLS>
void launch_exhaustive_dev_k(const SweepArgs& a, cudaStream_t s) {
  constexpr int smem = exhaustive_smem(CLS);
  const int per_sm = exhaustive_blocks_per_sm<K, CLS>();
  const unsigned grid = unsigned(dev_num_sms() * per_sm);
  k_exhaustive<K, CLS><<<grid, kBlock, smem, s>>>(a, 0x7FFFFFFF);
}

int launch_exhaustive(const SweepArgs& a, const unsigned long long* alloc, int k, cudaStream_t s,
                      uint32_t* kernels) {
  int n = 0;
  uint32_t mask = 0;
  unsigned long long total[kClasses];
  for (int c = 0; c < kClasses; c++) total[c] = alloc[c] & kChunkMask;
  if (total[4]) {
    launch_exhaustive_k<1, 5>(a, total[4], s);
    mask |= kSweepRegs;
    n++;
  }
  if (total[3]) {
    launch_exhaustive_k<1, 4>(a, total[3], s);
    mask |= kSweepWide;
    n++;
  }
  if (total[2]) {
    launch_exhaustive_k<1, 3>(a, total[2], s);
    mask |= kSweepCompact;
    n++;
  }
  if (total[0]) {
    launch_exhaustive_k<1, 0>(a, total[0], s);
    mask |= kSweepBits;
    n++;
  }
  if (total[1]) {
    if (a.xunit == kXBitsBlocks) {
      launch_exhaustive_k<1, 2>(a, total[1], s);
      mask |= kSweepXBits;
    } else {
      switch (k) {
        case 1: launch_exhaustive_k<1, 1>(a, total[1], s); mask |= kSweepScalarK1; break;
        case 2: launch_exhaustive_k<2, 1>(a, total[1], s); mask |= kSweepScalarK1 << 1; break;
        case 8: launch_exhaustive_k<8, 1>(a, total[1], s); mask |= kSweepScalarK1 << 3; break;
        default: launch_exhaustive_k<4, 1>(a, total[1], s); mask |= kSweepScalarK1 << 2; break;
      }
    }
    n++;
  }
  if (kernels) *kernels |= mask;
  return n;
}

template <int K, int CLS>
void warm_exhaustive_k() {
  (void)exhaustive_blocks_per_sm<K, CLS>();
}
void warm_exhaustive_dev(bool compact, bool wide, uint32_t xunit, int k) {
  (void)dev_num_sms();
  if (wide) {
    warm_exhaustive_k<1, 4>();
    warm_exhaustive_k<1, 5>();
  }
  if (compact) warm_exhaustive_k<1, 3>();
  warm_exhaustive_k<1, 0>();
  if (xunit == kXBitsBlocks) warm_exhaustive_k<1, 2>();
  else if (k == 1) warm_exhaustive_k<1, 1>();
  else if (k == 2) warm_exhaustive_k<2, 1>();
  else if (k == 8) warm_exhaustive_k<8, 1>();
  else warm_exhaustive_k<4, 1>();
}

int launch_exhaustive_dev(const SweepArgs& a, bool compact, bool wide, int k, const cudaStream_t* ss) {
  int n = 0;
  if (wide) {
    launch_exhaustive_dev_k<1, 5>(a, ss[0]);
    launch_exhaustive_dev_k<1, 4>(a, ss[1]);
    n += 2;
  }
  if (compact) {
    launch_exhaustive_dev_k<1, 3>(a, ss[2]);
    n++;
  }
  launch_exhaustive_dev_k<1, 0>(a, ss[3]);
  const cudaStream_t sx = ss[4];
  if (a.xunit == kXBitsBlocks) {
    launch_exhaustive_dev_k<1, 2>(a, sx);
  } else {
    switch (k) {
      case 1: launch_exhaustive_dev_k<1, 1>(a, sx); break;
      case 2: launch_exhaustive_dev_k<2, 1>(a, sx); break;
      case 8: launch_exhaustive_dev_k<8, 1>(a, sx); break;
      default: launch_exhaustive_dev_k<4, 1>(a, sx); break;
    }
  }
  return n + 2;
}

void launch_report(const Tally* t, const QCOut& q, uint32_t n, const uint32_t* rbase, const uint32_t* rcnt, uint32_t nr,
                   const RoundCtl* ctl, Report* out, cudaStream_t s) {
  k_report<<<1, 64, 0, s>>>(t, q, n, rbase, rcnt, nr, ctl, out);
}
void launch_lanes_init(const Lanes& L, uint32_t n, cudaStream_t s) {
  if (n) k_lanes_init<<<grid_for(2 * n, 256), 256, 0, s>>>(L, 2 * n);
}
void launch_scan_small(const uint32_t* in, uint32_t* out, uint32_t n, cudaStream_t s) {
  if (n) k_scan_small<<<1, n > 1024 ? 1024 : (n + 31u) / 32u * 32u, 0, s>>>(in, out, n);
}
void launch_midcheck(const DevTargets& T, const DevPool& P, const uint32_t* surv,
                     const uint32_t* surv_target, uint32_t nsurv, uint8_t* pass, cudaStream_t s) {
  if (!nsurv) return;
  unsigned long long need = (unsigned long long)nsurv * 32;
  unsigned grid = unsigned(need / 256 + 1);
  unsigned cap = unsigned(dev_num_sms() * 8);
  if (grid > cap) grid = cap;
  k_midcheck<<<grid, 256, 0, s>>>(T, P, surv, surv_target, nsurv, pass);
}
void launch_surv_targets(const QCOut& q, uint32_t n, uint32_t* st, cudaStream_t s) {
  if (!n) return;
  k_surv_targets<<<grid_for(n, 256), 256, 0, s>>>(q, n, st);
}
void launch_rule_count_first(const Lanes& L, const Lanes& L2, uint32_t n, uint32_t* cnt, const DevTargets& T,
                             unsigned long long* checked, uint32_t pool_enum, unsigned long long pool2_enum,
                             cudaStream_t s) {
  if (!n) return;
  k_rule_count_first<<<grid_for(n, 256), 256, 0, s>>>(L, L2, n, cnt, T, checked, pool_enum, pool2_enum);
}
void launch_rule_write_first(const Lanes& L, const Lanes& L2, uint32_t n, const uint32_t* base, const TargetMeta* meta,
                             const DevPool& P, const DevPool& P2, DevRule* out, cudaStream_t s) {
  if (!n) return;
  k_rule_write_first<<<grid_for(n, 256), 256, 0, s>>>(L, L2, n, base, meta, P, P2, out);
}
void launch_rule_count_all(const RoundBuf& R, uint32_t npairs, uint32_t* flag, cudaStream_t s) {
  if (!npairs) return;
  k_rule_count_all<<<grid_for(npairs, 256), 256, 0, s>>>(R, npairs, flag);
}
void launch_rule_write_all(const uint32_t* flag, const uint32_t* base, uint32_t nsurv, const uint32_t* surv,
                           const uint16_t* sdiff, const uint32_t* surv_target, const TargetMeta* meta, const DevPool& P,
                           DevRule* out, cudaStream_t s) {
  if (!nsurv) return;
  k_rule_write_all<<<grid_for(nsurv, 256), 256, 0, s>>>(flag, base, nsurv, surv, sdiff, surv_target, meta, P, out);
}
void launch_verify_small(const uint32_t* tgt, const uint8_t* tlens, const uint32_t* cand,
                         const uint8_t* clens, uint32_t stride, uint32_t n, const uint8_t* dead,
                         uint32_t tiers, uint8_t* out, uint8_t* flagdiff, cudaStream_t s) {
  if (!n) return;
  unsigned grid = unsigned(((unsigned long long)n * 32 + 255) / 256);
  unsigned cap = unsigned(dev_num_sms() * 8);
  if (grid > cap) grid = cap;
  k_verify_small<<<grid, 256, 0, s>>>(tgt, tlens, cand, clens, stride, n, dead, tiers, out, flagdiff);
}

void launch_pair_keys(const DevPool& P, const uint4* out, const uint32_t* valid, uint32_t n, uint32_t dregs,
                      unsigned long long* keys, cudaStream_t s) {
  if (n) k_pair_keys<<<grid_for(n, 256), 256, 0, s>>>(P, out, valid, n, dregs, keys);
}
void launch_pair_heads(const uint4* out, const unsigned long long* keys, const uint32_t* members, uint32_t n,
                       uint32_t dregs, uint32_t* head, cudaStream_t s) {
  if (n) k_pair_heads<<<grid_for(n, 256), 256, 0, s>>>(out, keys, members, n, dregs, head);
}
void launch_pair_groups(const uint4* out, const unsigned long long* keys, const uint32_t* members, uint32_t n,
                        const uint32_t* gid, uint4* groups, cudaStream_t s) {
  if (n) k_pair_groups<<<grid_for(n, 256), 256, 0, s>>>(out, keys, members, n, gid, groups);
}
void launch_pair_top(const uint4* groups, uint32_t n_groups, uint32_t* top, cudaStream_t s) {
  k_pair_top<<<grid_for(kPairTop + 1, 256), 256, 0, s>>>(groups, n_groups, top);
}
void launch_pair_lanes_init(const DevTargets& T, const Lanes& L1, const QCOut& q1, const Lanes& L2,
                            const PairScan& ps, cudaStream_t s) {
  if (!T.n) return;
  k_pair_lanes_init<<<grid_for(T.n, 256), 256, 0, s>>>(T, L1, q1, L2, ps);
}
// All lanes of a large job: a warp each and no more blocks than that needs;
// the blocks retire as their lanes are done, which evens out the long walks.
// A small job's lanes, and the lanes that wait (their number is on the device,
// mostly none or few): a block each.
void launch_pair_scan(const RoundArgs* a, uint32_t n, bool all, bool small, cudaStream_t s) {
  if (all && !small) {
    if (n) k_pair_scan<1><<<grid_for(n, kBlock / 64), kBlock, 0, s>>>(a, true);
  } else {
    const unsigned most = unsigned(dev_num_sms() * (small ? 1 : 2));
    const unsigned grid = all ? std::min(2u * n, 4u * most) : most;
    if (grid) k_pair_scan<kScanWarps><<<grid, 32 * kScanWarps, 0, s>>>(a, all);
  }
}

}  // namespace z80b
