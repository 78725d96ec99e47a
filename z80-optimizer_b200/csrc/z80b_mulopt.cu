// z80b_mulopt.cu -- constant-multiply search kernels (cmd/mulopt on the
// device; see z80b_mulopt.cuh for the search rule).
//
// The instruction model (four inputs per word) is z80b_mul_ops.cuh.
//
// Layout of the walk: four inputs x travel together as the four bytes of
// one 32-bit word per register (byte 0: x = 1, byte 1: x = 2, byte 2:
// x = 255, byte 3: x = 127), with the carry in bit 0 of each byte, so one
// instruction of a sequence costs a few 32-bit integer operations for four
// inputs.  A warp takes 32 consecutive odometer prefixes (one per lane) and
// walks the same suffix tree in lock step, so every lane dispatches the same
// instruction at the same time; the last level is unrolled per pool.  A leaf
// is filtered by one shared-memory lookup: with k = A at x = 1, the table
// row of k holds the A that x = 2, 255, 127 must give (2k, -k, 127k) when k
// is a wanted constant, and an impossible value otherwise, so constants
// already solved at a shorter length (and k = 0, 1) cost nothing further.
// The table has one copy per lane (row k, column lane), so the lookups of a
// warp never share a bank.  Survivors get the whole warp: it runs the
// sequence on all 256 inputs (8 per lane).
//
// Bound by issue and short dependences (some 12 thread instructions per leaf);
// what helps is to walk less.  Long searches take their prefixes from the
// states that are new at each length (StateTable): for the 21-op pool 357,000
// of the 4.1M prefixes of length 5.  The suffixes leave out what another
// suffix replaces (z80b_mul_words.h: 4,710 of the 9,261 triples before the
// last instruction remain), and the last instruction is drawn from those that
// change A, one per effect on A (15 of 21), or that read what the triple left
// to be read.  250 constants over 21 ops to length 9: 283 ms walking every
// sequence, 13 to 14 ms so (22 ms with prefixes of length 6 and all suffixes
// of 3).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "z80b_mul_ops.cuh"
#include "z80b_mul_words.h"
#include "z80b_mulopt.cuh"

namespace z80b {
namespace mul {
namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
using namespace ops;

struct Params {
  int len, plen;                 // sequence length, prefix length (L = plen + D)
  unsigned long long n_prefix;   // N^plen
  unsigned long long nd;         // N^D
  uint32_t b, c, f;
  uint32_t want[8];
  int min_len;
  WordBufs words;
  const unsigned long long* reps;  // the prefixes' keys; null: all of them
  unsigned long long* best_all;  // [kMaxLen * 256]
  unsigned long long* best;      // [256] the row of this length
  LenStats* st;
};

struct Walk {
  uint32_t pidx;                 // this lane's prefix (odometer digits 0..plen-1)
  uint32_t pcost;
  bool active;
  const uint32_t* tab;           // shared expected-A table, this lane's column
  const Params* p;
  unsigned long long n_slow, n_full, n_pass;  // warp-level counters (lane 0 adds them)
};

__device__ __forceinline__ S4 initial_state(const Params& p) {
  S4 s;
  s.a = 0x7FFF0201u;  // x = 1, 2, 255, 127
  s.b = (p.b & 0xFFu) * M1;
  s.c = (p.c & 0xFFu) * M1;
  s.cf = (p.f & 1u) * M1;
  s.as = s.bs = s.cs = s.cfs = 0;
  return s;
}

// The whole sequence (prefix digits of pidx, suffix digits of sidx) on all
// 256 inputs, 8 per lane; true on every lane iff A = x*k for every x.
template <class P, int D>
__device__ bool full_check(const Params& p, uint32_t pidx, uint32_t sidx, uint32_t k) {
  const int lane = threadIdx.x & 31;
  int dg[16];
  uint32_t v = pidx;
  for (int i = p.plen - 1; i >= 0; i--) {
    dg[i] = int(v % P::N);
    v /= P::N;
  }
  v = sidx;
  for (int i = p.plen + D - 1; i >= p.plen; i--) {
    dg[i] = int(v % P::N);
    v /= P::N;
  }
  S4 s0 = initial_state(p), s1 = s0;
  const uint32_t x0 = 8u * lane;
  s0.a = (x0 | ((x0 + 1) << 8) | ((x0 + 2) << 16) | ((x0 + 3) << 24));
  s1.a = s0.a + 0x04040404u;
  for (int i = 0; i < p.len; i++) {
    apply_at<P>(dg[i], s0);
    apply_at<P>(dg[i], s1);
  }
  uint32_t e0 = 0, e1 = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    e0 |= (((x0 + j) * k) & 0xFFu) << (8 * j);
    e1 |= (((x0 + 4 + j) * k) & 0xFFu) << (8 * j);
  }
  return __all_sync(FULL, s0.a == e0 && s1.a == e1);
}

// Rare path: some lane of the warp has a leaf under this parent that passes
// the table filter.  Re-derives the N leaves and runs the full test on each
// passing leaf whose key beats the best so far, one at a time.
template <class P, int D>
__device__ __noinline__ void slow_parent(const S4& s, uint32_t sidx_parent, uint32_t scost_parent, Walk& w) {
  const Params& p = *w.p;
  const int lane = threadIdx.x & 31;
  if (lane == 0) w.n_slow++;
  for (int i = 0; i < P::N; i++) {
    S4 t = s;
    apply_at<P>(i, t);
    const uint32_t a = t.a;
    const uint32_t k = a & 0xFFu;
    const uint32_t sidx = sidx_parent * P::N + uint32_t(i);
    bool q = w.active && (a >> 8) == w.tab[k << 5];
    unsigned long long key = 0;
    if (q) {
      const unsigned long long cost = w.pcost + scost_parent + cost_of<P>(i);
      key = (cost << kKeyShift) | (uint64_t(w.pidx) * p.nd + sidx);
      q = key < *(volatile unsigned long long*)&p.best[k];
    }
    unsigned m = __ballot_sync(FULL, q);
    while (m) {
      const int j = __ffs(m) - 1;
      m &= m - 1;
      const uint32_t kj = __shfl_sync(FULL, k, j);
      const uint32_t pj = __shfl_sync(FULL, w.pidx, j);
      const unsigned long long keyj = __shfl_sync(FULL, key, j);
      if (lane == 0) w.n_full++;
      if (full_check<P, D>(p, pj, sidx, kj) && lane == 0) {
        w.n_pass++;
        atomicMin(&p.best[kj], keyj);
      }
    }
  }
}

// Instruction i as the last one: 0 when A keeps its value (the sequence
// without it is shorter and computes the same), else a number per effect on A.
__host__ __device__ constexpr int last_effect(Kind k) {
  switch (k) {
    case K_LD_BA: case K_LD_CA: case K_OR_A: case K_SCF: case K_CCF: case K_EXX: return 0;
    case K_SLA_A: return 1 + K_ADD_AA;
    case K_RLA: return 1 + K_ADC_AA;
    default: return 1 + k;
  }
}
// Whether a walk needs instruction i as the last one: it changes A and no
// other with its effect costs less or comes first at its cost.  Only where
// shorter sequences are searched too.
template <class P>
__host__ __device__ constexpr bool last_needed(int i) {
  const int e = last_effect(P::kind[i]);
  if (e == 0) return false;
  for (int j = 0; j < P::N; j++) {
    if (j == i || last_effect(P::kind[j]) != e) continue;
    const bool i8 = (P::t8 >> i) & 1u, j8 = (P::t8 >> j) & 1u;
    if (j8 < i8 || (j8 == i8 && j < i)) return false;
  }
  return true;
}

// The last instructions of class CLS.
template <class P, bool SHORTER, int CLS, int I>
__device__ __forceinline__ void leaves(const S4& s, const uint32_t* tab, bool& hit) {
  if constexpr (I < P::N) {
    constexpr Kind k = P::kind[I];
    constexpr bool in_class = CLS == kLeafAll || (CLS == kLeafB && words::reads_b(k)) ||
                              (CLS == kLeafC && words::reads_c(k)) || (CLS == kLeafCarry && words::reads_carry(k)) ||
                              (CLS == kLeafBCarry && words::reads_b(k) && words::reads_carry(k));
    if constexpr (!SHORTER || (last_needed<P>(I) && in_class)) {
      S4 t = s;
      apply<k>(t);
      hit |= (t.a >> 8) == tab[(t.a & 0xFFu) << 5];
    }
    leaves<P, SHORTER, CLS, I + 1>(s, tab, hit);
  }
}

// widx: the inner word so far, in base N.
template <class P, bool SHORTER, int LVL, int D>
__device__ __forceinline__ void walk(const S4& s, uint32_t widx, uint32_t scost, Walk& w, uint32_t mask) {
  if constexpr (LVL == D - 1) {
    const uint32_t cls = (SHORTER && D > 1) ? __ldg(&w.p->words.leaf[widx]) : uint32_t(kLeafAll);
    bool hit = false;
    if (cls == kLeafAll) leaves<P, SHORTER, kLeafAll, 0>(s, w.tab, hit);
    else if (cls == kLeafB) leaves<P, SHORTER, kLeafB, 0>(s, w.tab, hit);
    else if (cls == kLeafC) leaves<P, SHORTER, kLeafC, 0>(s, w.tab, hit);
    else if (cls == kLeafCarry) leaves<P, SHORTER, kLeafCarry, 0>(s, w.tab, hit);
    else leaves<P, SHORTER, kLeafBCarry, 0>(s, w.tab, hit);
    if (__any_sync(FULL, w.active && hit)) slow_parent<P, D>(s, widx, scost, w);
  } else {
#pragma unroll 1
    for (; mask; mask &= mask - 1) {
      const int i = __ffs(int(mask)) - 1;
      S4 t = s;
      apply_at<P>(i, t);
      const uint32_t next = widx * P::N + uint32_t(i);
      uint32_t m = 0;
      if constexpr (LVL + 2 < D) m = __ldg(&w.p->words.mask[(LVL == 0 ? 1 : 1 + P::N) + next]);
      walk<P, SHORTER, LVL + 1, D>(t, next, scost + cost_of<P>(i), w, m);
    }
  }
}

// The walk of one length.  SHORTER: every length below it is searched as
// well (min_len 1).
template <class P, int D, bool SHORTER>
__device__ __forceinline__ void search_length(const Params& p) {
  // Row k: the A of x = 2, 255, 127 (bytes 0..2) for a wanted k >= 2, else
  // all ones (no A >> 8 equals it); 32 copies of each row, one per lane.
  __shared__ uint32_t expect[256 * 32];
  __shared__ bool s_want[256];
  {
    // thread k: constant k is wanted and no shorter length has answered it
    const uint32_t k = threadIdx.x;
    bool wanted = k >= 2u && ((p.want[k >> 5] >> (k & 31u)) & 1u);
    for (int l = p.min_len; wanted && l < p.len; l++) wanted = p.best_all[l * 256 + int(k)] == kNoKey;
    s_want[k] = wanted;
    if (!__syncthreads_or(wanted)) return;
  }
  for (int i = threadIdx.x; i < 256 * 32; i += blockDim.x) {
    const uint32_t k = uint32_t(i) >> 5;
    expect[i] = s_want[k] ? (((2u * k) & 0xFFu) | (((0u - k) & 0xFFu) << 8) | (((127u * k) & 0xFFu) << 16))
                       : 0xFFFFFFFFu;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  // From two inner instructions on, a warp takes a group of 32 prefixes and
  // one first instruction, so that few prefixes still fill the SMs.
  constexpr bool kSplit = D >= 3;
  const uint32_t mask0 = D > 1 ? __ldg(&p.words.mask[0]) : 0u;
  const uint32_t nf = kSplit ? p.words.first_ops : 1u;
  const unsigned long long items = (p.n_prefix + 31) / 32 * nf;
  const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32);
  Walk w;
  w.tab = expect + lane;
  w.p = &p;
  w.n_slow = w.n_full = w.n_pass = 0;
  for (unsigned long long it = (unsigned long long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; it < items;
       it += warps) {
    const unsigned long long g = it / nf;
    uint32_t mask = mask0;
    if (kSplit) {
      for (uint32_t skip = uint32_t(it - g * nf); skip; skip--) mask &= mask - 1;
      mask &= 0u - mask;
    }
    const unsigned long long pi = g * 32 + lane;
    w.active = pi < p.n_prefix;
    w.pidx = !w.active ? 0u : (p.reps ? uint32_t(p.reps[pi]) : uint32_t(pi));
    // Prefix state: digit by digit, each pool instruction applied (warp-
    // uniformly) to the lanes whose digit it is.
    S4 s = initial_state(p);
    uint32_t pcost = 0;
    uint32_t pw = 1;
    for (int i = 1; i < p.plen; i++) pw *= P::N;
    for (int d = 0; d < p.plen; d++) {
      const int dgt = int((w.pidx / pw) % P::N);
      pw /= P::N;
      for (int i = 0; i < P::N; i++) {
        if (__any_sync(FULL, dgt == i)) {
          S4 t = s;
          apply_at<P>(i, t);
          if (dgt == i) s = t;
        }
      }
      pcost += cost_of<P>(dgt);
    }
    w.pcost = pcost;
    walk<P, SHORTER, 0, D>(s, 0u, 0u, w, mask);
  }
  if (lane == 0 && (w.n_slow | w.n_full | w.n_pass)) {
    atomicAdd(&p.st->filter_nodes, w.n_slow);
    atomicAdd(&p.st->full_checks, w.n_full);
    atomicAdd(&p.st->full_pass, w.n_pass);
  }
}

// Four blocks an SM (64 registers): the walk waits on table lookups and short
// dependences, and more warps cover them better than the registers that it
// spills (21 ops to length 9: 17.0 ms at two blocks, 15.6 at three, 14.7 at
// four, before the short lengths shared a launch).
template <class P, int D, bool SHORTER>
__global__ void __launch_bounds__(256, 4) k_mul_length(Params p) {
  search_length<P, D, SHORTER>(p);
}
// Lengths p.len .. p.len + gridDim.y - 1, all prefixes of one instruction
// less, side by side: each is a few microseconds of work behind as many of
// launch and set-up.  A length may look up constants that a shorter one finds
// meanwhile; the shorter answer stands.
template <class P, bool SHORTER>
__global__ void __launch_bounds__(256, 4) k_mul_short(Params p0) {
  __shared__ Params p;
  if (threadIdx.x == 0) {
    p = p0;
    p.len = p0.len + int(blockIdx.y);
    p.plen = p.len - 1;
    p.n_prefix = 1;
    for (int i = 0; i < p.plen; i++) p.n_prefix *= P::N;
    p.best = p0.best_all + 256 * p.len;
  }
  __syncthreads();
  search_length<P, 1, SHORTER>(p);
}

// ---- states (StateTable)

// Two words of inputs per lane: x = 8 lane .. 8 lane + 7.
struct Pair {
  S4 lo, hi;
};
__device__ __forceinline__ Pair all_inputs(const Params& p) {
  Pair s;
  s.lo = initial_state(p);
  s.hi = s.lo;
  const uint32_t x0 = 8u * (threadIdx.x & 31u);
  s.lo.a = x0 | ((x0 + 1) << 8) | ((x0 + 2) << 16) | ((x0 + 3) << 24);
  s.hi.a = s.lo.a + 0x04040404u;
  return s;
}
template <class P>
__device__ __forceinline__ void run_digits(Pair& s, uint32_t idx, int len) {
  uint32_t pw = 1;
  for (int i = 1; i < len; i++) pw *= P::N;
  for (int i = 0; i < len; i++) {
    const int d = int((idx / pw) % P::N);
    pw /= P::N;
    apply_at<P>(d, s.lo);
    apply_at<P>(d, s.hi);
  }
}
// Hash of the state on all 256 inputs, the same in every lane (the multipliers
// are splitmix64's).  salt: 0, or the level where states of different levels are
// kept apart.
__device__ __forceinline__ unsigned long long state_hash(const Pair& s, uint32_t salt) {
  const uint32_t w[14] = {s.lo.a, s.lo.b, s.lo.c, s.lo.as, s.lo.bs, s.lo.cs, s.lo.cf | (s.lo.cfs << 1),
                          s.hi.a, s.hi.b, s.hi.c, s.hi.as, s.hi.bs, s.hi.cs, s.hi.cf | (s.hi.cfs << 1)};
  unsigned long long h = (threadIdx.x & 31u) * 0xD6E8FEB86659FD93ull + salt;
#pragma unroll
  for (int i = 0; i < 14; i++) {
    h = (h ^ w[i]) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 32;
  }
  h *= 0xBF58476D1CE4E5B9ull;
  h ^= h >> 29;
#pragma unroll
  for (int o = 16; o; o >>= 1) h += __shfl_xor_sync(FULL, h, o);
  return h ? h : 1ull;
}
__device__ __forceinline__ bool same_state(const Pair& x, const Pair& y) {
  const uint32_t d = (x.lo.a ^ y.lo.a) | (x.lo.b ^ y.lo.b) | (x.lo.c ^ y.lo.c) | (x.lo.as ^ y.lo.as) |
                     (x.lo.bs ^ y.lo.bs) | (x.lo.cs ^ y.lo.cs) | (x.lo.cf ^ y.lo.cf) | (x.lo.cfs ^ y.lo.cfs) |
                     (x.hi.a ^ y.hi.a) | (x.hi.b ^ y.hi.b) | (x.hi.c ^ y.hi.c) | (x.hi.as ^ y.hi.as) |
                     (x.hi.bs ^ y.hi.bs) | (x.hi.cs ^ y.hi.cs) | (x.hi.cf ^ y.hi.cf) | (x.hi.cfs ^ y.hi.cfs);
  return __all_sync(FULL, d == 0);
}
// The slot of hash h: its own, or (enter) the first free one, taken.  The
// table is at most half full; the bound only guards against a wrong size.
template <bool ENTER>
__device__ __forceinline__ unsigned long long find_slot(const StateTable& t, unsigned long long h) {
  unsigned long long i = (h ^ (h >> 32)) & t.mask;
  for (unsigned long long n = 0; n <= t.mask; n++, i = (i + 1) & t.mask) {
    const unsigned long long v = ENTER ? atomicCAS(&t.hash[i], 0ull, h) : t.hash[i];
    if (v == h || (ENTER && v == 0)) return i;
  }
  return 0;
}
template <class P>
__device__ __forceinline__ unsigned long long child_key(unsigned long long key, int level, int i) {
  const unsigned long long cost = ((key >> kKeyShift) & 0xFFFull) + cost_of<P>(i);
  return (unsigned long long)(level + 1) << kLevelShift | cost << kKeyShift | ((key & kIndexMask) * P::N + unsigned(i));
}
template <class P, int I>
__device__ __forceinline__ void hash_children(const Pair& s, uint32_t salt, unsigned long long& mine) {
  if constexpr (I < P::N) {
    Pair t = s;
    apply<P::kind[I]>(t.lo);
    apply<P::kind[I]>(t.hi);
    const unsigned long long h = state_hash(t, salt);
    if ((threadIdx.x & 31u) == I) mine = h;
    hash_children<P, I + 1>(s, salt, mine);
  }
}

__global__ void k_mul_root(Params p, unsigned long long* hash, unsigned long long* key) {
  const unsigned long long h = state_hash(all_inputs(p), 0u);
  if (threadIdx.x == 0) {
    *hash = h;
    *key = 0;
  }
}
__global__ void k_mul_enter(StateTable t, const unsigned long long* __restrict__ hash,
                            const unsigned long long* __restrict__ key, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicMin(&t.key[find_slot<true>(t, hash[i])], key[i]);
}
// Warp per prefix: its state from its digits, then each child's hash; lane i
// enters child i.  Bound by issue (about 120 warp instructions per child).
template <class P>
__global__ void __launch_bounds__(256) k_mul_children(Params p, StateTable t, const unsigned long long* __restrict__ key,
                                                      uint32_t n, int level, uint32_t salt,
                                                      unsigned long long* __restrict__ child_hash) {
  const uint32_t lane = threadIdx.x & 31u, nw = gridDim.x * (blockDim.x >> 5);
  for (uint32_t j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); j < n; j += nw) {
    const unsigned long long k = key[j];
    Pair s = all_inputs(p);
    run_digits<P>(s, uint32_t(k), level);
    unsigned long long h = 0;
    hash_children<P, 0>(s, salt, h);
    if (lane < P::N) {
      child_hash[(size_t)j * P::N + lane] = h;
      atomicMin(&t.key[find_slot<true>(t, h)], child_key<P>(k, level, int(lane)));
    }
  }
}
// Warp per prefix, lane i its child i: children that hold their slot are the
// next level's prefixes; each of the others is run beside its slot's holder,
// so that equal hashes are known to be equal states.
template <class P>
__global__ void __launch_bounds__(256) k_mul_select(Params p, StateTable t, const unsigned long long* __restrict__ key,
                                                    uint32_t n, int level,
                                                    const unsigned long long* __restrict__ child_hash,
                                                    unsigned long long* __restrict__ out_hash,
                                                    unsigned long long* __restrict__ out_key,
                                                    uint32_t* __restrict__ count) {
  const uint32_t lane = threadIdx.x & 31u, nw = gridDim.x * (blockDim.x >> 5);
  for (uint32_t j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); j < n; j += nw) {
    const unsigned long long k = key[j];
    unsigned long long h = 0, mine = 0, holder = 0;
    if (lane < P::N) {
      h = child_hash[(size_t)j * P::N + lane];
      mine = child_key<P>(k, level, int(lane));
      holder = t.key[find_slot<false>(t, h)];
    }
    const unsigned rep = __ballot_sync(FULL, lane < P::N && holder == mine);
    uint32_t at = 0;
    if (lane == 0 && rep) at = atomicAdd(&count[0], uint32_t(__popc(rep)));
    at = __shfl_sync(FULL, at, 0);
    if ((rep >> lane) & 1u) {
      const uint32_t o = at + __popc(rep & ((1u << lane) - 1u));
      out_hash[o] = h;
      out_key[o] = mine;
    }
    unsigned others = __ballot_sync(FULL, lane < P::N && holder != mine);
    if (!others) continue;
    Pair s = all_inputs(p);
    run_digits<P>(s, uint32_t(k), level);
    for (; others; others &= others - 1) {
      const int i = __ffs(others) - 1;
      Pair x = s, y = all_inputs(p);
      apply_at<P>(i, x.lo);
      apply_at<P>(i, x.hi);
      const unsigned long long ok = __shfl_sync(FULL, holder, i);
      run_digits<P>(y, uint32_t(ok), int(ok >> kLevelShift));
      if (!same_state(x, y) && lane == 0) count[1] = 1;
    }
  }
}

// Resident blocks per SM of a walk kernel, asked once per device.
template <class P, int D, bool SHORTER>
int walk_blocks_per_sm() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  if (dev < 64) {
    const int c = cache[dev].load(std::memory_order_relaxed);
    if (c) return c;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_mul_length<P, D, SHORTER>, 256, 0) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  if (dev < 64) cache[dev].store(per_sm, std::memory_order_relaxed);
  return per_sm;
}
template <class P, int D, bool SHORTER>
cudaError_t launch_walk(const Params& prm, int sms, cudaStream_t stream) {
  const unsigned long long need = ((prm.n_prefix + 31) / 32 * (D >= 3 ? prm.words.first_ops : 1u) + 7) / 8;
  const unsigned long long blocks = std::min<unsigned long long>(
      (unsigned long long)sms * walk_blocks_per_sm<P, D, SHORTER>(), std::max(need, 1ull));
  k_mul_length<P, D, SHORTER><<<unsigned(blocks), 256, 0, stream>>>(prm);
  return cudaGetLastError();
}
template <class P, bool SHORTER>
cudaError_t launch_depth(const Params& prm, int D, int sms, cudaStream_t stream) {
  switch (D) {
    case 1: return launch_walk<P, 1, SHORTER>(prm, sms, stream);
    case 2: return launch_walk<P, 2, SHORTER>(prm, sms, stream);
    case 3: return launch_walk<P, 3, SHORTER>(prm, sms, stream);
    default: return launch_walk<P, 4, SHORTER>(prm, sms, stream);
  }
}

const char* const kNamesGo[] = {"ADD A,A", "ADD A,B", "SUB B",   "LD B,A",  "SLA A",   "SRL A", "EX AF,AF'",
                                "EXX",     "ADC A,B", "ADC A,A", "SBC A,B", "SBC A,A", "OR A",  "NEG"};
const uint8_t kTGo[] = {4, 4, 4, 4, 8, 8, 4, 4, 4, 4, 4, 4, 4, 8};
const char* const kNamesWide[] = {"ADD A,A", "ADD A,B", "SUB B", "LD B,A", "SLA A",     "SRL A",  "RLA",
                                  "RRA",     "RLCA",    "RRCA",  "NEG",    "CPL",       "OR A",   "SCF",
                                  "CCF",     "EX AF,AF'", "LD C,A", "ADD A,C", "SUB C", "LD A,B", "LD A,C"};
const uint8_t kTWide[] = {4, 4, 4, 4, 8, 8, 4, 4, 4, 4, 8, 4, 4, 4, 4, 4, 4, 4, 4, 4, 4};
const char* const kNamesFast[] = {"ADD A,A", "ADD A,B", "SUB B", "LD B,A", "ADC A,B", "ADC A,A", "SBC A,B",
                                  "SBC A,A", "SRL A",   "RLA",   "RRA",    "RLCA",    "RRCA",    "NEG"};
const uint8_t kTFast[] = {4, 4, 4, 4, 4, 4, 4, 4, 8, 4, 4, 4, 4, 8};
const char* const kNamesCuda[] = {"ADD A,A", "ADD A,B", "SUB B", "LD B,A", "ADC A,B", "ADC A,A", "SBC A,B",
                                  "SBC A,A", "SLA A",   "SRA A", "SRL A",  "RLA",     "RRA",     "RLCA",
                                  "RRCA",    "RLC A",   "RRC A", "OR A",   "NEG",     "SCF",     "EX AF,AF'"};
const uint8_t kTCuda[] = {4, 4, 4, 4, 4, 4, 4, 4, 8, 8, 8, 4, 4, 4, 4, 8, 8, 4, 8, 4, 4};

// Longest length whose odometer index N^L stays below 2^48.
constexpr int max_len_for(int n) {
  int l = 0;
  unsigned long long v = 1;
  while (v * n < (1ull << kKeyShift)) {
    v *= n;
    l++;
  }
  return l;
}

const PoolInfo kInfo[kNumPools] = {{14, max_len_for(14), kNamesGo, kTGo},
                                   {21, max_len_for(21), kNamesWide, kTWide},
                                   {14, max_len_for(14), kNamesFast, kTFast},
                                   {21, max_len_for(21), kNamesCuda, kTCuda}};

// Split of length L into a prefix walked per lane and a suffix of D levels:
// prefixes for some 4,000 warps when L allows (a prefix costs as much as
// some hundred leaves, so no more than that), D <= kMaxInner + 1.
void split(int n, int len, int* plen, int* d) {
  int pt = 0;
  unsigned long long v = 1;
  while (v < (1ull << 17)) {
    v *= n;
    pt++;
  }
  int p = len - 1 < pt ? len - 1 : pt;
  int dd = len - p;
  if (dd > kMaxInner + 1) {
    dd = kMaxInner + 1;
    p = len - dd;
  }
  *plen = p;
  *d = dd;
}

Params params_of(const SearchArgs& a) {
  Params p{};
  p.b = a.b;
  p.c = a.c;
  p.f = a.f;
  p.min_len = a.min_len;
  for (int i = 0; i < 8; i++) p.want[i] = a.want[i];
  return p;
}
// Where not every shorter length is searched, a state of a shorter prefix
// does not replace that of a longer one: the levels' hashes are kept apart.
uint32_t salt_of(const SearchArgs& a, int level) { return a.min_len > 1 ? uint32_t(level) : 0u; }

template <class F>
auto with_pool(int pool, F f) {
  switch (pool) {
    case kPoolGo: return f(PGo{});
    case kPoolWide: return f(PWide{});
    case kPoolFast: return f(PFast{});
    default: return f(PCuda{});
  }
}
unsigned warp_grid(uint32_t n, int sms) { return unsigned(std::max(1u, std::min((n + 7u) / 8u, unsigned(sms) * 8u))); }

}  // namespace

const PoolInfo& pool_info(int pool) { return kInfo[pool]; }

WordImage word_image(int pool, int n, bool shorter) {
  const WordTable t = with_pool(pool, [&](auto P) { return word_table<decltype(P)>(n, shorter); });
  WordImage im;
  for (int l = 0; l < n; l++) im.mask.insert(im.mask.end(), t.mask[l].begin(), t.mask[l].end());
  im.leaf = t.leaf;
  im.first_ops = n ? uint32_t(__builtin_popcount(t.mask[0][0])) : 0u;
  return im;
}
int plain_suffix(int pool, int len) {
  int p = 0, d = 0;
  split(kInfo[pool].n, len, &p, &d);
  return d;
}

cudaError_t launch_length(const SearchArgs& a, int len, const unsigned long long* reps, uint32_t n_reps, int rep_len,
                          const WordBufs& words, unsigned long long* best, LenStats* st, int sms, cudaStream_t stream) {
  const PoolInfo& pi = kInfo[a.pool];
  Params p = params_of(a);
  p.len = len;
  int D = 1;
  if (reps) {
    p.plen = rep_len;
    D = len - rep_len;
    p.n_prefix = n_reps;
  } else {
    split(pi.n, len, &p.plen, &D);
    p.n_prefix = 1;
    for (int i = 0; i < p.plen; i++) p.n_prefix *= pi.n;
  }
  p.nd = 1;
  for (int i = 0; i < D; i++) p.nd *= pi.n;
  p.words = words;
  p.reps = reps;
  p.best_all = best;
  p.best = best + 256 * len;
  p.st = st;
  return with_pool(a.pool, [&](auto P) {
    return a.min_len == 1 ? launch_depth<decltype(P), true>(p, D, sms, stream)
                          : launch_depth<decltype(P), false>(p, D, sms, stream);
  });
}

cudaError_t launch_short(const SearchArgs& a, int first, int n, unsigned long long* best, LenStats* st, int sms,
                         cudaStream_t stream) {
  Params p = params_of(a);
  p.len = first;
  p.nd = unsigned(kInfo[a.pool].n);
  p.best_all = best;
  p.st = st;
  double prefixes = 1;
  for (int i = 0; i < first + n - 2; i++) prefixes *= kInfo[a.pool].n;
  const dim3 grid(unsigned(std::max(1.0, std::min(prefixes / 256.0 + 1.0, double(sms)))), unsigned(n));
  return with_pool(a.pool, [&](auto P) {
    if (a.min_len == 1) k_mul_short<decltype(P), true><<<grid, 256, 0, stream>>>(p);
    else k_mul_short<decltype(P), false><<<grid, 256, 0, stream>>>(p);
    return cudaGetLastError();
  });
}

cudaError_t launch_root(const SearchArgs& a, unsigned long long* hash, unsigned long long* key, cudaStream_t stream) {
  k_mul_root<<<1, 32, 0, stream>>>(params_of(a), hash, key);
  return cudaGetLastError();
}
cudaError_t launch_enter(const StateTable& t, const unsigned long long* hash, const unsigned long long* key, uint32_t n,
                         cudaStream_t stream) {
  if (!n) return cudaSuccess;
  k_mul_enter<<<(n + 255) / 256, 256, 0, stream>>>(t, hash, key, n);
  return cudaGetLastError();
}
cudaError_t launch_children(const SearchArgs& a, const StateTable& t, const unsigned long long* key, uint32_t n,
                            int level, unsigned long long* child_hash, int sms, cudaStream_t stream) {
  if (!n) return cudaSuccess;
  return with_pool(a.pool, [&](auto P) {
    k_mul_children<decltype(P)><<<warp_grid(n, sms), 256, 0, stream>>>(params_of(a), t, key, n, level,
                                                                       salt_of(a, level + 1), child_hash);
    return cudaGetLastError();
  });
}
cudaError_t launch_select(const SearchArgs& a, const StateTable& t, const unsigned long long* key, uint32_t n, int level,
                          const unsigned long long* child_hash, unsigned long long* out_hash,
                          unsigned long long* out_key, uint32_t* count, int sms, cudaStream_t stream) {
  if (!n) return cudaSuccess;
  return with_pool(a.pool, [&](auto P) {
    k_mul_select<decltype(P)><<<warp_grid(n, sms), 256, 0, stream>>>(params_of(a), t, key, n, level, child_hash,
                                                                     out_hash, out_key, count);
    return cudaGetLastError();
  });
}

}  // namespace mul
}  // namespace z80b
