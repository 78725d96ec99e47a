// z80b_mul_words.h -- which suffixes the constant-multiply walk needs (host).
//
// A walk appends every suffix of d instructions to each of its prefixes.  A
// suffix w can be left out for every prefix when another one computes the
// same from every state and gives the smaller key (shortest, then fewest
// T-states, then first in odometer order): most pairs and triples of
// instructions have such a partner (LD B,A : LD C,A and its mirror image,
// a carry instruction before one that overwrites the carry, SLA A for
// ADD A,A).  "The same" is decided on names of values: each register holds the
// name of an input or of an expression over names, two equal names are equal
// values whatever the inputs are, and the rules that make names equal
// (x + x is a doubling, NOT NOT x is x, ...) hold for all byte values.  Only
// A counts after the last instruction, so a register or carry written in the
// last steps has to be read by it.
//
// Inner words (the first n = d - 1 instructions of the suffix) are kept as a
// tree of masks, one bit per next instruction; a word's class says which last
// instructions can follow it.
#pragma once
#include <array>
#include <cstdint>
#include <map>
#include <utility>
#include <vector>

#include "z80b_mul_ops.cuh"

namespace z80b {
namespace mul {

enum LeafClass : uint8_t { kLeafNone = 0, kLeafAll = 1, kLeafB = 2, kLeafC = 3, kLeafCarry = 4, kLeafBCarry = 5 };

struct WordTable {
  // level l < n: one mask per word of l instructions (index in base N); then
  // the classes of the words of n instructions
  std::vector<uint32_t> mask[3];
  std::vector<uint8_t> leaf;
};

namespace words {

// Names of values: interned expressions.
class Names {
 public:
  enum Form : int { kVar, kConst, kDbl, kTop, kAdd, kCAdd, kSub, kCSub, kAdc, kCAdc, kSbc, kCSbc, kShlC, kMask, kShr,
                    kLow, kSra, kShrC, kRol, kRor, kNeg, kCNeg, kNot, kNotC };
  int get(int f, int a = -1, int b = -1, int c = -1) {
    auto r = ids_.emplace(std::array<int, 4>{f, a, b, c}, int(ids_.size()));
    if (r.second) forms_.push_back({f, a, b, c});
    return r.first->second;
  }
  int zero() { return get(kConst, 0); }
  int one() { return get(kConst, 1); }  // a set carry
  bool is(int id, int f) const { return forms_[size_t(id)][0] == f; }
  int arg(int id) const { return forms_[size_t(id)][1]; }
  int unary(int f, int x, int inverse) { return is(x, inverse) ? arg(x) : get(f, x); }
  int sorted(int f, int x, int y, int c = -1) { return x <= y ? get(f, x, y, c) : get(f, y, x, c); }

 private:
  std::map<std::array<int, 4>, int> ids_;
  std::vector<std::array<int, 4>> forms_;
};

struct State {  // names
  int a, b, c, as, bs, cs, cf, cfs;
  std::array<int, 8> key() const { return {a, b, c, as, bs, cs, cf, cfs}; }
};

inline void step(Names& n, State& s, ops::Kind k) {
  using namespace ops;
  using N = Names;
  const int a = s.a;
  auto add = [&](int y) {
    s.a = a == y ? n.get(N::kDbl, a) : n.sorted(N::kAdd, a, y);
    s.cf = a == y ? n.get(N::kTop, a) : n.sorted(N::kCAdd, a, y);
  };
  auto sub = [&](int y) {
    s.a = a == y ? n.zero() : n.get(N::kSub, a, y);
    s.cf = a == y ? n.zero() : n.get(N::kCSub, a, y);
  };
  auto rla = [&] {
    s.a = s.cf == n.zero() ? n.get(N::kDbl, a) : n.get(N::kShlC, a, s.cf);
    s.cf = n.get(N::kTop, a);
  };
  switch (k) {
    case K_ADD_AA: case K_SLA_A: add(a); break;
    case K_ADD_AB: add(s.b); break;
    case K_ADD_AC: add(s.c); break;
    case K_SUB_B: sub(s.b); break;
    case K_SUB_C: sub(s.c); break;
    case K_LD_BA: s.b = a; break;
    case K_LD_CA: s.c = a; break;
    case K_LD_AB: s.a = s.b; break;
    case K_LD_AC: s.a = s.c; break;
    case K_ADC_AB:
      if (s.cf == n.zero()) add(s.b);
      else if (a == s.b) rla();
      else {
        const int c = s.cf;
        s.cf = n.sorted(N::kCAdc, a, s.b, c);
        s.a = n.sorted(N::kAdc, a, s.b, c);
      }
      break;
    case K_ADC_AA: case K_RLA: rla(); break;
    case K_SBC_AB:
      if (s.cf == n.zero()) sub(s.b);
      else {
        const int c = s.cf;
        s.cf = n.get(N::kCSbc, a, s.b, c);
        s.a = n.get(N::kSbc, a, s.b, c);
      }
      break;
    case K_SBC_AA: s.a = s.cf == n.zero() ? n.zero() : n.get(N::kMask, s.cf); break;
    case K_SRA_A: s.a = n.get(N::kSra, a); s.cf = n.get(N::kLow, a); break;
    case K_SRL_A: s.a = n.get(N::kShr, a); s.cf = n.get(N::kLow, a); break;
    case K_RRA:
      s.a = s.cf == n.zero() ? n.get(N::kShr, a) : n.get(N::kShrC, a, s.cf);
      s.cf = n.get(N::kLow, a);
      break;
    case K_RLCA: s.a = n.unary(N::kRol, a, N::kRor); s.cf = n.get(N::kTop, a); break;
    case K_RRCA: s.a = n.unary(N::kRor, a, N::kRol); s.cf = n.get(N::kLow, a); break;
    case K_NEG: s.a = n.unary(N::kNeg, a, N::kNeg); s.cf = n.get(N::kCNeg, a); break;
    case K_CPL: s.a = n.unary(N::kNot, a, N::kNot); break;
    case K_OR_A: s.cf = n.zero(); break;
    case K_SCF: s.cf = n.one(); break;
    case K_CCF: s.cf = s.cf == n.zero() ? n.one() : (s.cf == n.one() ? n.zero() : n.unary(N::kNotC, s.cf, N::kNotC)); break;
    case K_EX_AF: std::swap(s.a, s.as); std::swap(s.cf, s.cfs); break;
    case K_EXX: std::swap(s.b, s.bs); std::swap(s.c, s.cs); break;
  }
}

Z80B_MUL_HD constexpr bool reads_b(ops::Kind k) {
  using namespace ops;
  return k == K_ADD_AB || k == K_SUB_B || k == K_LD_AB || k == K_ADC_AB || k == K_SBC_AB || k == K_EXX;
}
Z80B_MUL_HD constexpr bool reads_c(ops::Kind k) {
  using namespace ops;
  return k == K_ADD_AC || k == K_SUB_C || k == K_LD_AC || k == K_EXX;
}
Z80B_MUL_HD constexpr bool reads_carry(ops::Kind k) {
  using namespace ops;
  return k == K_ADC_AB || k == K_ADC_AA || k == K_SBC_AB || k == K_SBC_AA || k == K_RLA || k == K_RRA || k == K_CCF ||
         k == K_EX_AF;
}
Z80B_MUL_HD constexpr bool writes_carry(ops::Kind k) {
  using namespace ops;
  switch (k) {
    case K_LD_BA: case K_LD_CA: case K_LD_AB: case K_LD_AC: case K_SBC_AA: case K_CPL: case K_EX_AF: case K_EXX: return false;
    default: return true;
  }
}

}  // namespace words

// The inner words of n instructions (n = 0..3) that a walk needs.  shorter:
// every shorter length is searched as well, so a word that a shorter one
// replaces, or that writes a register or the carry (by an instruction that
// does nothing else) which is not read before the end, is left out; otherwise
// only words that another of their length replaces are.
template <class P>
WordTable word_table(int n, bool shorter) {
  using namespace words;
  Names names;
  auto var = [&](int i) { return names.get(Names::kVar, i); };
  const State start{var(0), var(1), var(2), var(3), var(4), var(5), var(6), var(7)};
  names.zero();
  names.one();
  // the smallest (length, cost, index) of each state
  struct Best {
    int len;
    uint32_t cost, idx;
  };
  std::map<std::array<int, 8>, Best> best;
  best[start.key()] = Best{0, 0, 0};
  std::vector<State> cur{start};
  std::vector<uint32_t> cost{0};
  std::vector<std::vector<uint8_t>> kept;  // [l - 1][word]
  for (int l = 1; l <= n; l++) {
    if (!shorter) best.clear();
    std::vector<State> next;
    std::vector<uint32_t> nc;
    for (size_t w = 0; w < cur.size(); w++)
      for (int i = 0; i < P::N; i++) {
        State s = cur[w];
        step(names, s, P::kind[i]);
        next.push_back(s);
        nc.push_back(cost[w] + ops::cost_of<P>(i));
        const Best b{l, nc.back(), uint32_t(next.size() - 1)};
        auto it = best.emplace(s.key(), b).first;
        if (it->second.len == l && b.cost < it->second.cost) it->second = b;
      }
    cur.swap(next);
    cost.swap(nc);
    // the words of this level that are their state's smallest
    kept.emplace_back(cur.size());
    for (size_t w = 0; w < cur.size(); w++) {
      const Best& b = best.at(cur[w].key());
      kept.back()[w] = b.len == l && b.idx == w;
    }
  }
  WordTable t;
  size_t size = 1;
  for (int l = 0; l < n; l++) {
    t.mask[l].assign(size, 0u);
    size *= P::N;
  }
  t.leaf.assign(size, uint8_t(kLeafNone));
  for (size_t w = 0; w < size; w++) {
    // every beginning of the word is needed itself (a word that begins with a
    // replaceable one is replaceable)
    int digit[3];
    size_t v = w;
    for (int i = n - 1; i >= 0; i--) {
      digit[i] = int(v % P::N);
      v /= P::N;
    }
    bool ok = true;
    size_t prefix = 0;
    for (int i = 0; i < n; i++) {
      prefix = prefix * P::N + size_t(digit[i]);
      ok = ok && kept[size_t(i)][prefix];
    }
    if (!ok) continue;
    uint8_t leaf = kLeafAll;
    if (shorter) {
      bool b = false, c = false, carry = false;  // written and not read since
      for (int i = 0; i < n && ok; i++) {
        const ops::Kind k = P::kind[digit[i]];
        if (reads_b(k)) b = false;
        if (reads_c(k)) c = false;
        if (reads_carry(k)) carry = false;
        if ((k == ops::K_LD_BA && b) || (k == ops::K_LD_CA && c) || (writes_carry(k) && carry)) ok = false;
        if (k == ops::K_LD_BA) b = true;
        if (k == ops::K_LD_CA) c = true;
        if (k == ops::K_OR_A || k == ops::K_SCF || k == ops::K_CCF) carry = true;
      }
      // the last instruction has to read what is left: B and the carry (ADC,
      // SBC A,B), or one of the three
      if (!ok || (c && (b || carry))) continue;
      if (b) leaf = carry ? kLeafBCarry : kLeafB;
      else if (c) leaf = kLeafC;
      else if (carry) leaf = kLeafCarry;
    }
    t.leaf[w] = leaf;
    prefix = 0;
    for (int i = 0; i < n; i++) {
      t.mask[i][prefix] |= 1u << digit[i];
      prefix = prefix * P::N + size_t(digit[i]);
    }
  }
  return t;
}

}  // namespace mul
}  // namespace z80b
