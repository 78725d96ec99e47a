// Host check of the constant-multiply walk's suffix tables
// (z80b_mul_words.h), per pool, against every suffix run on random states
// (four per word, 24 words).  For n inner instructions and one last one:
// (1) shorter lengths searched: for every effect on A that some suffix of at
// most n + 1 instructions has, the smallest (length, T-states, index) suffix
// with it is among those the tables keep, at its own length.
// (2) otherwise: the same within the suffixes of n + 1 instructions.
#include <cstdio>
#include <map>
#include <random>
#include <tuple>
#include <vector>

#include "../../z80-optimizer_b200/csrc/z80b_mul_words.h"

using namespace z80b::mul;
using namespace z80b::mul::ops;

constexpr int kSamples = 24;
struct Sample {
  S4 w[kSamples];
};
typedef std::vector<uint32_t> Sig;

template <class P>
static bool keeps(const WordTable& t, int n, bool shorter, uint32_t word, int last) {
  uint32_t div = 1;
  for (int i = 0; i < n; i++) div *= P::N;
  uint32_t prefix = 0;
  for (int l = 0; l < n; l++) {
    div /= P::N;
    const uint32_t d = word / div % P::N;
    if (!((t.mask[l][prefix] >> d) & 1u)) return false;
    prefix = prefix * P::N + d;
  }
  const Kind k = P::kind[last];
  switch (t.leaf[word]) {
    case kLeafNone: return false;
    case kLeafB: return !shorter || words::reads_b(k);
    case kLeafC: return !shorter || words::reads_c(k);
    case kLeafCarry: return !shorter || words::reads_carry(k);
    case kLeafBCarry: return !shorter || (words::reads_b(k) && words::reads_carry(k));
    default: return true;
  }
}

template <class P>
static int check(const char* name, int max_n) {
  std::mt19937_64 rng(17);
  Sample s0;
  for (S4& s : s0.w) {
    s.a = uint32_t(rng());
    s.b = uint32_t(rng());
    s.c = uint32_t(rng());
    s.as = uint32_t(rng());
    s.bs = uint32_t(rng());
    s.cs = uint32_t(rng());
    s.cf = uint32_t(rng()) & M1;
    s.cfs = uint32_t(rng()) & M1;
  }
  auto a_of = [](const Sample& s) {
    Sig g(kSamples);
    for (int i = 0; i < kSamples; i++) g[size_t(i)] = s.w[i].a;
    return g;
  };
  // effect on A -> smallest (length, T-states, index) over the lengths so far
  std::map<Sig, std::tuple<int, uint32_t, uint32_t>> best;
  best[a_of(s0)] = std::make_tuple(0, 0u, 0u);
  std::vector<Sample> cur{s0};
  std::vector<uint32_t> cost{0};
  long kept = 0, all = 0;
  for (int n = 0; n <= max_n; n++) {
    std::map<Sig, std::tuple<int, uint32_t, uint32_t>> here;
    std::vector<Sample> next;
    std::vector<uint32_t> nc;
    for (size_t w = 0; w < cur.size(); w++)
      for (int i = 0; i < P::N; i++) {
        Sample s = cur[w];
        for (S4& x : s.w) apply_at<P>(i, x);
        const uint32_t c = cost[w] + cost_of<P>(i);
        const auto key = std::make_tuple(n + 1, c, uint32_t(w * P::N + size_t(i)));
        const Sig g = a_of(s);
        auto it = here.emplace(g, key).first;
        if (key < it->second) it->second = key;
        if (n < max_n) next.push_back(s);
        nc.push_back(c);
      }
    for (const auto& h : here) {
      auto it = best.emplace(h.first, h.second).first;
      if (h.second < it->second) it->second = h.second;
    }
    for (int shorter = 0; shorter < 2; shorter++) {
      const WordTable t = word_table<P>(n, shorter != 0);
      for (const auto& h : here) {
        if (shorter && best[h.first] != h.second) continue;  // a shorter suffix has this effect
        const uint32_t idx = std::get<2>(h.second);
        if (!keeps<P>(t, n, shorter != 0, idx / P::N, int(idx % P::N))) {
          std::printf("%s: %d inner instructions (shorter %d): suffix %u is left out although it is the smallest of its "
                      "effect\n", name, n, shorter, idx);
          return 1;
        }
      }
      if (shorter && n == max_n)
        for (uint8_t l : t.leaf) {
          kept += l != kLeafNone;
          all++;
        }
    }
    cur.swap(next);
    cost.swap(nc);
  }
  std::printf("%s: %ld of %ld inner words kept\n", name, kept, all);
  return kept < all ? 0 : 1;
}

int main() {
  if (check<PGo>("14 ops, cmd/mulopt", 3) || check<PWide>("21 ops, workload", 3) || check<PFast>("14 ops, fast", 3) ||
      check<PCuda>("21 ops, cuda", 3))
    return 1;
  std::printf("OK words\n");
  return 0;
}
