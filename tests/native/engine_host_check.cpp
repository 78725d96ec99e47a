// Host checks of the engine's order of work, its behaviour when a call fails
// and what it keeps, on a CUDA runtime without a device (fake_cudart.h).
// Usage: engine_host_check <check>; prints "OK <check>".
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/z80b200.h"
#include "../../z80-optimizer_b200/csrc/z80_plan.cuh"
#include "../../z80-optimizer_b200/csrc/z80_tables.h"
#include "../../z80-optimizer_b200/csrc/z80b_kernels.cuh"
#include "fake_cudart.h"

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("FAILED %s:%d: %s\n", __FILE__, __LINE__, #x); \
      return 1;                                               \
    }                                                         \
  } while (0)

static int verify(z80b_ctx* ctx, uint32_t tiers, std::vector<uint8_t>* out = nullptr) {
  const uint32_t tgt[2] = {0, 1}, cand[2] = {0, 0};
  const uint8_t len[2] = {1, 1};
  std::vector<uint8_t> o(2);
  const int r = z80b_verify_pairs(ctx, tgt, len, cand, len, 1, 2, nullptr, tiers, o.data(), nullptr);
  if (out) *out = o;
  return r;
}
// An allocation that fails is reported by the call that made it, once.
static int error_reported_once(z80b_ctx* ctx) {
  fake::fail_malloc = 1;
  CHECK(verify(ctx, 7) == Z80B_ENOMEM);
  CHECK(verify(ctx, 7) == Z80B_OK);
  z80b_destroy(ctx);
  return 0;
}

// Verification keeps no events: their number does not grow with the calls.
static int verify_events(z80b_ctx* ctx) {
  CHECK(verify(ctx, 7) == Z80B_OK);
  const int events = fake::events;
  for (int i = 0; i < 200; i++) CHECK(verify(ctx, 7) == Z80B_OK);
  CHECK(fake::events == events);
  z80b_destroy(ctx);
  CHECK(fake::events == 0);
  return 0;
}

// Few pairs go up in one copy, and come back in one where nothing is swept.
static int verify_copies(z80b_ctx* ctx) {
  CHECK(verify(ctx, 7) == Z80B_OK);
  const int in = fake::copies_in, out = fake::copies_out;
  CHECK(verify(ctx, 7) == Z80B_OK);
  CHECK(fake::copies_in == in + 1 && fake::copies_out == out + 1);
  CHECK(verify(ctx, 3) == Z80B_OK);
  CHECK(fake::copies_in == in + 2 && fake::copies_out == out + 2);
  z80b_destroy(ctx);
  return 0;
}

static int mul(z80b_ctx* ctx, int min_len, int max_len) {
  const int32_t k = 37;
  z80b_mul_result r;
  return z80b_mul_search(ctx, 0, 0, 0, 0, min_len, max_len, &k, 1, &r, nullptr);
}

// The suffix tables of a walk are ordered before it, and a table whose copy
// failed is copied again by the next search.
static int mul_tables(z80b_ctx* ctx) {
  CHECK(mul(ctx, 1, 6) == Z80B_OK);
  CHECK(fake::unordered == 0);
  const int before = fake::copies_in;
  CHECK(mul(ctx, 2, 6) == Z80B_OK);  // other tables
  const int copies = fake::copies_in - before;
  CHECK(copies > 0 && fake::unordered == 0);
  CHECK(mul(ctx, 2, 6) == Z80B_OK);
  CHECK(fake::copies_in == before + copies);  // kept
  for (int nth = 1; nth <= copies; nth++) {
    z80b_ctx* c = nullptr;
    CHECK(z80b_init(0, &c) == Z80B_OK);
    fake::fail_copy_in = nth;
    CHECK(mul(c, 2, 6) != Z80B_OK);
    const int at = fake::copies_in;
    CHECK(mul(c, 2, 6) == Z80B_OK);
    CHECK(fake::copies_in == at + copies);
    z80b_destroy(c);
  }
  z80b_destroy(ctx);
  return 0;
}

// A search whose levels of states do not fit the device walks every prefix.
static int mul_no_room(z80b_ctx* ctx) {
  z80b_destroy(ctx);
  int refused = 0, done = 0;
  for (int nth = 1;; nth++) {
    z80b_ctx* c = nullptr;
    CHECK(z80b_init(0, &c) == Z80B_OK);
    fake::fail_malloc = nth;
    const int r = mul(c, 1, 9);
    const bool hit = fake::fail_malloc == 0;
    fake::fail_malloc = 0;
    CHECK(r == Z80B_OK || (r == Z80B_ENOMEM && hit));
    CHECK(mul(c, 1, 9) == Z80B_OK);
    z80b_destroy(c);
    if (!hit) break;
    (r == Z80B_OK ? done : refused)++;
  }
  // what any walk takes: the answers, the counters and the suffix tables of
  // the depths 1 (length 6), 2 (length 7) and 4 (behind the states)
  CHECK(refused == 5 && done >= 10);
  return 0;
}

// One search with candidates of two instructions.
static int search2(z80b_ctx* ctx) {
  const uint32_t targets[4] = {0, 0, 0, 0};
  z80b_job job{};
  job.targets = targets;
  job.n_targets = 1;
  job.target_len = job.target_stride = 4;
  job.max_cand_len = 2;
  job.global_dead_flags = 0x28;
  job.mode = Z80B_MODE_FIRST;
  job.path = Z80B_PATH_BATCHED;
  z80b_rule rules[8];
  uint64_t n = 0;
  return z80b_search(ctx, &job, rules, 8, &n, nullptr);
}
// One small search; lens: per-target lengths instead of one.
static int search1(z80b_ctx* ctx, uint32_t n, uint32_t len, uint32_t stride, bool lens, bool masks) {
  const std::vector<uint32_t> targets(size_t(n) * stride);
  const std::vector<uint8_t> tl(n, uint8_t(len)), dead(n, 0x28);
  z80b_job job{};
  job.targets = targets.data();
  job.n_targets = n;
  job.target_len = lens ? 0 : len;
  job.target_lens = lens ? tl.data() : nullptr;
  job.target_stride = stride;
  job.dead_flags = masks ? dead.data() : nullptr;
  job.max_cand_len = 1;
  job.mode = Z80B_MODE_FIRST;
  job.path = Z80B_PATH_BATCHED;
  std::vector<z80b_rule> rules(2 * n);
  uint64_t got = 0;
  return z80b_search(ctx, &job, rules.data(), rules.size(), &got, nullptr);
}
// The round loop of small searches is captured once, whatever the form of
// their targets, and anew only when a search of twice the size comes.
static int small_graphs(z80b_ctx* ctx) {
  CHECK(search1(ctx, 8, 1, 1, false, false) == Z80B_OK);
  CHECK(fake::graphs == 1);
  for (uint32_t len = 1; len <= 4; len++)
    for (uint32_t stride : {len, 4u, 7u})
      for (int form = 0; form < 4; form++) CHECK(search1(ctx, 8, len, stride, form & 1, form & 2) == Z80B_OK);
  CHECK(fake::graphs == 1);
  for (uint32_t n = 1; n <= 1024; n += 3) CHECK(search1(ctx, n, 2, 2, false, false) == Z80B_OK);
  CHECK(fake::graphs == 1 + 7);  // room for 16 .. 1,024 targets
  z80b_destroy(ctx);
  return 0;
}
// What goes up with the pair pool is ordered before the work that reads it.
static int pair_pool_order(z80b_ctx* ctx) {
  CHECK(search2(ctx) == Z80B_OK);
  CHECK(fake::unordered == 0);
  return 0;
}

// An allocation that fails anywhere in the first such search leaves nothing
// half-built: the next search, of this context or another, makes all that is
// missing (it ends with the memory of a search that nothing disturbed).
static int pair_pool_retry(z80b_ctx* first) {
  CHECK(search2(first) == Z80B_OK);
  const size_t whole = fake::bytes;
  z80b_destroy(first);  // the pool goes with its last context
  int failed = 0;
  for (int nth = 1;; nth++) {
    z80b_ctx *a = nullptr, *b = nullptr;
    CHECK(z80b_init(0, &a) == Z80B_OK);
    CHECK(search1(a, 1, 4, 4, false, true) == Z80B_OK);  // what any search takes is there
    fake::fail_malloc = nth;
    const int r = search2(a);
    if (fake::fail_malloc) {  // no allocation left to fail
      fake::fail_malloc = 0;
      CHECK(r == Z80B_OK && fake::bytes == whole);
      z80b_destroy(a);
      break;
    }
    failed++;
    CHECK(r == Z80B_ENOMEM);
    if (nth % 2) {
      CHECK(search2(a) == Z80B_OK);
    } else {
      CHECK(z80b_init(0, &b) == Z80B_OK);
      CHECK(search2(b) == Z80B_OK);
      CHECK(search2(a) == Z80B_OK);
      z80b_destroy(b);
    }
    CHECK(fake::bytes == whole);
    z80b_destroy(a);
  }
  CHECK(failed > 15);
  return 0;
}

// No chunk of a sweep is empty (the sweep kernels count what a chunk covers
// from its first unit on), the chunks cover the sweep, and those of a full
// round can be numbered.
static int chunks(z80b_ctx* ctx) {
  std::vector<unsigned long long> caps{1, 2, 3, 4096, 1ull << 19, (1ull << 19) + 1, (1ull << 20) - 1, 1ull << 20,
                                       20000001, z80b::kMaxRoundPairs};
  for (unsigned long long n = 1; n < 40000000; n = n * 3 / 2 + 1) caps.push_back(n);
  for (unsigned long long cap : caps) {
    if (cap > z80b::kMaxRoundPairs) continue;
    const uint32_t most = z80b::max_chunks(cap);
    CHECK(cap * most <= z80b::kChunkMask);
    for (uint32_t blocks : {1u, 2u, 3u, 7u, 8u, 31u, 32u, 33u, 100u, 511u, 512u, 4095u, 4096u})
      for (int k = 0; k <= 40; k++) {  // a sweep's units are a power of two
        const unsigned long long units = 1ull << k;
        const uint32_t n = z80b::chunk_count(units, blocks, most);
        const unsigned long long per = z80b::chunk_units(units, n);
        CHECK(n >= 1 && n <= most);
        CHECK((n - 1ull) * per < units && n * per >= units);
      }
  }
  z80b_destroy(ctx);
  return 0;
}

// All-hits searches over a list of n instructions, dead-register masks 0..masks-1.
static int load(z80b_ctx* ctx, uint32_t n) {
  uint16_t op = 0;
  while (z80b::op_table()[op].imm != 2) op++;
  std::vector<uint32_t> c(n);
  for (uint32_t i = 0; i < n; i++) c[i] = op | i << 16;
  return z80b_load_candidates(ctx, c.data(), n, 1);
}
static int all_hits(z80b_ctx* ctx, uint32_t masks) {
  std::vector<uint32_t> targets(masks, 0u);
  std::vector<uint8_t> dregs(masks);
  for (uint32_t i = 0; i < masks; i++) dregs[i] = uint8_t(i);
  z80b_job job{};
  job.targets = targets.data();
  job.n_targets = masks;
  job.target_len = job.target_stride = 1;
  job.dead_regs = dregs.data();
  job.max_cand_len = 1;
  job.mode = Z80B_MODE_ALL;
  job.path = Z80B_PATH_BATCHED;
  z80b_rule rule;
  uint64_t n = 0;
  return z80b_search(ctx, &job, &rule, 1, &n, nullptr);
}
// The QuickCheck index of a large list takes memory for the masks in use, and
// a search that has no room for it is done without.
static int qc_index_memory(z80b_ctx* ctx) {
  const uint32_t n = 266675;
  const size_t mask = 20ull * n, fixed = 64ull * 65537 * 4 + 24ull * n + (8u << 20);
  CHECK(load(ctx, n) == Z80B_OK);
  const size_t before = fake::bytes;
  fake::limit = before + (3u << 20);  // room for the search, none for the index
  CHECK(all_hits(ctx, 2) == Z80B_OK);
  CHECK(fake::bytes < before + (3u << 20));
  fake::limit = 0;
  CHECK(all_hits(ctx, 1) == Z80B_OK);
  CHECK(fake::bytes > before + mask && fake::bytes < before + fixed + mask);
  const size_t one = fake::bytes;
  fake::limit = one + (3u << 20);
  CHECK(all_hits(ctx, 5) == Z80B_OK);
  CHECK(fake::bytes < one + (3u << 20));
  fake::limit = 0;
  for (uint32_t k = 2; k <= 64; k += k < 8 ? 1 : 14) {
    CHECK(all_hits(ctx, k) == Z80B_OK);
    CHECK(fake::bytes >= before + k * mask && fake::bytes < before + fixed + 2 * k * mask);
    const int launches = fake::launches;
    CHECK(all_hits(ctx, k) == Z80B_OK);
    const int again = fake::launches - launches;
    CHECK(all_hits(ctx, 1) == Z80B_OK && fake::launches - launches == 2 * again);  // nothing built again
  }
  CHECK(fake::bytes < before + fixed + 64 * mask);
  CHECK(fake::peak < before + fixed + 128 * mask);  // while the last growth copies
  z80b_destroy(ctx);
  return 0;
}

// A large list is indexed for many masks at once only when the searches that
// ask for them have scanned it for as long as that takes.
static int qc_index_debt(z80b_ctx* ctx) {
  const uint32_t n = 266675;
  CHECK(load(ctx, n) == Z80B_OK);
  const size_t before = fake::bytes, no_index = before + (3u << 20);
  for (int i = 0; i < 2; i++) {
    CHECK(all_hits(ctx, 64) == Z80B_OK);
    CHECK(fake::bytes < no_index);
  }
  CHECK(all_hits(ctx, 64) == Z80B_OK);
  CHECK(fake::bytes > before + 64 * 20ull * n);
  CHECK(load(ctx, n) == Z80B_OK);  // another list: from the beginning
  int launches = fake::launches;
  CHECK(all_hits(ctx, 64) == Z80B_OK);
  const int scanned = fake::launches - launches;
  CHECK(all_hits(ctx, 64) == Z80B_OK);
  CHECK(fake::launches - launches == 2 * scanned);
  launches = fake::launches;
  CHECK(all_hits(ctx, 64) == Z80B_OK);
  CHECK(fake::launches - launches > scanned + 64);
  z80b_destroy(ctx);
  return 0;
}
// The counters of fingerprint queries are clear before the first one: where
// clearing them failed, the next query clears them.
static int query_counters(z80b_ctx* ctx) {
  CHECK(load(ctx, 8) == Z80B_OK);
  const uint8_t fp[80] = {};
  uint32_t hits[8], n = 0;
  for (int i = 0; i < 2; i++) {
    fake::fail_memset = 1;
    CHECK(z80b_quickcheck(ctx, fp, 0, hits, 8, &n) != Z80B_OK);
    CHECK(fake::fail_memset == 0);
  }
  CHECK(z80b_quickcheck(ctx, fp, 0, hits, 8, &n) == Z80B_OK);
  fake::fail_memset = 1;
  CHECK(z80b_quickcheck(ctx, fp, 0, hits, 8, &n) == Z80B_OK);  // a query leaves them clear
  fake::fail_memset = 0;
  z80b_destroy(ctx);
  return 0;
}

// The sizes of what a search brings back.
static int sizes(z80b_ctx* ctx) {
  std::printf("OK sizes %zu %zu\n", sizeof(z80b::DevRule), sizeof(z80b::Report));
  z80b_destroy(ctx);
  return 0;
}

int main(int argc, char** argv) {
  const std::string name = argc > 1 ? argv[1] : "";
  struct {
    const char* name;
    int (*run)(z80b_ctx*);
  } checks[] = {{"error_reported_once", error_reported_once}, {"mul_tables", mul_tables}, {"mul_no_room", mul_no_room},
                {"pair_pool_order", pair_pool_order},
                {"pair_pool_retry", pair_pool_retry}, {"chunks", chunks},
                {"verify_events", verify_events}, {"verify_copies", verify_copies}, {"qc_index_memory", qc_index_memory},
                {"query_counters", query_counters}, {"qc_index_debt", qc_index_debt},
                {"small_graphs", small_graphs}, {"sizes", sizes}};
  for (const auto& c : checks)
    if (name == c.name) {
      z80b_ctx* ctx = nullptr;
      CHECK(z80b_init(0, &ctx) == Z80B_OK);
      CHECK(fake::unordered == 0);
      if (c.run(ctx)) return 1;
      std::printf("OK %s\n", c.name);
      return 0;
    }
  std::printf("unknown check '%s'\n", name.c_str());
  return 1;
}
