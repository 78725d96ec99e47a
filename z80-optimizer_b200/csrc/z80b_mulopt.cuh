// z80b_mulopt.cuh -- constant-multiply search (cmd/mulopt) on the device.
//
// One enumeration per sequence length serves every constant K at once: a
// sequence that maps x = 1 to k is a candidate for K = k only, so instead
// of one odometer per K (cmd/mulopt/main.go:186-229) the device walks the
// N^L sequences of length L once and files each sequence that passes the
// all-256-inputs test under its own K.  Per K and length the winner is the
// minimum of (T-states, odometer index), which is the reference's rule
// (shortest length, then `c < bestCost` in odometer order).
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace z80b {
namespace mul {

// Instruction pools (numbers shared with the C ABI).
enum PoolId : int { kPoolGo = 0, kPoolWide = 1, kPoolFast = 2, kPoolCuda = 3, kNumPools = 4 };

struct PoolInfo {
  int n;                 // instructions in the pool
  int max_len;           // longest length whose odometer index fits the 48-bit key
  const char* const* names;
  const uint8_t* tstates;
};
const PoolInfo& pool_info(int pool);

struct SearchArgs {
  int pool;
  uint8_t b, c, f;       // initial B, C, F (A', F' and the shadows start at 0)
  int min_len, max_len;
  uint32_t want[8];      // bit k: constant k is searched (k = 2..255)
};

struct LenStats {
  unsigned long long filter_nodes;  // warp-level nodes whose leaves passed the x=2/x=255 filter
  unsigned long long full_checks;   // all-256 tests run
  unsigned long long full_pass;     // tests passed
};

// Key of a sequence: level << 60 | tstates << 48 | odometer index (the level,
// its length, in the keys of prefixes only).
constexpr int kKeyShift = 48, kLevelShift = 60;
constexpr unsigned long long kIndexMask = (1ull << kKeyShift) - 1;
constexpr unsigned long long kNoKey = ~0ull;
constexpr int kMaxLen = 16;

// The inner words of a suffix of n + 1 instructions (z80b_mul_words.h) on the
// device: the masks of levels 0..n-1 one behind the other, and the classes.
struct WordBufs {
  const uint32_t* mask;
  const uint8_t* leaf;
  uint32_t first_ops;      // instructions in the level-0 mask (n = 0: 0)
};
constexpr int kMaxInner = 3;
// Their host image: mask words, then the classes.
struct WordImage {
  std::vector<uint32_t> mask;
  std::vector<uint8_t> leaf;
  uint32_t first_ops;
};
WordImage word_image(int pool, int n, bool shorter);
// Instructions of the suffix that a walk of length len appends to every
// prefix (without states).
int plain_suffix(int pool, int len);

// Launches the search of one length L on `stream`.  best[l * 256 + k] (rows
// 0..kMaxLen-1, pre-set to kNoKey) receives in row L the minimum key per
// constant; constants that a shorter length's row answers are no longer
// searched, and a launch with nothing left to search returns at once.  The
// sequences are every prefix of L - d instructions, or the n_reps prefixes in
// `reps` (keys), each followed by the suffixes of d instructions in `words`
// (of d - 1 inner instructions, d at most kMaxInner + 1).  `st`
// (device) accumulates the counters.  Returns the CUDA error of the launch.
cudaError_t launch_length(const SearchArgs& a, int len, const unsigned long long* reps, uint32_t n_reps, int rep_len,
                          const WordBufs& words, unsigned long long* best, LenStats* st, int sms, cudaStream_t stream);

// The same for the n lengths from `first` on in one launch (short ones: every
// prefix, suffixes of one instruction).
cudaError_t launch_short(const SearchArgs& a, int first, int n, unsigned long long* best, LenStats* st, int sms,
                         cudaStream_t stream);

// ---- prefixes with distinct states
// Two prefixes of one length that leave the same state (A, B, C, carry and the
// shadows, for all 256 inputs) can be followed by the same suffixes, and the
// one with the smaller key always gives the smaller key of the whole; and a
// prefix whose state a shorter one already reaches starts no shortest
// sequence (when every shorter length is searched too).  So the walk only
// needs, per length, one prefix per new state: the smallest key.  The states
// of the next level are the children of these (state, instruction).
struct StateTable {
  unsigned long long* hash;   // 0: free
  unsigned long long* key;    // smallest key of the state
  unsigned long long mask;    // slots - 1 (a power of two, at least twice the entries)
};
// The empty prefix: its hash and key.
cudaError_t launch_root(const SearchArgs& a, unsigned long long* hash, unsigned long long* key, cudaStream_t stream);
// Enters n known prefixes.
cudaError_t launch_enter(const StateTable& t, const unsigned long long* hash, const unsigned long long* key, uint32_t n,
                         cudaStream_t stream);
// Hashes the children of n prefixes of `level` instructions (child i of prefix
// j: child_hash[j * pool size + i]) and enters them.
cudaError_t launch_children(const SearchArgs& a, const StateTable& t, const unsigned long long* key, uint32_t n,
                            int level, unsigned long long* child_hash, int sms, cudaStream_t stream);
// Appends to out_hash / out_key the children that hold their slot (count[0]
// of them); every other child is compared with its slot's holder on all 256
// inputs, and count[1] is set if one differs (two states of one hash).
cudaError_t launch_select(const SearchArgs& a, const StateTable& t, const unsigned long long* key, uint32_t n, int level,
                          const unsigned long long* child_hash, unsigned long long* out_hash,
                          unsigned long long* out_key, uint32_t* count, int sms, cudaStream_t stream);

}  // namespace mul
}  // namespace z80b
