// z80b_kernels.cuh -- kernel declarations and launch parameters.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "z80b_device.cuh"

namespace z80b {

// Surviving (target, candidate) pairs of the QuickCheck scan.
struct QCOut {
  uint32_t* cnt_f;   // [n] full-equivalence survivors per target
  uint32_t* cnt_m;   // [n] masked-only survivors per target
  uint32_t* cnt_all; // [n] cnt_f + cnt_m (scan input)
  const uint32_t* base;  // [n] exclusive prefix of cnt_f + cnt_m (collect pass)
  uint32_t* surv;    // survivor pool indices
  uint16_t* sdiff;   // FlagDiff (low byte) | differing registers << 8
  TargetMeta* meta;  // [n]
  unsigned long long* checks;  // eligible pairs evaluated (count pass)
  // Single-pass QuickCheck (bucket index only; null: count and collect
  // passes): the count pass also keeps the survivors of each target that has
  // at most kQCSlots of them, in enumeration order, as candidate | diff << 16
  // | masked << 31 in tmp[t * kQCSlots ...], and counts the targets with more
  // in *over; k_qc_compact moves the kept ones to their places and the
  // collect pass runs for the others alone.
  uint32_t* tmp;
  uint32_t* over;
  // Bucket index: the targets whose range of entries is long (k_qc_long takes
  // them), and their number.
  uint32_t* longs;
  uint32_t* nlong;
};
constexpr uint32_t kQCSlots = 8;

struct QCConfig {
  uint32_t w2mask;   // 0xFFFFFFFF: compare SP and M; 0x0000FFFF: fingerprint (SP only)
  int all_hits;      // 1: pkg/gpu semantics (one list: masked-QC passes)
  int use_smem;      // pool QC0 staged in shared memory
  uint32_t* bad;     // bucket index: the programs' opcodes are checked here, the least bad target
                     // goes to *bad (null: the host has checked them)
  uint32_t first;    // index of the launch's first target
};

// QuickCheck index of a candidate pool: per dead-register mask in use the
// unpruned candidates by a hash of what QuickCheck compares whatever the dead
// flags are (A, the live registers, SP and, where compared, M, on all eight
// vectors), in pool order within a hash, each with its eight F bytes; a table
// of the first entry of each range of the top hash bits; and the unpruned
// candidates shorter than b bytes (the count of QuickCheck units a target of b
// bytes evaluates).  Two entries with both hashes equal have equal outputs
// (the build checks it), so a target compares its outputs with one of them
// and its F bytes with each.  Ranges of about one entry for the 4,531
// instructions (12 bits) and four for the 266,675 first-op instructions (16
// bits): a target reads its range eight entries at a time.
constexpr uint32_t kQCIndexBits = 26;           // candidate number in a sort key and an entry
// Device memory: 20 bytes per candidate and mask, for the masks in use (as
// much again at most where their room has doubled); 16 bytes per candidate of
// sort scratch for the masks of one sort; 64 top tables (17 MB at 16 bits).
constexpr uint32_t kQCIndexMax = 1u << 20;
constexpr uint32_t kQCAllMasksMax = 65536;      // pools up to here: all 64 masks in one sort
inline uint32_t qc_top_bits(uint32_t n) { return n <= kQCAllMasksMax ? 12u : 16u; }
struct QCIndex {
  const uint4* entries;            // {hash, candidate | bytes << kQCIndexBits, F of vectors 0-3, F of vectors 4-7}
  const uint32_t* hash2;           // per entry a second hash
  const uint32_t* top;             // [64 * ((1 << top_bits) + 1)] positions in entries
  const uint32_t* elig_lt;         // [256]
  uint32_t top_bits;
  uint32_t check_h2;               // entries of one hash can have different second ones
};

// Per-(target, kind) progress of the first-found rounds.
struct Lanes {
  uint32_t* next;    // [2n] survivor index to try next; bit31 = resolved
  uint32_t* win;     // [2n] winning pool index or kNone
  uint16_t* windiff; // [2n] sdiff of the winner
  uint8_t* spec;     // [2n] log2 of the lane's survivor window in the next round
};

// A-independent sweeps: 128 A-blocks per unit in the scalar kernel, 1,024
// (32 per lane, 32 states per lane word) in the bit-sliced one.
constexpr uint32_t kXScalarBlocks = 128, kXBitsBlocks = 1024;

// Survivor windows: a lane whose survivors keep failing ExhaustiveCheck
// takes 1, 2, 4, ... of its next survivors (in enumeration order) into one
// round, up to these caps; the first one that passes wins, as if they had
// been tried one per round.
constexpr uint32_t kMaxSpec1 = 6;  // length-1 pass: windows up to 64
constexpr uint32_t kMaxSpec2 = 5;  // length-2 pass: windows up to 32 (the lane's slots)

// The sweep classes: 0 full state, A-dependent; 1 A-independent; 2 compact;
// 3 wide compact; 4 register state.
constexpr int kClasses = 5;

// Device-side state of a round and of its loop.
struct RoundCtl {
  // Chunk lists of the classes: entries << kChunkBits | chunks, so that one
  // atomic hands a pair both its entry and its first chunk, and the entries
  // of a class ascend by first chunk.
  unsigned long long alloc[kClasses];
  unsigned long long counter[kClasses];  // chunk dispensers
  unsigned long long pairs;              // pairs swept, all rounds
  uint32_t npairs;                       // slots handed out in this round (may exceed the capacity)
  uint32_t active;                       // set when a lane has something left after this round
  uint32_t nscan;                        // length-2 pass: lanes that wait for a rescan
  uint32_t more;                         // the last round's active
  uint32_t np;                           // the last round's pairs
  uint32_t rounds;                       // rounds with pairs
  uint32_t iters;                        // loop iterations
  uint32_t overrun;                      // set when the loop stopped at kMaxRoundIters (an error)
};
constexpr int kChunkBits = 39;
constexpr unsigned long long kChunkMask = (1ull << kChunkBits) - 1;
// Most pair slots of a round (an entry number takes the bits above
// kChunkBits) and most chunks of a pair, so that the chunks of a full round
// stay below 2^kChunkBits.  A power of two, as the units of every sweep are:
// any other limit leaves a long sweep's last chunks empty, and the kernels
// count a chunk from its first unit on.
constexpr unsigned long long kMaxRoundPairs = (1ull << (64 - kChunkBits)) - 1;
inline uint32_t max_chunks(unsigned long long pairs) {
  uint32_t c = 1u << 20;
  while (c > 1 && c * pairs > kChunkMask) c >>= 1;
  return c;
}

struct RoundBuf {
  PairRec* pairs;
  uint32_t* pair_src;              // index of the (target, kind) lane or survivor
  // Per class, the pairs that have chunks in it: first chunk and pair index
  // of each entry (cpair null: entry i is pair i).
  unsigned long long* cbase[kClasses];
  uint32_t* cpair[kClasses];
  uint32_t compact;                // pairs whose registers fit the compact state get that class
  uint32_t wide;                   // the wide compact and the register-state classes are in use
  uint32_t* rejected;              // per pair: 1 a mismatch was found, 2 cancelled
  uint8_t* wlen;                   // per pair: survivors in the window it heads (0: not a head)
  // First-found windows (null for independent pairs): per pair the end
  // (exclusive) of its survivor window, and the chunks of its sweep that
  // finished without a mismatch.  A pair whose every chunk finished so
  // passed; the pairs after it in its window can no longer win, and their
  // sweeps are cancelled (rejected = 2).
  uint32_t* wend;
  uint32_t* cdone;
  uint32_t cap;                    // pair slots of the buffers
  uint32_t max_chunks;             // chunks of one pair at most
  unsigned long long* states;      // [2]: states of the reference's sweeps covered, states evaluated
  uint32_t chunk_blocks;           // sweep units per work chunk
  uint32_t xunit;                  // A-blocks per unit of an A-independent sweep: kXBitsBlocks
                                   // (bit-sliced kernel), else (0 too) the scalar kernel's 128
  RoundCtl* ctl;
};

// Length-2 candidate pass (pair pool): indexes and per-lane slots.
constexpr uint32_t kSlots2 = 32;  // survivors held per (target, kind) lane
// Index of the unpruned pairs for one dead-register mask.  The pairs are
// sorted by (encoded size, hash of A, SP, M and the live registers after all
// eight QuickCheck vectors, hash of the eight F bytes) and cut into groups
// of pairs that agree on all of these outputs themselves, not only on the
// hashes: one comparison with a group's first pair answers the QuickCheck
// for every member under any dead-flag mask.
struct PairIndex {
  const uint32_t* members;  // pair indices, ascending within a group
  const uint4* groups;      // {pair_group_key, first member's position, F bytes 0-3, F bytes 4-7},
                            // sorted by key; one more entry ends the last group
  const uint32_t* top;      // [kPairTop + 1] first group of each range of the key's top bits
};
constexpr uint32_t kPairTopBits = 18, kPairTop = 1u << kPairTopBits;
// Group key: the size class (pairs take 2, 3 or 4 bytes) and 30 hash bits.
constexpr uint32_t kPairSizes = 3;
struct PairScan {
  const PairIndex* idx;                  // [64] per dead-register mask (those in use)
  const uint4* out;                      // [pairs * 8] outputs on the vectors, 128 bytes per pair
  uint32_t* cnt;                         // [2n] survivors in the lane's slots
  uint32_t* resume;                      // [2n] pair index to go on from; kNone: exhausted
  uint32_t* surv;                        // [2n * kSlots2] pair-pool indices
  uint16_t* sdiff;                       // [2n * kSlots2]
  uint32_t* scan;                        // [2n] the lanes waiting for a rescan (ctl->nscan of them)
  const unsigned long long* eligible;    // [16] unpruned pairs shorter than b bytes
  unsigned long long* checks;            // QuickCheck units (eligible pairs per target)
};

struct DevRule {
  uint32_t target;
  uint32_t cand;
  uint16_t diff;   // flag diff | reg diff << 8
  uint8_t kind;    // 0 full, 1 masked, 2 all-hits
  uint8_t clen;    // candidate length: 1 (pool index) or 2 (pair-pool index)
  int16_t bytes_saved, cycles_saved;
};

// Moves the survivors the count pass kept (targets with 1..kQCSlots) to
// their places after base[t]: the full ones first, then the masked ones,
// each in enumeration order.
void launch_qc_compact(const QCOut& q, uint32_t n, cudaStream_t s);
void dev_upload_tables(cudaStream_t s);
int dev_num_sms();

// by_pair: the eight QuickCheck outputs of a candidate side by side (qc[c * 8
// + v]) instead of vector-major (qc[v * n + c]).
void launch_pool_outputs(const uint32_t* insn, uint32_t n, uint32_t len, uint4* qc, uint4* mid, bool by_pair,
                         cudaStream_t s);
void launch_exec(const uint32_t* in_states, const uint32_t* seqs, const uint8_t* lens, uint32_t len,
                 uint32_t stride, uint32_t n, uint32_t* out_states, cudaStream_t s);
void launch_fingerprints(const uint32_t* seqs, uint32_t n, uint32_t len, uint8_t* out, cudaStream_t s);
void launch_qc_scan(const DevTargets& T, const DevPool& P, const QCConfig& cfg, const QCOut& o,
                    bool collect, cudaStream_t s);
// One fingerprint query: packed words by vector; the counters a query leaves
// cleared; what the host reads (page-locked memory).
struct FpQuery {
  uint32_t w[24];
};
struct FpCounters {
  uint32_t hits, done;
};
constexpr uint32_t kFpHere = 2046;
struct FpAnswer {
  uint32_t count, pad;
  uint32_t hits[kFpHere];  // the first of them, in no order
};
// Indices of the candidates with the fingerprint, flags in `dead` aside: all
// of them in hits (P.n slots), their number and the first kFpHere in answer.
void launch_fp_query(const DevPool& P, const FpQuery& fp, uint32_t dead, uint32_t* hits, FpCounters* ctr,
                     FpAnswer* answer, cudaStream_t s);
// Sort keys of masks [m0, m0 + nm): keys[i * P.n + c] for mask m0 + i.
void launch_qc_keys(const DevPool& P, uint32_t w2mask, uint32_t m0, uint32_t nm, unsigned long long* keys,
                    cudaStream_t s);
// From the nm * nv sorted keys at keys[0]: the entries at positions first on,
// and their masks' top tables; flags[0] is set when two entries of equal
// hashes differ in their outputs, flags[1] when two of equal first hashes
// differ in the second.
void launch_qc_entries(const DevPool& P, uint32_t w2mask, const unsigned long long* keys, uint32_t nv, uint32_t first,
                       uint32_t m0, uint32_t nm, uint32_t top_bits, uint4* entries, uint32_t* hash2, uint32_t* top,
                       uint32_t* flags, cudaStream_t s);
void launch_qc_bucket(const DevTargets& T, const DevPool& P, const QCConfig& cfg, const QCIndex& ix,
                      const QCOut& o, bool collect, cudaStream_t s);
// Counters of one pipeline run on the device, cleared before it.
constexpr int kMaxCountParts = 5;  // chunks of targets in a count pass, and the collect pass
struct Tally {
  unsigned long long checks, checked;    // QuickCheck units; the reference's 'checked' counter
  unsigned long long states[2];          // RoundBuf::states
  uint32_t over;                         // QCOut::over
  uint32_t nlong[kMaxCountParts];        // QCOut::nlong
  uint32_t bad, pad;                     // QCConfig::bad, complemented: 0 none
};
// What the host reads of a run, written to page-locked host memory by one
// small kernel where several copies would each cost a few microseconds.
struct Report {
  Tally tally;
  unsigned long long nsurv, nrules;      // totals of the survivor and the rule prefix sums
  RoundCtl pass[2];                      // the two passes' rounds
};
// survivors: base / cnt_f / cnt_m of q over n targets; rules: rbase / rcnt
// over nr items (nr 0: none yet); ctl: RoundCtl[2] or null.
void launch_report(const Tally* t, const QCOut& q, uint32_t n, const uint32_t* rbase, const uint32_t* rcnt, uint32_t nr,
                   const RoundCtl* ctl, Report* out, cudaStream_t s);
// The lanes of n targets before their first round.
void launch_lanes_init(const Lanes& L, uint32_t n, cudaStream_t s);
// Exclusive sum of n <= kScanSmall items in one block.
constexpr uint32_t kScanSmall = 8192;
void launch_scan_small(const uint32_t* in, uint32_t* out, uint32_t n, cudaStream_t s);

// Everything the kernels of a round need, in device memory: a captured round
// graph reads the job at hand from here, so a job of another size replays the
// same graph (the sweeps' own share: SweepArgs).
struct RoundArgs {
  DevTargets T;
  DevPool P;
  QCOut q;              // survivors and metadata of the length-1 QuickCheck
  Lanes L;              // the lanes of this pass
  RoundBuf R;
  PairScan ps;          // length-2 pass only
  const uint16_t* sdiff;  // per survivor: FlagDiff | differing registers << 8
  uint32_t max_spec;    // windows of up to 2^max_spec survivors
};
// Writes a to *dst and clears a.R.ctl.
void launch_round_args(const RoundArgs& a, RoundArgs* dst, cudaStream_t s);

// One round, in stream order: [rescan,] build, plan, sweeps, resolve, end.
// `small`: launch shapes for jobs of few targets (any job may use either).
void launch_round_build(const RoundArgs* a, bool pair, bool small, cudaStream_t s);
void launch_pair_plan(const RoundArgs* a, bool small, cudaStream_t s);
void launch_round_resolve(const RoundArgs* a, bool pair, bool small, cudaStream_t s);
// The counters for the next round, and the loop's condition (in_loop).
void launch_round_end(const RoundArgs* a, bool in_loop, cudaGraphConditionalHandle loop, cudaStream_t s);
// Bound on the iterations of one device-driven loop: a loop that has not
// ended by then stops and reports an error instead of running on.
constexpr uint32_t kMaxRoundIters = 1u << 20;

// What the sweep kernels read, by value: their registers are all taken by the
// states, and a field in the kernel's parameters costs none (the same fields
// behind a pointer made every class spill, 100 to 400 bytes a thread).  None
// of it depends on the number of targets, so a captured graph holds for jobs
// of any size until a buffer grows or the form of the targets changes.
struct SweepArgs {
  const uint32_t *tinsn, *pinsn;
  const uint8_t *tlens, *plens;   // null: tlen / plen
  uint32_t tlen, tstride, plen, pstride;
  const PairRec* pairs;
  uint32_t* rejected;
  const uint32_t* wend;           // null: independent pairs
  uint32_t* cdone;
  const unsigned long long* cbase[kClasses];
  const uint32_t* cpair[kClasses];
  unsigned long long* states;
  RoundCtl* ctl;
  uint32_t xunit, pad;
};
SweepArgs sweep_args(const RoundArgs& a);

// k = states per lane per dispatch: 1, 2, 4 or 8.
// Launches the sweep kernel of each class that has chunks (alloc: the round's
// RoundCtl::alloc on the host); returns the number of launches and ORs the
// launched instantiations into *kernels (may be NULL): kSweep* bits.
constexpr uint32_t kSweepBits = 1u, kSweepXBits = 2u, kSweepCompact = 4u;
constexpr uint32_t kSweepScalarK1 = 8u;  // scalar A-independent kernel, K = 1, 2, 4, 8: bits 3..6
constexpr uint32_t kSweepWide = 128u, kSweepRegs = 256u;
int launch_exhaustive(const SweepArgs& a, const unsigned long long* alloc, int k, cudaStream_t s,
                      uint32_t* kernels = nullptr);
// The sweep kernels of the configured classes on persistent grids, the chunk
// totals read on the device.  ss[0..4]: the streams of the register-state,
// wide, compact, bit-sliced and A-independent classes (the classes share no
// chunk, pair or dispenser, so their launches may run side by side: one
// class's blocks take the SMs that another's finished blocks leave).
int launch_exhaustive_dev(const SweepArgs& a, bool compact, bool wide, int k, const cudaStream_t* ss);
// Sets up (outside any stream capture) the launch facts of the kernels
// launch_exhaustive_dev will launch.
void warm_exhaustive_dev(bool compact, bool wide, uint32_t xunit, int k);
// Pairs (i, i) of n independent pairs.
void launch_pairs_identity(uint32_t n, const RoundBuf& R, cudaStream_t s);
// One pair per MidCheck survivor among survivors [lo, hi).
void launch_pairs_from_survivors(const QCOut& q, const uint8_t* midpass, uint32_t lo, uint32_t hi,
                                 const uint32_t* surv_target, const RoundBuf& R, cudaStream_t s);
void launch_midcheck(const DevTargets& T, const DevPool& P, const uint32_t* surv,
                     const uint32_t* surv_target, uint32_t nsurv, uint8_t* pass, cudaStream_t s);
void launch_surv_targets(const QCOut& q, uint32_t n, uint32_t* surv_target, cudaStream_t s);
// L2: the lanes of the length-2 candidate pass (all pointers null when the
// job stops at length 1); pool2_enum: the enumerated length-2 sequences.
void launch_rule_count_first(const Lanes& L, const Lanes& L2, uint32_t n, uint32_t* cnt, const DevTargets& T,
                             unsigned long long* checked, uint32_t pool_enum, unsigned long long pool2_enum,
                             cudaStream_t s);
// P / P2: the pools of the two passes; meta: the targets' bytes and T-states.
void launch_rule_write_first(const Lanes& L, const Lanes& L2, uint32_t n, const uint32_t* base, const TargetMeta* meta,
                             const DevPool& P, const DevPool& P2, DevRule* out, cudaStream_t s);
void launch_rule_write_all(const uint32_t* flag, const uint32_t* base, uint32_t nsurv, const uint32_t* surv,
                           const uint16_t* sdiff, const uint32_t* surv_target, const TargetMeta* meta, const DevPool& P,
                           DevRule* out, cudaStream_t s);
void launch_rule_count_all(const RoundBuf& R, uint32_t npairs, uint32_t* flag, cudaStream_t s);
// The steps of a pair index (PairIndex) over the n unpruned pairs `valid`:
// their sort keys for a dead-register mask; after the sort, which positions
// begin a group (flag 1); after the flags' inclusive sum, the group records;
// and the top table.
void launch_pair_keys(const DevPool& P, const uint4* out, const uint32_t* valid, uint32_t n, uint32_t dregs,
                      unsigned long long* keys, cudaStream_t s);
void launch_pair_heads(const uint4* out, const unsigned long long* keys, const uint32_t* members, uint32_t n,
                       uint32_t dregs, uint32_t* head, cudaStream_t s);
void launch_pair_groups(const uint4* out, const unsigned long long* keys, const uint32_t* members, uint32_t n,
                        const uint32_t* gid, uint4* groups, cudaStream_t s);
void launch_pair_top(const uint4* groups, uint32_t n_groups, uint32_t* top, cudaStream_t s);
void launch_pair_lanes_init(const DevTargets& T, const Lanes& L1, const QCOut& q1, const Lanes& L2,
                            const PairScan& ps, cudaStream_t s);
// Fills the slots of the lanes that have none left: every lane of a job
// (all), or those in PairScan::scan.
void launch_pair_scan(const RoundArgs* a, uint32_t n, bool all, bool small, cudaStream_t s);
void launch_verify_small(const uint32_t* tgt, const uint8_t* tlens, const uint32_t* cand,
                         const uint8_t* clens, uint32_t stride, uint32_t n, const uint8_t* dead,
                         uint32_t tiers, uint8_t* out, uint8_t* flagdiff, cudaStream_t s);

}  // namespace z80b
