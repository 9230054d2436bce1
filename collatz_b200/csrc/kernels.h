// kernels.h -- argument blocks and launchers of the hot-path kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rec.h"
#include "tables.h"

namespace cz {

// ---------------- cases mode (cases.cu) ----------------
struct CasesArgs {
  const uint32_t* pairs;   // npairs x 8 words: base limbs 0..3, number limbs 0..3 (cu:521-528)
  uint32_t npairs;
  int bigindex;            // >= 0: bucket of every pair; < 0: per pair in base limb 3
  const uint32_t* bv;      // CaseTables
  const uint32_t* mod9;
  const uint32_t* magic;
  const uint32_t* pow3;
  uint32_t mbi, tpo;
  uint32_t* pair_counter;  // scratch, zero before launch
  ReqRec* rec;
  uint32_t* overflow;      // overflow seeds, 4 words each
  uint32_t overflow_cap;
  unsigned long long* overflow_count;
  uint32_t iter_cap;       // checkpoints per seed before ERR_ITER_CAP
  uint32_t multi;          // line batch: base limb 3 = bigindex | line << 8, rec[line] per line
  uint32_t four = 4, p5 = 1u << 5, p29 = 1u << 29;  // unknown to the compiler (cases_win.cu: additions and
                                                    // shifts on the multiply-add pipe)
  uint32_t unit = 0;       // of the table-driven kernel's limits (case_limits.h), set by its launcher
};
int cases_variants();
cudaError_t launch_cases(const CasesArgs& a, int variant, uint32_t sm_count, cudaStream_t st);
// For every context, before its first launch; the tables are filled by a device's first.  Ends with st idle.
cudaError_t cases_win_init(cudaStream_t st);
cudaError_t launch_cases_win(const CasesArgs& a, uint32_t sm_count, cudaStream_t st);  // N <= 52

// ---------------- device Step 1 (step1_dev.cu) ----------------
// A node of search1's tree (cu:497-505): base and number as little-endian
// 64-bit halves; sigfig | line << 8 (line: the node's cases line in a line
// batch), threepower, doubleeven, numevens.
struct S1Node {
  unsigned long long base_lo, base_hi, num_lo, num_hi;
  uint32_t sig, tp, de, ne;
};
static_assert(sizeof(S1Node) == 48, "S1Node layout");

// Counters of one device Step 1 run (zeroed before it starts).
struct S1Scalars {
  uint32_t level[128];  // frontier size after each breadth-first level
  uint32_t cursor[32];  // [0] count pass, [1 + chunk % 31] emit passes
  unsigned long long total;
  unsigned long long hist[17];  // leaves per bigindex; [16] = bigindex >= 16
};

struct Step1Args {
  uint32_t mbi, tpo;
  const S1Node* in;          // frontier
  const uint32_t* in_count;  // its size (device)
  S1Node* out;               // expand: children
  uint32_t* out_count;
  unsigned long long* off;   // walk: per frontier node, first leaf index
  unsigned long long* cnt;   // walk: per frontier node, leaves
  unsigned long long* total;
  unsigned long long* hist;
  unsigned long long* hist_lines;  // line batches: leaves per (line, bigindex), 17 per line; else null
  uint32_t* cursor;          // walk: zero before the launch
  ulonglong2* stk_num;       // walk: pending siblings, [level][thread]
  uint4* stk_meta;
  uint32_t nthreads;         // walk: threads of the launch (grid x 128)
  uint32_t* pairs;           // emit: pairs with leaf index in [w_lo, w_hi)
  unsigned long long w_lo, w_hi;
};
constexpr uint32_t STEP1_WALK_BLOCKS_PER_SM = 8;
cudaError_t launch_step1_expand(const Step1Args& a, uint32_t bound, cudaStream_t st);
cudaError_t launch_step1_walk(const Step1Args& a, bool emit, cudaStream_t st);

// ---------------- range mode (range.cu) ----------------
constexpr uint32_t RANGE_ITEM = 64;     // survivor-table entries per work item (a row)
constexpr uint32_t DENSE_ITEM = 64;     // consecutive integers per dense work item

// A segment of work items of one request.  kind 0: survivor entries
// [s_lo, s_hi) of one mod-9 class of the class-major table, for
// nq blocks from q on (seeds n = q 2^k + r): consecutive ones, or (qstride 9)
// those that keep the class under the mod-9 sieve; item i is entries s_lo +
// 64 (i / nq) onwards of the (i mod nq)-th block;
// kind 1: integers [d_lo, d_hi) iterated without the residue sieve.
struct RangeSeg {
  unsigned long long item_begin;  // global index of the first item
  unsigned long long q_lo;        // kind 0: first block, low 64 bits; kind 1: d_lo
  unsigned long long d_hi;        // kind 1: end (exclusive)
  uint32_t q_hi;                  // kind 0: first block, bits 64..95
  uint32_t nq;                    // kind 0: number of blocks
  uint32_t s_lo, s_hi;            // kind 0: survivor index range
  uint32_t req, pad;              // request index (ReqRec)
  uint16_t kind;
  uint16_t qstride;               // kind 0: 0 or 1: consecutive blocks; 9: the blocks that keep the class
  uint32_t mod9;                  // kind 0: the class (r mod 9); kind 1: 1 to apply the mod-9 sieve
  // Item index within the original segment of item_begin (non-zero when a
  // scheduler cuts a segment into slices; local indices stay < 2^32 for kind 0).
  uint32_t local0_lo, local0_hi;
};
static_assert(sizeof(RangeSeg) == 64, "RangeSeg");

struct WidenEntry {  // a seed to re-run with wider limbs
  uint32_t req, n0, n1, n2;
};

// A seed that may be its request's maximum stopping time (kind 0) or excursion (kind 1).
struct RangeCand {
  uint32_t req, kind, st, pad;
  uint32_t E[4];
  uint32_t seed[4];
};
static_assert(sizeof(RangeCand) == 48, "RangeCand");

// Counters of a launch, zero before it.
struct RangeHead {
  unsigned long long item_cursor;  // next item to claim
  uint32_t widened, cands;         // entries of the widen list and of the candidate list
  uint32_t pad[12];
};
static_assert(sizeof(RangeHead) == 64, "RangeHead");

// Lists of a launch; their lengths are in the head.
constexpr uint32_t WIDEN_CAP = 1u << 16;
constexpr uint32_t CAND_CAP = 1u << 16;  // candidates beyond it take the record's lock in the kernel
struct RangeLists {
  RangeCand cand[CAND_CAP];
  WidenEntry widen[WIDEN_CAP];
};

// What the diagnostics form of the range kernel counts.
enum RangeStat : int {
  RS_RUNS,            // runs of rows opened
  RS_ENTRIES,         // table entries (or integers) handed to lanes
  RS_WINDOWS,         // windows of the window loop, by lanes with a seed
  RS_PASSES,          // groups of four windows of a warp
  RS_SCREENED,        // seeds that reached a limit and were screened
  RS_SCREEN_WINDOWS,  // their windows in the screen
  RS_EXACT,           // seeds on the exact path
  RS_RUN_PAIRS,       // their run pairs
  RS_OFFERS,          // offers of a maximum
  RS_SCOUTS,          // head starts of a request's maxima
  RS_CYCLES_WINDOWS,  // clock cycles of all warps in the window loop,
  RS_CYCLES_ENTRIES,  // handing out entries,
  RS_CYCLES_RUNS,     // opening runs (and waiting for the block at the end),
  RS_CYCLES_SCREEN,   // in the screen,
  RS_CYCLES_EXACT,    // on the exact path,
  RS_CYCLES,          // and in all of these
  RANGE_STATS
};

struct RangeArgs {
  const RangeEntry* table;        // survivor table of the 2^k sieve
  uint32_t k;
  const RangeSeg* segs;
  uint32_t nsegs;
  unsigned long long item_limit;    // items >= limit are not claimed in this launch
  RangeHead* head;
  RangeLists* lists;
  ReqRec* recs;
  uint32_t iter_cap;              // odd/even run pairs per seed before ERR_ITER_CAP
  uint32_t negative;              // 1: the negative-integer variant (a table built for it)
  unsigned long long* stats;      // diagnostics counts (RangeStat); null: the kernel without them
  uint32_t seed_bits;             // bit length of the launch's largest seed (0: not known)
  uint32_t one = 1, mone = ~0u, eight = 8;  // 1, -1 and 8, unknown to the compiler (range.cu: window)
  uint32_t rl = 0, rs = 0;        // the variant's thresholds (range_variants.h), set by launch_range
};
// Largest N that runs the kernel with run pairs from a table (cases_win.cu), whose values go to the
// exact path from 2^71 on: at N = 48 a line of 304 724 seeds took 0.156 ms with it and 0.392
// with four limbs, at N = 52 one of 3.75 M seeds 0.274 and 0.578.  There is no smallest N: the
// whole tree took 0.17 and 0.22 ms at N = 20, 0.16 and 0.36 at 26, 2.2 and 5.1 at 36, 21 and 59 at 40.
constexpr uint32_t CASES_WIN_MAX_BITS = 52;
int range_variants();
int range64_variants();
// Hash of the variant table (part of the autotuner's cache key).
uint32_t range_variant_rev();
// Launches whose seeds have at most this many bits may run on two-word values.
uint32_t range64_max_seed_bits();
cudaError_t range_init(cudaStream_t st);  // as cases_win_init
// The range kernel with values of 2, 3 or 4 words (a seed that outgrows them
// takes the kernel's exact path, so any width gives the same results).
cudaError_t launch_range(const RangeArgs& a, int words, int variant, uint32_t sm_count, cudaStream_t st);
// After the range kernel: the candidates into the records, and the widened seeds re-run
// from scratch with 6 and then 8 limbs.  The list lengths are read on the device, so the
// launch can sit in a captured graph.
cudaError_t launch_range_finish(const RangeArgs& a, cudaStream_t st);

// ---------------- trajectory queries (traj.cu) ----------------
// All limb classes in one launch (traj.cu): index = the seed ids sorted by
// limb class (4, 6, 8, 12, 16 limbs; class j at [cstart[j], cstart[j + 1])),
// one cursor (zero before the launch); a seed that needs more limbs is run
// again by the same thread with the next width.
struct TrajAllArgs {
  const uint32_t* seeds;       // nseeds x 8 limbs
  const uint32_t* index;       // cstart[5] entries
  uint32_t cstart[6];
  unsigned long long* st;      // out: stopping time
  uint32_t* exc;               // out: 16 limbs each
  uint32_t* status;            // out: 0 ok, 1 trivial, 2 overflow, 3 iteration cap
  uint32_t* cursor;            // scratch
  uint32_t iter_cap;
};
cudaError_t launch_traj_all(const TrajAllArgs& a, uint32_t grid, cudaStream_t st);
// Limb class of a seed of at most 256 bits (8 little-endian limbs): 0..4 for
// 4, 6, 8, 12, 16 limbs, leaving room for the value to grow before it is
// handed on.
inline uint32_t traj_class(const uint32_t* w) {
  uint32_t bl = 0;
  for (int j = 7; j >= 0; j--)
    if (w[j]) {
      bl = 32u * j + (32u - __builtin_clz(w[j]));
      break;
    }
  return bl <= 96 ? 0 : bl <= 160 ? 1 : bl <= 224 ? 2 : bl <= 352 ? 3 : 4;
}

}  // namespace cz
