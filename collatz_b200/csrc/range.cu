// range.cu -- range verification: every seed n of [offset, offset + size)
// that survives the 2^k residue sieve and the mod-9 sieve is shown to fall
// below its start; outputs are the seeds checked, the maximum stopping time
// and the maximum excursion (each with the smallest seed on ties) and the
// seeds that did not finish.
//
// Work.  The host lowers requests into segments: one mod-9 class of the
// class-major survivor table (64 entries to a row) over a run of blocks q.
// Persistent warps claim rows of a segment in block-minor order, so that a
// claim is a few table entries over many blocks.  A lane keeps one entry
// (r, f, c): n = q 2^k + r has T^k(n) = q 3^f + c, and going from block to block
// is one addition.
//
// Windows.  A seed is advanced JW steps at a time: for x = a 2^JW + r,
// T^JW(x) = a 3^(f_r) + T^JW(r), one look-up in a 2^JW-entry shared-memory table
// and one multiply-add, whatever happens to the seed inside the window.  What
// happened follows from the coefficient C_i = 3^(F_i) / 2^i of T^i(n) = C_i n +
// rho_i alone (F_i odd steps among the first i), kept as the integer D_i = 485 F_i -
// 306 i:
//   * 306/485 is a convergent of log 2 / log 3 with no fraction of a smaller
//     denominator between them, so D_i > 0 iff C_i > 1 for 0 < i < 485.
//   * While C_t > 1 for all 0 < t < i, each odd step adds at most C_i / 3 to the
//     remainder: 0 <= rho_i <= C_i F_i / 3.
//   * So C_i > 1 keeps T^i(n) above n, and at the first i with C_i < 1, T^i(n) <
//     n as soon as n > F_i / (3 (1/C_i - 1)); for i < 485 that bound is below
//     27 100 (the nearest 2^i / 3^F above 1 is 2^401 / 3^253 = 1.0031).  For the
//     negative variant rho_i is subtracted: C_i < 1 gives T'^i(m) < m at once, and
//     C_i > 1 keeps T'^i(m) above m when m > F_i / (3 (1 - 1/C_i)), below 8 600
//     (3^265 / 2^420 = 1.0105).  Seeds of at least 2^16 satisfy both.
//   * T^i(n) <= C_i (n + F_i / 3), so D_i / 306 + log2(n) bounds log2 T^i(n) from
//     above to within 0.0024.
// A seed whose D is negative after a window has therefore fallen below its
// start within it.  Its stopping time is at most the steps taken and its
// excursion at most what D allowed; both are below the request's running maxima
// (the windows' limits see to that), so it can change no output and is done.
//
// The screen and the exact path.  A seed that might change an output -- D or the step count
// reaches its limit, or a value could leave the words it is kept in -- is queued, and 32 such
// seeds at a time take their windows again from the start, with four words and a peak per
// window (screen).  What may still change an output then, and every seed below 2^16, is
// run one run pair at a time for the exact stopping time and excursion (exact_seeds):
// some 55 000 of the 3.2 million queued ones in 2^38 seeds.  A value that could leave 2^128 sends the
// seed to the widen list, re-run with 6 and then 8 limbs.  A request whose maxima are still zero
// gets a head start from a run's first seeds (scout).
//
// 2^38 seeds at 2^40, k 24: 5.9 ms, against 43 ms with run pairs in each lane.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "fill_once.h"
#include "kernels.h"
#include "range_variants.h"
#include "tables.h"

namespace cz {

typedef unsigned __int128 u128;

constexpr u32 KEEP9 = 0xCBu;     // n mod 9 in {0,1,3,6,7} survives (cu:488)
// Negative variant T'(m) = (3m-1)/2, m/2: m = 1 mod 3 (m > 1) is T' of the smaller
// (2m+1)/3 and m = 5 mod 9 (m > 5) is T'^3 of the smaller (8m+5)/9, so m mod 9 in
// {0,2,3,6,8} survives (and m = 5, the minimum of a cycle).
constexpr u32 KEEP9N = 0x14Du;
constexpr u32 OVF3 = 1u << 23;   // v >= 2^119 after an odd run: the next run could leave 128 bits
constexpr u32 ST_CAP = 1u << 20; // steps per seed before ERR_ITER_CAP

constexpr int DA = 485, DB = 306;         // D = DA F - DB i
constexpr u32 MIN_WINDOW_SEED = 1u << 16; // smaller seeds take the exact path
constexpr int LIM_MAX = 28000;            // D stays below 2^15 with a window to spare
// Rows of a claim (claim_rows): 2^36 seeds at 2^40, k 24, took 2.37 ms with first claims of a
// quarter of a warp's share (an entry's seeds are one lane's work, and some entries' take three
// times as long as others'), 1.81 with an eighth; 2^30 seeds 188 us with claims
// of at least 4 rows and 164 with 8 (opening a run costs a warp about 6 us).
constexpr u32 CLAIM_DIV = 4, CLAIM_CAP = 2, CLAIM_MIN = 8;
constexpr u32 RUN_MAX = 1024;             // rows of a run
constexpr u32 SLOWQ = 64;                 // seeds queued for the screen and for the exact path (31 left over + 32 new)
constexpr u32 SLOTS = 16;                 // runs that a warp's lanes may be in at a time
constexpr u32 GAPS = RUN_MAX + 16;
constexpr u32 DENSE_STEP = 576;           // integers below 2^k: one lane's seeds are this far apart (64 x 9, so that
                                          // they share their residue mod 9)

// Largest rise of D inside a window above both of its ends: a odd steps, then
// JW - a even ones.
constexpr int window_slack(int jw) {
  int s = 0;
  for (int a = 0; a <= jw; a++) {
    const int up = (DA - DB) * a, down = DB * (jw - a);
    const int m = up < down ? up : down;
    s = m > s ? m : s;
  }
  return s;
}

// Window tables, one per sign, layout and length.  Entry r: T^JW(r) << 11 | m << 7 | f, or
// (layout 1) f << 3, with f the odd steps and m = floor(-min D_i / 128) of the window's D_i (at
// most 15; 0 when none is negative): a seed with D < 128 m at the window's start falls
// below its start inside it.
constexpr u32 MIN_JW = 12, MAX_JW = 13;  // T^13(r) < 3^13 < 2^21
constexpr u32 WIN_M = 0x780u;
__device__ u32 g_win[2][2][MAX_JW - MIN_JW + 1][1u << MAX_JW];
// The largest D_i of the window, in units of 16, rounded up (for the screen).
__device__ uint8_t g_peak[2][MAX_JW - MIN_JW + 1][1u << MAX_JW];
__device__ u32 g_win_ready;  // 1: the tables above are filled
// P = U << 16 | D (k_range) changes by P_ODD with each odd step of a window and by P_STEP with each step.
constexpr u32 P_ODD = (u32)(-DA * 65535), P_STEP = (u32)(DB * 65535);

__global__ void k_win_tables() {
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
  for (u32 neg = 0; neg < 2; neg++)
    for (u32 jw = MIN_JW; jw <= MAX_JW; jw++) {
      if (t >> jw) continue;
      u32 x = t, f = 0;
      int D = 0, m = 0, h = 0;
      for (u32 i = 0; i < jw; i++) {
        if (x & 1u) {
          x = x + (x >> 1) + (neg ? 0u : 1u);  // (3x + 1) / 2, or (3x - 1) / 2
          f++;
          D += DA - DB;
        } else {
          x >>= 1;
          D -= DB;
        }
        m = min(m, D);
        h = max(h, D);
      }
      g_peak[neg][jw - MIN_JW][t] = (uint8_t)((h + 15) >> 4);  // at most 13 x 179 / 16 < 256
      const u32 e = (x << 11) | (min((u32)(-m) >> 7, 15u) << 7);
      g_win[neg][0][jw - MIN_JW][t] = e | f;
      g_win[neg][1][jw - MIN_JW][t] = e | (f << 3);
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// (a2:a1:a0) mod 9 (2^32 = 4, 2^64 = 7).
__device__ __forceinline__ u32 mod9_96(u32 a0, u32 a1, u32 a2) {
  return ((a0 % 9u) + 4u * (a1 % 9u) + 7u * (a2 % 9u)) % 9u;
}

// log2 of an excursion key's value (rounded down).
__device__ __forceinline__ float key_log2(ull ek) {
  return ek ? (float)((int)(ek >> 54) - 54) + __log2f(__ull2float_rd(ek & ((1ull << 54) - 1))) : -1.0f;
}

// log2 of n, from above.
__device__ __forceinline__ float log2_up(u128 n) {
  return 1e-5f + __log2f(__fmaf_ru(__ull2float_ru((u64)(n >> 64)), 18446744073709551616.0f, __ull2float_ru((u64)n)));
}

// Queue a seed for the 192/256-bit re-run.
__device__ __forceinline__ void widen_seed(const RangeArgs& A, u32 req, u32 n0, u32 n1, u32 n2) {
  const u32 wi = atomicAdd(&A.head->widened, 1u);
  if (wi < WIDEN_CAP) {
    A.lists->widen[wi] = WidenEntry{req, n0, n1, n2};
    atomicAdd(&A.recs[req].widened, 1ull);
  } else {
    atomicOr(&A.recs[req].errors, ERR_WIDEN_FULL);
    atomicAdd(&A.recs[req].failures, 1ull);
  }
}

// ------------------------------------------------------------------
// The exact path: up to 32 seeds, one per lane, from their starts.
// ------------------------------------------------------------------
enum : u32 { EX_NONE, EX_OK, EX_WIDEN, EX_CYCLE, EX_CAP };
struct ExactSeed {
  u32 how;   // EX_OK: fell below its start; EX_WIDEN: a value reached 2^119; EX_CYCLE: negative
             // variant, back at its start; EX_CAP: ST_CAP steps
  u32 st;    // stopping time
  u32 E[4];  // excursion
  u32 pairs; // STATS: run pairs taken
};

// Runs the seeds n of all lanes together (lanes with have = false idle): odd runs of at most
// 7 steps and even runs of at most 31 on four limbs.  Written for size: the code is
// fetched anew by every launch, and few seeds come here.
template <bool STATS>
__device__ __forceinline__ ExactSeed exact_run(u32 n0, u32 n1, u32 n2, bool have, bool neg) {
  ExactSeed R;
  R.how = EX_NONE;
  R.st = 0;
  if constexpr (STATS) R.pairs = 0;
  R.E[0] = n0;
  R.E[1] = n1;
  R.E[2] = n2;
  R.E[3] = 0;
  // the run state: n + 1, or n - 1 for the negative variant
  u32 v0 = neg ? n0 - 1 : n0 + 1;
  const u32 c0 = neg ? (n0 == 0 ? FULL : 0u) : (v0 == 0);
  u32 v1 = n1 + c0;
  const u32 c1 = neg ? (c0 && n1 == 0 ? FULL : 0u) : (c0 & (v1 == 0));
  u32 v2 = n2 + c1, v3 = (!neg && c1 && v2 == 0) ? 1u : 0u;
  const u32 nbl = bitlen96(n0, n1, n2);
  bool alive = have;
#pragma unroll 1
  while (__any_sync(FULL, alive)) {
    if (alive) {
      if constexpr (STATS) R.pairs++;
      const u32 a = ctz32(v0 | 0x80u);
      odd_run4(v0, v1, v2, v3, a, pow3_le7(a));
      u32 x0, x1, x2, x3;  // the value
      if (neg) {
        x0 = v0 + 1;
        x1 = v1;
        x2 = v2;
        x3 = v3;
        add_carry3(x1, x2, x3, x0 == 0);
      } else {
        x0 = v0 - 1;
        x1 = v1 - (v0 == 0);
        x2 = v2 - ((v0 | v1) == 0);
        x3 = v3 - ((v0 | v1 | v2) == 0);
      }
      const u32 b = ctz32(x0 | 0x80000000u);
      const u32 w0 = __funnelshift_r(x0, x1, b), w1 = __funnelshift_r(x1, x2, b);
      const u32 w2 = __funnelshift_r(x2, x3, b), w3 = x3 >> b;
      if (v3 >= OVF3) {
        R.how = EX_WIDEN;
      } else {
        if (R.E[3] < x3 || (R.E[3] == x3 && lt96c(R.E[0], R.E[1], R.E[2], x0, x1, x2))) {
          R.E[0] = x0;
          R.E[1] = x1;
          R.E[2] = x2;
          R.E[3] = x3;
        }
        R.st += a;
        if ((w3 == 0) & (b != 0) & lt96c(w0, w1, w2, n0, n1, n2)) {
          R.st += first_below(x0, x1, x2, x3, n0, n1, n2, nbl);
          R.how = EX_OK;
        } else if (neg && ((w0 ^ n0) | (w1 ^ n1) | (w2 ^ n2) | w3) == 0) {
          R.how = EX_CYCLE;
        } else {
          R.st += b;
          if (R.st > ST_CAP) R.how = EX_CAP;
          v0 = neg ? w0 - 1 : w0 + 1;
          v1 = w1;
          v2 = w2;
          v3 = w3;
          if (neg) {  // (w >= 1)
            v1 -= w0 == 0;
            v2 -= (w0 | w1) == 0;
            v3 -= (w0 | w1 | w2) == 0;
          } else {
            add_carry3(v1, v2, v3, v0 == 0);
          }
        }
      }
      alive = R.how == EX_NONE;
    }
  }
  return R;
}

// The candidate of the lane with lead goes to the launch's list, or, when that is full, into the
// record under its lock.  The keys of the record rise at once, for the other warps' limits;
// the maxima themselves are settled after the kernel, where most candidates are already
// beaten: with the lock taken here, the warps that offer at the same time (at a launch's
// start and end) waited for one another, 60 us of a 245 us launch of 2^30 seeds.  All lanes
// together; the lock's loop has a vote for its condition, as a spin by one lane makes the
// compiler take the warp to be diverged at every later vote (k_range: three instructions each).
__device__ __forceinline__ void offer(const RangeArgs& A, bool lead, const RangeCand& c) {
  ReqRec* r = A.recs + c.req;
  bool full = false;
  if (lead) {
    if (c.kind == 0) atomicMax(&r->st_key, (ull)c.st);
    else atomicMax(&r->e_key, key_of<4>(c.E));
    const u32 i = atomicAdd(&A.head->cands, 1u);
    full = i >= CAND_CAP;
    if (!full) A.lists->cand[i] = c;
  }
  rec_offer_vote<false>(r, full, c.kind, 0, c.st, c.E, c.seed);
}

// The exact path for the warp's queued seeds e (n limbs 0..2, request), one per
// lane with have: failures, widening and errors are recorded, and of the seeds of
// one request that may raise a maximum only the best is offered (larger, or equal
// with a smaller seed).  STATS: counts the lane's run pairs and the warp's offers.
template <bool STATS>
__device__ __forceinline__ void exact_seeds(const RangeArgs& A, uint4 e, bool have, ull* xs) {
  const u32 lane = lane_id();
  const ExactSeed R = exact_run<STATS>(e.x, e.y, e.z, have, A.negative != 0);
  if constexpr (STATS) xs[RS_RUN_PAIRS] += R.pairs;
  ReqRec* rec = A.recs + e.w;
  bool ps = false, pe = false;
  if (R.how == EX_OK) {
    ps = R.st >= *(volatile ull*)&rec->st_key;
    pe = key_of<4>(R.E) >= *(volatile ull*)&rec->e_key;
  } else if (R.how == EX_WIDEN) {
    widen_seed(A, e.w, e.x, e.y, e.z);
  } else if (R.how != EX_NONE) {
    if (R.how == EX_CAP) atomicOr(&rec->errors, ERR_ITER_CAP);
    atomicAdd(&rec->failures, 1ull);
  }
  u32 pm = __ballot_sync(FULL, ps | pe);
#pragma unroll 1
  while (pm) {
    const u32 req = __shfl_sync(FULL, e.w, __ffs(pm) - 1);
    const bool in = (ps | pe) & (e.w == req);
    const u32 sm = __reduce_max_sync(FULL, (in & ps) ? R.st + 1 : 0u);  // 0: nobody
    u32 cs = __ballot_sync(FULL, in & ps & (R.st + 1 == sm));
    u32 ce = __ballot_sync(FULL, in & pe);
#pragma unroll
    for (int i = 3; i >= 0; i--) {  // the lanes with the largest excursion
      const u32 m = __reduce_max_sync(FULL, ((ce >> lane) & 1u) ? R.E[i] : 0u);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && R.E[i] == m);
    }
    const u32 nl[3] = {e.x, e.y, e.z};
#pragma unroll
    for (int i = 2; i >= 0; i--) {  // the smallest seed of each
      const u32 a = __reduce_min_sync(FULL, ((cs >> lane) & 1u) ? nl[i] : FULL);
      cs = __ballot_sync(FULL, ((cs >> lane) & 1u) && nl[i] == a);
      const u32 b = __reduce_min_sync(FULL, ((ce >> lane) & 1u) ? nl[i] : FULL);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && nl[i] == b);
    }
#pragma unroll 1
    for (u32 kind = 0; kind < 2; kind++) {
      const u32 set = kind ? ce : cs;
      if (STATS && set && lane == 0) xs[RS_OFFERS]++;
      if (set)
        offer(A, lane == (u32)__ffs(set) - 1,
              RangeCand{req, kind, R.st, 0u, {R.E[0], R.E[1], R.E[2], R.E[3]}, {e.x, e.y, e.z, 0u}});
    }
    pm &= ~__ballot_sync(FULL, in);
  }
}

// ------------------------------------------------------------------
// The range kernel.
// ------------------------------------------------------------------

// A run of rows staged for a warp (warp-uniform): rows of one chunk of 64 entries
// over consecutive or kept blocks, or (kind 1) rows of 64 consecutive integers, which the
// lanes take as up to 576 entries (integers) with every 576th integer after each.
struct StagedRun {
  ull q_lo;          // kind 0: first block (low 64 bits); kind 1: first integer
  u32 q_hi;          // kind 0: first block, bits 64..95
  u32 ph;            // index in S.gap of the first block's offset
  u32 sbase, ents;   // kind 0: first entry in the survivor table; entries
  u32 rows;          // kind 0: rows; kind 1: integers
  u32 items;         // work items (rows of 64)
  u32 req, kind, mod9, valid;
  float lgn;         // log2 of the largest seed, from above
  u32 small;         // seeds too small for windows
};

// Per-warp state in shared memory.
struct RangeWarp {
  uint4 slow[SLOWQ];                // seeds for the screen: n limbs 0..2, request
  uint4 exact[SLOWQ];               // seeds for the exact path
  uint4 stage[2][RANGE_ITEM];       // survivor entries of the current run and the staged one, in turn (cp.async)
  uint4 base[32];                   // per lane: its entry's seed at gap 0 (limbs 0..2, modulo 2^96) and request
  ulonglong2 keys;                  // st_key, e_key of the staged run's request (cp.async)
  ulonglong2 cur;                   // the current request's keys, as last read
  StagedRun run[SLOTS];             // the staged run, the current one and the earlier ones lanes are still in
  RangeSeg seg;                     // cached segment
  ull pos, claim_hi, seg_lo, seg_hi;
  ull acc_seeds, acc_rows;          // of the current request, not yet added to its record
  u32 req;                          // the current request
  int lim, elim;                    // the current run's limits
  u32 ud;
};

// Shared memory of a block: window table, powers of 3, then the warps' state.
template <int JW, int WARPS>
struct RangeShared {
  u32 win[1u << JW];
  uint8_t peak[1u << JW];
  uint2 cls[16];   // 4 3^f, P's change by a window with f odd steps (less ud)
  u32 last[WARPS]; // seeds each warp has left for the exact path at the end
  ull p3[42];      // 3^f
  u32 gap[2 * GAPS]; // offsets of blocks: [j] of the j-th that keeps a class (from one with (q 2^k) mod 9 = 0
                     // on), [GAPS + j] j
  u32 phase[9];      // index in gap of the first offset q with (q 2^k) mod 9 = the index
  RangeWarp w[WARPS];
};

extern __shared__ __align__(16) unsigned char range_smem[];

// Rows of the next claim: a quarter of a warp's share of the rows left, so that the warps
// finish together, but no more than the first claim's (an eighth of its share of all) and
// no less than 8 where a share has as many.
__device__ __forceinline__ u32 claim_rows(ull left, u32 nwarps, u32 most) {
  // (64-bit divisions are function calls)
  const u32 l = (u32)min(left, 0xFFFFFFFFull) / nwarps;
  return min(most, max(l / CLAIM_DIV, max(1u, min(CLAIM_MIN, l))));
}

// Advances to the next run (claiming rows as needed) and starts copying its
// survivor entries and its request's keys, so that they arrive while the current
// run is worked on.  Warp-uniform.
template <class SH>
__device__ __forceinline__ void stage_next(const SH& S, RangeWarp& W, u32 ring, const RangeArgs& A, u32 lane,
                                           u32 nwarps, u32 first) {
  StagedRun& nxt = W.run[ring & (SLOTS - 1)];
  ull pos = W.pos;
  ull claim_hi = W.claim_hi;
  // (votes around warp-uniform conditions: the compiler then knows that they are)
  if (__any_sync(FULL, pos >= claim_hi)) {
    const u32 claim = claim_rows(A.item_limit - claim_hi, nwarps, first);
    ull c = 0;
    if (lane == 0) c = atomicAdd(&A.head->item_cursor, (ull)claim);
    c = __shfl_sync(FULL, c, 0) + (ull)first * nwarps;
    if (__any_sync(FULL, c >= A.item_limit)) {
      __syncwarp();
      if (lane == 0) nxt.valid = 0;
      __syncwarp();
      return;
    }
    pos = c;
    claim_hi = min(c + claim, A.item_limit);
    __syncwarp();
    if (lane == 0) W.claim_hi = claim_hi;
  }
  if (__any_sync(FULL, pos < W.seg_lo || pos >= W.seg_hi)) {
    u32 lo = 0, span = __reduce_max_sync(FULL, A.nsegs);  // the last segment beginning at or before pos: 32 probes at a time
#pragma unroll 1
    while (__any_sync(FULL, span > 1)) {
      const u32 step = (span + 31) >> 5, at = lane * step;
      const bool below = at < span && A.segs[lo + at].item_begin <= pos;
      const u32 j = 31u - __clz(__ballot_sync(FULL, below));  // (lane 0 is always below)
      lo += j * step;
      span = min(step, span - j * step);
    }
    __syncwarp();
    const u32* src = reinterpret_cast<const u32*>(A.segs + lo);
    if (lane < sizeof(RangeSeg) / 4) reinterpret_cast<u32*>(&W.seg)[lane] = src[lane];
    if (lane == 0) {
      W.seg_lo = A.segs[lo].item_begin;
      W.seg_hi = (lo + 1 < A.nsegs) ? A.segs[lo + 1].item_begin : A.item_limit;
    }
    __syncwarp();
  }
  const ull local = pos - W.seg_lo + (((ull)W.seg.local0_hi << 32) | W.seg.local0_lo);
  u32 items = (u32)min((ull)RUN_MAX, min(claim_hi, W.seg_hi) - pos);
  StagedRun it;
  it.req = W.seg.req;
  it.kind = W.seg.kind;
  it.mod9 = W.seg.mod9;
  it.valid = 1;
  if (it.kind == 0) {  // segments hold fewer than 2^32 rows
    const u32 l32 = (u32)local, nq = W.seg.nq;
    const u32 chunk = l32 / nq, qi = l32 - chunk * nq;
    items = min(items, nq - qi);
    it.rows = items;
    u128 q = ((u128)W.seg.q_hi << 64) | W.seg.q_lo;
    if (W.seg.qstride == 9) {
      // n mod 9 of the first kept block's seeds gives its place among the kept ones (2^6 = 1 mod 9)
      const u32 ph0 = S.phase[(mod9_96((u32)q, (u32)(q >> 32), (u32)(q >> 64)) * (u32)((1ull << (A.k % 6)) % 9ull) + W.seg.mod9) % 9u];
      q += (u128)(qi / 5u) * 9u + (S.gap[ph0 + qi % 5u] - S.gap[ph0]);
      it.ph = (ph0 + qi) % 5u;
    } else {
      q += qi;
      it.ph = GAPS;
    }
    it.q_lo = (u64)q;
    it.q_hi = (u32)(q >> 64);
    it.sbase = W.seg.s_lo + chunk * RANGE_ITEM;
    it.ents = min(RANGE_ITEM, W.seg.s_hi - it.sbase);
    const uint4* T = reinterpret_cast<const uint4*>(A.table);
#pragma unroll
    for (u32 j = 0; j < RANGE_ITEM / 32; j++)
      if (j * 32 + lane < it.ents) cp_async16(&W.stage[ring & 1u][j * 32 + lane], T + it.sbase + j * 32 + lane);
    const u128 ql = q + (S.gap[it.ph + items - 1] - S.gap[it.ph]) + 1;
    it.lgn = (float)A.k + log2_up(ql);
    it.small = A.k < 16 && it.q_hi == 0 && it.q_lo < (MIN_WINDOW_SEED >> A.k);
  } else {
    it.q_lo = W.seg.q_lo + local * DENSE_ITEM;
    it.q_hi = it.sbase = 0;
    it.ph = GAPS;
    it.rows = (u32)min((ull)items * DENSE_ITEM, W.seg.d_hi - it.q_lo);
    it.ents = min(it.rows, DENSE_STEP);
    it.lgn = log2_up(it.q_lo + it.rows);
    it.small = it.q_lo < MIN_WINDOW_SEED;
  }
  if (lane == 0) cp_async16(&W.keys, &A.recs[it.req].st_key);
  cp_async_commit();
  it.items = items;
  __syncwarp();
  if (lane == 0) {
    W.pos = pos + items;
    nxt = it;
  }
  __syncwarp();
}

// The limits of a request's windows for the seeds of one run, from its keys.
struct RunLimits {
  int lim;   // a seed may take a window while D <= lim (0 < D); below 0: none
  int elim;  // 306 log2 of the least excursion that counts, over the run's largest seed
  u32 ud;    // what U loses by a window (see k_range), in P's place, negated
};

template <int L, int JW>
__device__ __forceinline__ RunLimits run_limits(ulonglong2 keys, float lgn, int s0) {
  const ull sk = keys.x;
  RunLimits R;
  // the margins cover the float arithmetic and the 0.0024 of the bound on T^i(n)
  R.elim = (int)floorf((float)DB * (key_log2(keys.y) - lgn)) - 2;
  const int lo = (int)floorf((float)DB * ((float)(32 * L - 2) - lgn)) - 2;  // values stay in L words
  R.lim = min(min(R.elim, lo), LIM_MAX) - window_slack(JW) - 1;
  const int thr = (int)min(sk, 485ull);  // D decides only below 485 steps
  const int wmax = thr - 1 >= s0 ? (thr - 1 - s0) / JW : 0;
  if (wmax < 1) R.lim = -1;
  R.ud = (R.lim > 0 ? (u32)(-((R.lim + wmax - 1) / wmax)) << 16 : 0u) + P_STEP * JW;
  return R;
}

// A window's entry e for the value y = 4 x (bits 0 and 1 are arbitrary): c.x = 4 3^f, c.y = P's change
// less ud.  With two words the multiply-add pipe has room: the class's multiplier alone is
// loaded, half the wavefronts, and P's change computed.  With more the pipe is the
// busiest, and the pair is loaded from the other table layout.
template <int L, class SH>
__device__ __forceinline__ uint2 window_class(u32 e, const SH& S, u32 cls, u32 ud, u32 eight) {
  uint2 c;
  if (L == 2) {
    const u32 f = e & 0xFu;
    asm("{\n\t.reg .u32 a;\n\tmad.lo.u32 a, %1, %2, %3;\n\tld.shared.u32 %0, [a];\n\t}" : "=r"(c.x) : "r"(f), "r"(eight), "r"(cls));
    c.y = f * P_ODD + ud;
  } else {
    c = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(S.cls) + (e & 0x78u));
    c.y += ud;
  }
  return c;
}

// y = 4 T^JW(x) from y = 4 x, t = 4 T^JW(r) (and two bits of m) and m = 4 3^f.
template <int L, int JW>
__device__ __forceinline__ void advance(u32* y, u32 t, u32 m) {
  u64 w = t;
#pragma unroll
  for (int i = 0; i < L; i++) {
    const u32 a = (i + 1 < L) ? __funnelshift_r(y[i], y[i + 1 < L ? i + 1 : i], JW + 2) : (y[i] >> (JW + 2));
    if (i + 1 < L) {
      w += (u64)a * m;
      y[i] = (u32)w;
      w >>= 32;
    } else {
      y[i] = a * m + (u32)w;
    }
  }
}

// One window of a value y of four words and P's change by it, for a kernel of L words.  Returns a
// word with bit 15 set when the seed fell below its start inside the window.
template <int L, int JW, class SH>
__device__ __forceinline__ u32 window(u32* y, u32& P, const SH& S, u32 mone) {
  const u32 e = S.win[(y[0] >> 2) & ((1u << JW) - 1u)], f = L == 2 ? e & 0xFu : (e >> 3) & 0xFu;
  const u32 low = P + (e & WIN_M) * mone;
  advance<4, JW>(y, e >> 9, S.cls[f].x);
  P += f * P_ODD + P_STEP * JW;
  return P | low;
}

// The value of a lane's entry at a block offset: y = yb + p4 g.
template <int L>
__device__ __forceinline__ void value_at(u32* y, const u32* yb, u64 p4, u32 g) {
  if (L == 2) {
    const u64 v = ((((u64)yb[1] << 32) | yb[0]) + (u64)(u32)p4 * g) + ((u64)((u32)(p4 >> 32) * g) << 32);
    y[0] = (u32)v;
    y[1] = (u32)(v >> 32);
  } else {
    u64 t = (u64)(u32)p4 * g + yb[0];
    y[0] = (u32)t;
    t = (u64)(u32)(p4 >> 32) * g + (t >> 32) + yb[1];
    y[1] = (u32)t;
    if (L == 3) {
      y[L > 2 ? 2 : 0] = yb[L > 2 ? 2 : 0] + (u32)(t >> 32);
    } else {
      t = (u64)yb[L > 2 ? 2 : 0] + (t >> 32);
      y[L > 2 ? 2 : 0] = (u32)t;
      y[L > 3 ? 3 : 0] = yb[L > 3 ? 3 : 0] + (u32)(t >> 32);
    }
  }
}

// The hot step: one window of every lane's seed; a lane whose seed fell below its
// start inside it takes its entry's next one, y = yb + p4 g with g the block offset at the
// shared-memory address ti, which moves on.  A seed at a limit (P < 0) stays as it is.
// Everything that only some lanes do is predicated, without a select or a branch; mone and one
// are -1 and 1, unknown to the compiler: multiplying by them puts additions on the
// multiply-add pipe, the ALU being the busy one.  Bound by the shared-memory loads
// (the window's entry in ~3.5 wavefronts of random banks, its class, the offset), by
// issue and the ALU, at 68, 79 and 71 % with two words; 2^38 seeds at 2^40 took 6.95 ms with the
// taken seed selected and the limit voted on after every window, 5.93 so (and 8.1 with three words).
template <int L, int JW, class SH>
__device__ __forceinline__ void hot_step(u32* y, const u32* yb, u64 p4, u32& g, u32& P, u32 Pn, u32 ud, u32& ti,
                                         const SH& S, u32 cls, u32 one, u32 mone, u32 eight) {
  const u32 e = *reinterpret_cast<const u32*>(reinterpret_cast<const char*>(S.win) + (y[0] & (((1u << JW) - 1u) << 2)));
  const uint2 c = window_class<L>(e, S, cls, ud, eight);
  const u32 low = P + (e & WIN_M) * mone;
  u32 yn[L];
  value_at<L>(yn, yb, p4, g);
  advance<L, JW>(y, e >> 9, c.x);
  if (L == 2) {
    asm("{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 w;\n\t"
        "setp.lt.s32 p, %0, 0;\n\t"
        "@!p add.u32 %0, %0, %5;\n\t"
        "or.b32 w, %0, %6;\n\t"
        "and.b32 w, w, 0x8000;\n\t"
        "setp.ne.and.u32 q, w, 0, !p;\n\t"
        "@q mul.lo.u32 %0, %7, %8;\n\t"
        "@q mad.lo.u32 %1, %8, 4, %1;\n\t"
        "selp.b32 %3, %9, %3, q;\n\t"
        "selp.b32 %4, %10, %4, q;\n\t"
        "@q ld.shared.u32 %2, [%1];\n\t"
        "}"
        : "+r"(P), "+r"(ti), "+r"(g), "+r"(y[0]), "+r"(y[1])
        : "r"(c.y), "r"(low), "r"(Pn), "r"(one), "r"(yn[0]), "r"(yn[1]));
  } else if (L == 3) {
    asm("{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 w;\n\t"
        "setp.lt.s32 p, %0, 0;\n\t"
        "@!p add.u32 %0, %0, %6;\n\t"
        "or.b32 w, %0, %7;\n\t"
        "and.b32 w, w, 0x8000;\n\t"
        "setp.ne.and.u32 q, w, 0, !p;\n\t"
        "@q mul.lo.u32 %0, %8, %9;\n\t"
        "@q mad.lo.u32 %1, %9, 4, %1;\n\t"
        "selp.b32 %3, %10, %3, q;\n\t"
        "selp.b32 %4, %11, %4, q;\n\t"
        "selp.b32 %5, %12, %5, q;\n\t"
        "@q ld.shared.u32 %2, [%1];\n\t"
        "}"
        : "+r"(P), "+r"(ti), "+r"(g), "+r"(y[0]), "+r"(y[1]), "+r"(y[2 % L])
        : "r"(c.y), "r"(low), "r"(Pn), "r"(one), "r"(yn[0]), "r"(yn[1]), "r"(yn[2 % L]));
  } else {
    asm("{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 w;\n\t"
        "setp.lt.s32 p, %0, 0;\n\t"
        "@!p add.u32 %0, %0, %7;\n\t"
        "or.b32 w, %0, %8;\n\t"
        "and.b32 w, w, 0x8000;\n\t"
        "setp.ne.and.u32 q, w, 0, !p;\n\t"
        "@q mov.b32 %0, %9;\n\t"
        "@q mad.lo.u32 %1, %10, 4, %1;\n\t"
        "selp.b32 %3, %11, %3, q;\n\t"
        "selp.b32 %4, %12, %4, q;\n\t"
        "selp.b32 %5, %13, %5, q;\n\t"
        "selp.b32 %6, %14, %6, q;\n\t"
        "@q ld.shared.u32 %2, [%1];\n\t"
        "}"
        : "+r"(P), "+r"(ti), "+r"(g), "+r"(y[0]), "+r"(y[1]), "+r"(y[2 % L]), "+r"(y[3 % L])
        : "r"(c.y), "r"(low), "r"(Pn), "r"(one), "r"(yn[0]), "r"(yn[1]), "r"(yn[2 % L]), "r"(yn[3 % L]));
  }
}

// The seed of a lane for the screen: its entry's seed at gap 0, plus g blocks (kind 0) or
// steps of 576.
__device__ __forceinline__ uint4 seed_at(uint4 b, u32 g, u32 shift, u32 mul) {
  const u64 d = (u64)(g * mul) << shift;  // below 2^12 2^34, or 2^12 576
  u32 n0, n1, n2;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, 0;"
      : "=r"(n0), "=r"(n1), "=r"(n2)
      : "r"(b.x), "r"(b.y), "r"(b.z), "r"((u32)d), "r"((u32)(d >> 32)));
  return make_uint4(n0, n1, n2, b.w);
}

// The screen: which of the seeds e (n limbs 0..2, request; lanes with have) may still change an
// output under their requests' keys as they are now.  Windows from the seed's start
// with four words, the excursion bounded window by window by its own largest D, so that
// what the window loop's coarser limits stop (a bit of slack and the words' width among
// them) seldom goes on to the exact path.  STATS: counts the lane's windows.
template <int L, int JW, bool STATS, class SH>
__device__ __forceinline__ bool screen(const SH& S, const RangeArgs& A, uint4 e, bool have, ull* xs) {
  const u128 n = ((u128)e.z << 64) | ((u64)e.y << 32) | e.x;
  const ReqRec* r = A.recs + e.w;
  const ull sk = have ? *(volatile const ull*)&r->st_key : 0ull, ek = have ? *(volatile const ull*)&r->e_key : 0ull;
  const float lgn = log2_up(n);
  const int lim = min((int)floorf((float)DB * (fminf(key_log2(ek), 126.0f) - lgn)) - 2, LIM_MAX);
  const int smax = (int)min(sk, 485ull) - 1 - JW;  // a window may start after this many steps
  bool exact = have && n < MIN_WINDOW_SEED, alive = have && !exact;
  u32 y[4] = {e.x << 2, __funnelshift_l(e.x, e.y, 2), __funnelshift_l(e.y, e.z, 2), e.z >> 30};
  u32 P = 0;  // D in its low half
#pragma unroll 1
  for (int s = 0; __any_sync(FULL, alive); s += JW) {
    const int peak = 16 * (int)S.peak[(y[0] >> 2) & ((1u << JW) - 1u)];
    if (alive && (s > smax || (int)(short)P + peak >= lim)) {
      exact = true;
      alive = false;
    }
    if constexpr (STATS) xs[RS_SCREEN_WINDOWS] += alive;
    const u32 t = window<L, JW>(y, P, S, A.mone);
    P &= 0xFFFFu;
    if (t & 0x8000u) alive = false;
  }
  return exact;
}

// A head start for the keys of a request that has none yet: under zero keys every seed
// would go to the exact path.  The run's first seeds (one per lane, value y = 4 T^k(n), D0 in
// P) take windows while they certainly stay above their starts; the values at the windows'
// ends and the steps survived are lower bounds of the request's maxima.  Returns them as
// keys.
template <int L, int JW, class SH>
__device__ __forceinline__ ulonglong2 scout(const SH& S, const RangeArgs& A, u32* y, u32 P, float lgn, int s0,
                                            bool have) {
  const int lim = min((int)floorf((float)DB * (126.0f - lgn)) - 2, LIM_MAX) - window_slack(JW) - 1;
  ull ek = 0;
  int s = 0;  // steps survived
  bool alive = have && (int)P <= lim;
#pragma unroll 1
  for (int t = s0; __any_sync(FULL, alive); t += JW) {  // (the vote alone: known to be uniform)
    alive = alive && t < 485 - JW;
    if (alive) {
      const u32 x[4] = {__funnelshift_r(y[0], y[1], 2), __funnelshift_r(y[1], y[2], 2), __funnelshift_r(y[2], y[3], 2),
                        y[3] >> 2};
      ek = max(ek, key_of<4>(x));
      s = t + 1;
    }
    // the window's least D is above -128 (m + 1), or any when m is clipped: on while it is
    // certain that the seed does not fall inside the window
    const u32 m = S.win[(y[0] >> 2) & ((1u << JW) - 1u)] & WIN_M;
    if (P < (m == WIN_M ? (u32)(DB * JW) : m + 128u)) alive = false;
    window<L, JW>(y, P, S, A.mone);
    P &= 0xFFFFu;
    if ((int)P > lim) alive = false;
  }
  s = (int)__reduce_max_sync(FULL, (u32)s);
#pragma unroll 1
  for (u32 d = 16; d; d >>= 1) ek = max(ek, (ull)__shfl_xor_sync(FULL, ek, d));
  return make_ulonglong2((ull)s, ek);
}

// The kernel.  It makes no function calls: with one, the compiler takes the warp to be
// possibly diverged at every vote and spends three instructions on each.  L: words of a value; JW:
// window length; WARPS per block, one block per SM; STATS: the diagnostics form, which counts into
// A.stats (RangeStat).
template <int L, int JW, int WARPS, bool STATS>
__global__ void __launch_bounds__(WARPS * 32, 1) k_range(const __grid_constant__ RangeArgs A) {
  typedef RangeShared<JW, WARPS> Shared;
  Shared& S = *reinterpret_cast<Shared*>(range_smem);
  {
    const uint4* src = reinterpret_cast<const uint4*>(g_win[A.negative ? 1 : 0][L == 2 ? 0 : 1][JW - MIN_JW]);
#pragma unroll 1
    for (u32 i = threadIdx.x; i < (1u << JW) / 4; i += WARPS * 32) cp_async16(reinterpret_cast<uint4*>(S.win) + i, src + i);
    const uint4* pk = reinterpret_cast<const uint4*>(g_peak[A.negative ? 1 : 0][JW - MIN_JW]);
#pragma unroll 1
    for (u32 i = threadIdx.x; i < (1u << JW) / 16; i += WARPS * 32) cp_async16(reinterpret_cast<uint4*>(S.peak) + i, pk + i);
    cp_async_commit();
  }
  if (threadIdx.x < 42) {
    ull p = 1;
#pragma unroll 1
    for (u32 i = 0; i < threadIdx.x; i++) p *= 3;
    S.p3[threadIdx.x] = p;
    if (threadIdx.x < 16) S.cls[threadIdx.x] = make_uint2(4u * (u32)p, threadIdx.x * P_ODD);
  }
#pragma unroll 1
  for (u32 i = threadIdx.x; i < GAPS; i += WARPS * 32) {
    const u32 keep9 = A.negative ? KEEP9N : KEEP9, k9 = (u32)((1ull << (A.k % 6)) % 9ull);
    u32 q = 0, c = i % 5u;  // the c-th kept offset below 9
#pragma unroll 1
    while (!((keep9 >> (q * k9 % 9u)) & 1u) || c-- != 0) q++;
    S.gap[i] = q + i / 5u * 9u;
    S.gap[GAPS + i] = i;
    if (i < 5) S.phase[q * k9 % 9u] = i;
  }
  __syncthreads();
  const u32 lane = lane_id();
  RangeWarp& W = S.w[threadIdx.x >> 5];
  const u32 nwarps = gridDim.x * WARPS;
  const u32 first = claim_rows(A.item_limit, nwarps * CLAIM_CAP, RUN_MAX);  // rows of each warp's first claim, neighbours in different blocks
  if (lane == 0) {
    W.pos = min((ull)first * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x), A.item_limit);
    W.claim_hi = min(W.pos + first, A.item_limit);
    W.seg_lo = 1;
    W.seg_hi = 0;
    W.acc_seeds = W.acc_rows = 0;
    W.req = FULL;
    W.cur = W.keys = make_ulonglong2(0ull, 0ull);
    W.run[SLOTS - 1] = StagedRun{0, 0, 0, 0, 0, 0, 0, FULL, 0, 0, 1, 64.0f, 0};  // a run without entries comes first
  }
  cp_async_wait_all();
  __syncthreads();

  ull xs[STATS ? RANGE_STATS : 1], xt;  // STATS: counts; the clock at the last look
  if constexpr (STATS) {
    for (ull& x : xs) x = 0;
    xt = clock64();
  }
  auto clocked = [&](int what) {  // the cycles since then
    if constexpr (STATS) {
      const ull t = clock64();
      xs[what] += t - xt;
      xs[RS_CYCLES] += t - xt;
      xt = t;
    }
  };
  u32 slow = 0, ex = 0;             // seeds queued for the screen and for the exact path
  u32 ring = FULL, next = 0, ents = 0;  // runs begun less one; entries of the current run handed out, of all
  int thr = 0;                      // idle lanes that call for new entries
  bool last = false, end = false;   // no more runs; the block's last seeds for the exact path
  // Lane state: a seed is y, P; the next one of its entry is at the shared-memory address
  // ti of gap, with Pn and the value yb + p4 g, g being that offset.  ti >= te: the lane is idle (and runs on
  // beyond its rows, to no effect); pk: D0 and emax of the entry, bit 31 for kind 1; slot: its run's.
  const u32 cls = (u32)__cvta_generic_to_shared(S.cls), gaps = (u32)__cvta_generic_to_shared(S.gap);
  u32 y[L], yb[L], P = 0xC000u, Pn = 0xC000u, ud = 0, pk = 0, slot = 0, ti = gaps, te = gaps, g = 0;
  u64 p4 = 0;
#pragma unroll
  for (int i = 0; i < L; i++) y[i] = yb[i] = 0;
  // P = U << 16 | D with U = lim - D less u for every window taken: u wmax >= lim > lim - D, so
  // that U turns negative when D passes lim (less u per window) and after wmax windows at
  // the latest; a seed with a negative U goes to the exact path.  Pn: P at a seed's start.
  auto limits = [&](int lim, int elim, u32 u, u32 small) {
    const int D0 = (int)(short)pk, emx = DB * (int)((pk >> 16) & 0xFFu);
    const bool none = small || lim < D0 || emx >= elim;
    Pn = none ? 0x80000000u : ((u32)lim << 16) - (u32)(D0 * 65535);
    ud = u;
  };
  auto gap_at = [&](u32 t) {
    u32 v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(t));
    return v;
  };
  auto take_next = [&]() {
    P = Pn;
    value_at<L>(y, yb, p4, g);
    ti += 4;
    g = gap_at(ti);
  };
  // One loop, one place for each kind of work: the exact path's registers then never
  // meet the window loop's (the lanes' state is put away around it).
  for (;;) {
    if (slow >= 32u || (last && slow) || (end && ex)) {
      volatile u32 keep[2 * L + 9];
#pragma unroll
      for (int i = 0; i < L; i++) {
        keep[i] = y[i];
        keep[L + i] = yb[i];
      }
      keep[2 * L] = P;
      keep[2 * L + 1] = ud;
      keep[2 * L + 2] = ti;
      keep[2 * L + 3] = (u32)p4;
      keep[2 * L + 4] = (u32)(p4 >> 32);
      keep[2 * L + 5] = pk;
      keep[2 * L + 6] = slot;
      keep[2 * L + 7] = Pn;
      keep[2 * L + 8] = te;
      __syncwarp();
      if (slow) {
        const u32 cnt = min(slow, 32u);
        slow -= cnt;
        const uint4 e = lane < cnt ? W.slow[slow + lane] : make_uint4(0u, 0u, 0u, 0u);
        const bool on = screen<L, JW, STATS>(S, A, e, lane < cnt, xs);
        if constexpr (STATS) {
          xs[RS_SCREENED] += lane < cnt;
          clocked(RS_CYCLES_SCREEN);
        }
        const u32 b = __ballot_sync(FULL, on);
        if (on) W.exact[ex + __popc(b & ((1u << lane) - 1u))] = e;
        ex += __popc(b);
        __syncwarp();
      }
      if (ex >= 32u || end) {
        const u32 cnt = min(ex, 32u);
        ex -= cnt;
        exact_seeds<STATS>(A, lane < cnt ? W.exact[ex + lane] : make_uint4(0u, 0u, 0u, 0u), lane < cnt, xs);
        // (in every form: without this branch 2^32 seeds with k 16 took 406 us and not 397)
        if (A.stats && lane == 0) atomicAdd(&A.stats[RS_EXACT], (ull)cnt);
        clocked(RS_CYCLES_EXACT);
      }
#pragma unroll
      for (int i = 0; i < L; i++) {
        y[i] = keep[i];
        yb[i] = keep[L + i];
      }
      P = keep[2 * L];
      ud = keep[2 * L + 1];
      ti = keep[2 * L + 2];
      g = gap_at(ti);
      p4 = ((u64)keep[2 * L + 4] << 32) | keep[2 * L + 3];
      pk = keep[2 * L + 5];
      slot = keep[2 * L + 6];
      Pn = keep[2 * L + 7];
      te = keep[2 * L + 8];
      if (!end) {  // the current request's keys may have risen
        const ReqRec* r = A.recs + W.req;
        const ull sk = *(volatile const ull*)&r->st_key, ek = *(volatile const ull*)&r->e_key;
        __syncwarp();
        if (lane == 0) {
          W.cur.x = max(W.cur.x, sk);
          W.cur.y = max(W.cur.y, ek);
        }
        __syncwarp();
#pragma unroll 1
        for (u32 pass = 0; pass < 2; pass++) {  // the current run's limits, then those of the lane's own run
          const StagedRun& ru = W.run[pass ? slot : (ring - 1u) & (SLOTS - 1)];
          const RunLimits rl = run_limits<L, JW>(W.cur, ru.lgn, ru.kind ? 0 : (int)A.k);
          if (pass) {
            if (ti < te && ru.req == W.req) limits(rl.lim, rl.elim, rl.ud, ru.small);
          } else if (lane == 0) {
            W.lim = rl.lim;
            W.elim = rl.elim;
            W.ud = rl.ud;
          }
        }
        __syncwarp();
      }
    }
    if (end) break;
    __syncwarp();
    const u32 idle = __ballot_sync(FULL, ti >= te);
    if ((int)__popc(idle) >= thr) {
      if (__any_sync(FULL, next < ents)) {
        // ---- the idle lanes take the run's next entries ----
        const StagedRun& cu = W.run[(ring - 1u) & (SLOTS - 1)];
        const u32 idx = next + __popc(idle & ((1u << lane) - 1u));
        const bool take = ti >= te && idx < ents;
        u32 cnt = 0;  // kind 1: the entry's seeds
        if (take) {
          slot = (ring - 1u) & (SLOTS - 1);
          ti = gaps + 4 * cu.ph;
          g = gap_at(ti);
          if (cu.kind == 0) {
            const uint4 e = W.stage[(ring - 1u) & 1u][idx];
            const u32 f = (e.y >> 8) & 0xFFu;
            pk = ((u32)(DA * (int)f - DB * (int)A.k) & 0xFFFFu) | ((e.y >> 24) << 16);
            const u64 p = S.p3[f], c = ((u64)e.w << 32) | e.z;
            {
              const u128 n = (((((u128)cu.q_hi << 64) | cu.q_lo) - g) << A.k) + (((ull)(e.y & 0xFFu) << 32) | e.x);
              W.base[lane] = make_uint4((u32)n, (u32)(n >> 32), (u32)(n >> 64), cu.req);
            }
            p4 = p << 2;
            // the value at block offset g is T^k of the first block's seed
            if (L == 2) {
              const u64 x = ((cu.q_lo - g) * p + c + (A.negative ? 1ull : ~0ull)) << 2;
              yb[0] = (u32)x;
              yb[1] = (u32)(x >> 32);
            } else {
              const u128 x =
                  (((((u128)cu.q_hi << 64) | cu.q_lo) - g) * p + c + (A.negative ? (u128)1 : ~(u128)0)) << 2;
#pragma unroll
              for (int i = 0; i < L; i++) yb[i] = (u32)(x >> (32 * i));
            }
            te = ti + 4 * cu.rows + 4;
          } else {  // an integer and every 576th after it: no residue sieve, no jump
            const ull n = cu.q_lo + idx;
            W.base[lane] = make_uint4((u32)n, (u32)(n >> 32), 0u, cu.req);
            pk = 0x80000000u;
            p4 = 4 * DENSE_STEP;
#pragma unroll
            for (int i = 0; i < L; i++) yb[i] = i == 0 ? (u32)(n << 2) : i == 1 ? (u32)(n >> 30) : 0u;
            cnt = (cu.rows - 1 - idx) / DENSE_STEP + 1;
            if (cu.mod9 && !(((A.negative ? KEEP9N : KEEP9) >> (u32)(n % 9u)) & 1u))
              cnt = (A.negative && n == 5) ? 1 : 0;
            te = ti + 4 * cnt + 4;
            if (n < 2 && cnt) {  // 0 and 1 are not run: the entry begins with its second seed
              ti += 4;
              g = gap_at(ti);
              cnt--;
            }
          }
          limits(W.lim, W.elim, W.ud, cu.small);
          take_next();
          if constexpr (STATS) xs[RS_ENTRIES]++;
        }
        cnt = __reduce_add_sync(FULL, cnt);
        if (lane == 0) W.acc_seeds += cnt;
        next += min(__popc(idle), ents - next);
        clocked(RS_CYCLES_ENTRIES);
      } else {
        // ---- the next run ----
        cp_async_wait_all();
        __syncwarp();
        const StagedRun& nx = W.run[ring & (SLOTS - 1)];
        if (__any_sync(FULL, nx.valid == 0)) {
          if (idle == FULL) {
            last = true;
            if (slow) continue;
            // the warps' last seeds for the exact path, together: 32 to a warp
            if (lane == 0) S.last[threadIdx.x >> 5] = ex;
            __syncthreads();
            u32 total = 0;
            uint4 e = make_uint4(0u, 0u, 0u, 0u);
            bool have = false;
#pragma unroll 1
            for (u32 i = 0; i < WARPS; i++) {
              const u32 c = S.last[i];
              if (!have && threadIdx.x - total < c) {
                e = S.w[i].exact[threadIdx.x - total];
                have = true;
              }
              total += c;
            }
            __syncthreads();
            W.exact[lane] = e;
            ex = __popc(__ballot_sync(FULL, have));
            end = true;
            clocked(RS_CYCLES_RUNS);
            continue;
          }
          thr = 32;  // no more runs: the lanes finish what they have
        } else if (__any_sync(FULL, ti < te && slot == ((ring + 1u) & (SLOTS - 1)))) {
          thr = 32;  // the slot that the run after the next will be staged in is still in use: wait for its lanes
        } else {
          ring++;
          next = 0;
          ents = __reduce_max_sync(FULL, nx.ents);  // (a reduction and a vote, so that they are known to be uniform)
          thr = (int)(__any_sync(FULL, nx.rows >= 64) ? A.rl : A.rs);
          ulonglong2 keys = W.keys;
          if (__any_sync(FULL, keys.x == 0 && nx.ents != 0 && nx.small == 0)) {
            const bool have = lane < nx.ents;
            u128 x;
            u32 D0 = 0;
            if (nx.kind == 0) {
              const uint4 e = W.stage[(ring - 1u) & 1u][lane];
              const u32 f = have ? (e.y >> 8) & 0xFFu : 0u;
              D0 = (u32)(DA * (int)f - DB * (int)A.k);
              x = (((u128)nx.q_hi << 64) | nx.q_lo) * S.p3[f] + (((u64)e.w << 32) | e.z) +
                  (A.negative ? (u128)1 : ~(u128)0);
            } else {
              x = nx.q_lo + lane;
            }
            u32 y4[4] = {(u32)(x << 2), (u32)(x >> 30), (u32)(x >> 62), (u32)(x >> 94)};
            const bool kept = nx.kind == 0 || !nx.mod9 || (((A.negative ? KEEP9N : KEEP9) >> (u32)((nx.q_lo + lane) % 9u)) & 1u);
            const ulonglong2 found = scout<L, JW>(S, A, y4, D0, nx.lgn, nx.kind ? 0 : (int)A.k, have && kept);
            ReqRec* r = A.recs + nx.req;
            if constexpr (STATS) xs[RS_SCOUTS] += lane == 0;
            if (lane == 0) {
              atomicMax(&r->st_key, found.x);
              atomicMax(&r->e_key, found.y);
            }
            __syncwarp();
            keys = make_ulonglong2(max(found.x, *(volatile ull*)&r->st_key), max(found.y, *(volatile ull*)&r->e_key));
          }
          const ulonglong2 cur = nx.req == W.req ? make_ulonglong2(max(W.cur.x, keys.x), max(W.cur.y, keys.y)) : keys;
          const RunLimits rl = run_limits<L, JW>(cur, nx.lgn, nx.kind ? 0 : (int)A.k);
          __syncwarp();
          if (lane == 0) {
            if (nx.req != W.req) {
              if (W.req != FULL) {
                if (W.acc_seeds) atomicAdd(&A.recs[W.req].seeds, W.acc_seeds);
                atomicAdd(&A.recs[W.req].items_done, W.acc_rows);
              }
              W.req = nx.req;
              W.acc_seeds = W.acc_rows = 0;
            }
            W.cur = cur;
            W.acc_rows += nx.items;
            if (nx.kind == 0) W.acc_seeds += (ull)nx.rows * nx.ents;
            W.lim = rl.lim;
            W.elim = rl.elim;
            W.ud = rl.ud;
          }
          __syncwarp();
          stage_next(S, W, ring, A, lane, nwarps, first);
        }
        clocked(RS_CYCLES_RUNS);
      }
      if ((int)__popc(__ballot_sync(FULL, ti >= te)) >= thr) continue;
    }
    // ---- windows, until a seed is at a limit or thr lanes are idle (looked at after every
    // fourth window) ----
    __syncwarp();
    while (!__any_sync(FULL, (int)P < 0)) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if constexpr (STATS) xs[RS_WINDOWS] += ti < te && (int)P >= 0;
        hot_step<L, JW>(y, yb, p4, g, P, Pn, ud, ti, S, cls, A.one, A.mone, A.eight);
      }
      if constexpr (STATS) xs[RS_PASSES] += lane == 0;
      ti = min(ti, te);  // (an idle lane stays within the table's margin)
      if ((int)__popc(__ballot_sync(FULL, ti >= te)) >= thr) break;
    }
    clocked(RS_CYCLES_WINDOWS);
    // ---- the seeds at a limit go to the exact path (rare) ----
    if (__any_sync(FULL, (int)P < 0)) {
      const bool bad = (int)P < 0 && ti < te;
      const u32 b = __ballot_sync(FULL, bad);
      if (bad) {
        const u32 dense = pk >> 31;
        W.slow[slow + __popc(b & ((1u << lane) - 1u))] =
            seed_at(W.base[lane], gap_at(ti - 4), dense ? 0u : A.k, dense ? DENSE_STEP : 1u);
        take_next();
      }
      slow += __popc(b);
      if (ti >= te) P = Pn = 0xC000u;  // an idle lane is at no limit
    }
  }
  if (lane == 0 && W.req != FULL) {
    if (W.acc_seeds) atomicAdd(&A.recs[W.req].seeds, W.acc_seeds);
    atomicAdd(&A.recs[W.req].items_done, W.acc_rows);
  }
  if (A.stats && lane == 0) atomicAdd(&A.stats[RS_RUNS], (ull)(ring + 1u));
  if constexpr (STATS) {
#pragma unroll
    for (int i = 0; i < RANGE_STATS; i++)
      if (xs[i] && (i < RS_CYCLES_WINDOWS || lane == 0)) atomicAdd(&A.stats[i], xs[i]);
  }
}

// ------------------------------------------------------------------
// After the range kernel: candidates and wide seeds.
// ------------------------------------------------------------------

enum : u32 { WIDE_OK, WIDE_LEFT, WIDE_CAP, WIDE_CYCLE };

// One seed with L limbs, from scratch: its stopping time and excursion.  WIDE_LEFT: a value
// could leave L limbs; WIDE_CAP: iter_cap run pairs; WIDE_CYCLE: back at the seed.
template <int L>
__device__ __noinline__ u32 wide_seed(const WidenEntry& e, bool neg, u32 iter_cap, ull& st, u32* E8) {
  Limbs<L> v, N, E;
#pragma unroll
  for (int j = 0; j < L; j++) N.w[j] = (j == 0) ? e.n0 : (j == 1) ? e.n1 : (j == 2) ? e.n2 : 0u;
  v = N;
  if (neg) dec_l<L>(v); else inc_l<L>(v);  // v = n + 1, or u = n - 1 for T'
  E = N;
  st = 0;
  for (u32 it = 1;; it++) {
    if (it > iter_cap) return WIDE_CAP;
    if (v.w[L - 1] >= (1u << 19)) return WIDE_LEFT;
    const u32 a = ctz32(v.w[0] | (1u << 8));
    u32 m = 1;
    for (u32 j = 0; j < a; j++) m *= 3u;
    odd_run_l<L>(v, a, m);
    st += a;
    Limbs<L> x = v;  // the value: v - 1, or u + 1 for T'
    if (neg) inc_l<L>(x); else dec_l<L>(x);
    if (limbs_lt<L>(E, x)) E = x;
    // even run on the value x
    const u32 b = ctz32(x.w[0] | 0x80000000u);
    Limbs<L> w = x;
    shr_l<L>(w, b);
    if (b != 0 && limbs_lt<L>(w, N)) {
      u32 s = 1;
      for (; s < b; s++) {
        Limbs<L> y = x;
        shr_l<L>(y, s);
        if (limbs_lt<L>(y, N)) break;
      }
      st += s;
#pragma unroll
      for (int j = 0; j < 8; j++) E8[j] = (j < L) ? E.w[j < L ? j : 0] : 0u;
      return WIDE_OK;
    }
    st += b;
    if (neg && !limbs_lt<L>(w, N) && !limbs_lt<L>(N, w)) return WIDE_CYCLE;
    v = w;
    if (neg) dec_l<L>(v); else inc_l<L>(v);
  }
}

__global__ void __launch_bounds__(128) k_range_finish(const __grid_constant__ RangeArgs A) {
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x, lane = lane_id();
  const u32 nc = min(A.head->cands, CAND_CAP), nw = min(A.head->widened, WIDEN_CAP);
  // candidates still at their record's keys: one lane at a time for a request (record locks), the
  // requests of a warp's lanes side by side.  A batch of small requests has two candidates for each:
  // 1000 requests of 64 to 256 seeds take 75 us, and took 129 with one lane at a time for all; 20 000 take
  // 0.22 ms and took 0.52 (with half the list's length as well).
  for (u32 i0 = t - lane; i0 < nc; i0 += nt) {
    bool live = i0 + lane < nc;
    RangeCand c{};
    if (live) {
      c = A.lists->cand[i0 + lane];
      const ReqRec* r = A.recs + c.req;
      live = c.kind == 0 ? c.st >= *(volatile const ull*)&r->st_key
                         : key_of<4>(c.E) >= *(volatile const ull*)&r->e_key;
    }
    while (__any_sync(FULL, live)) {
      const u32 same = __match_any_sync(FULL, live ? (ull)c.req : (1ull << 32) + lane);
      if (live && lane == (u32)__ffs(same) - 1) {
        if (c.kind == 0) rec_offer_st(A.recs + c.req, c.st, c.seed);
        else rec_offer_e<4>(A.recs + c.req, c.E, c.seed);
        live = false;
      }
      __syncwarp();
    }
  }
  // widened seeds, one per thread: 6 limbs, then 8
  for (u32 i0 = t - lane; i0 < nw; i0 += nt) {
    bool ok = false;
    WidenEntry e{0, 0, 0, 0};
    ull st = 0;
    u32 E[8];
    if (i0 + lane < nw) {
      e = A.lists->widen[i0 + lane];
      u32 how = wide_seed<6>(e, A.negative != 0, A.iter_cap, st, E);
      if (how == WIDE_LEFT) how = wide_seed<8>(e, A.negative != 0, A.iter_cap, st, E);
      ok = how == WIDE_OK;
      if (!ok) {
        if (how == WIDE_CAP) atomicOr(&A.recs[e.req].errors, ERR_ITER_CAP);
        atomicAdd(&A.recs[e.req].failures, 1ull);
      }
    }
    for (u32 m = __ballot_sync(FULL, ok); m; m &= m - 1) {
      if (lane == (u32)__ffs(m) - 1) {
        const u32 seed[4] = {e.n0, e.n1, e.n2, 0};
        rec_offer_st(A.recs + e.req, st, seed);
        rec_offer_e<8>(A.recs + e.req, E, seed);
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------
// Launchers.
// ------------------------------------------------------------------

int range_variants() { return RANGE_VARIANTS; }
int range64_variants() { return RANGE_VARIANTS; }
uint32_t range64_max_seed_bits() { return 48; }

// FNV-1a of the variant table's parameters: part of the autotuner's cache key, so that a
// choice cached for another table is not applied to this one.
uint32_t range_variant_rev() {
  u32 h = 2166136261u;
  for (const RangeVariant& v : RANGE_VARIANT)
    for (u32 x : {v.jw, v.rl, v.rs, v.warps}) h = (h ^ x) * 16777619u;
  return h;
}

// The bodies that the variants use (range_variants.h): window length and warps per block.
#define CZ_RANGE_BODIES(X) X(13, 32) X(13, 24) X(12, 32) X(12, 24)
#define X(j, w) static_assert(sizeof(RangeShared<j, w>) <= MAX_BLOCK_SMEM, "shared memory of a block");
CZ_RANGE_BODIES(X)
#undef X

template <int L>
static cudaError_t launch_t(const RangeArgs& a, u32 jw, u32 warps, u32 grid, cudaStream_t st) {
  if (a.stats) {  // diagnostics: the long launches' body
    k_range<L, 13, 32, true><<<grid, 32 * 32, sizeof(RangeShared<13, 32>), st>>>(a);
    return cudaGetLastError();
  }
#define X(j, w)                                                                                    \
  if (jw == j && warps == w) {                                                                     \
    k_range<L, j, w, false><<<grid, w * 32, sizeof(RangeShared<j, w>), st>>>(a);                   \
    return cudaGetLastError();                                                                     \
  }
  CZ_RANGE_BODIES(X)
#undef X
  return cudaErrorInvalidValue;
}

cudaError_t launch_range(const RangeArgs& args, int words, int variant, u32 sm_count, cudaStream_t st) {
  if (variant < 0 || variant >= RANGE_VARIANTS) return cudaErrorInvalidValue;
  const RangeVariant v = range_pick(variant, args.item_limit, sm_count);
  RangeArgs a = args;
  a.rl = v.rl;
  a.rs = v.rs;
  const u32 grid = (u32)std::max<unsigned long long>(1, std::min<unsigned long long>(sm_count, a.item_limit));
  switch (words) {
    case 2: return launch_t<2>(a, v.jw, v.warps, grid, st);
    case 3: return launch_t<3>(a, v.jw, v.warps, grid, st);
    case 4: return launch_t<4>(a, v.jw, v.warps, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int L>
static cudaError_t init_t() {
  cudaError_t e = cudaSuccess;
#define X(j, w)                                                                                               \
  if (e == cudaSuccess)                                                                                       \
    e = cudaFuncSetAttribute(k_range<L, j, w, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,            \
                             (int)sizeof(RangeShared<j, w>));
  CZ_RANGE_BODIES(X)
#undef X
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_range<L, 13, 32, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(RangeShared<13, 32>));
  return e;
}

// Opts every range kernel into its dynamic shared memory and fills the window tables if the device
// has not got them yet.
cudaError_t range_init(cudaStream_t st) {
  cudaError_t e = init_t<2>();
  if (e == cudaSuccess) e = init_t<3>();
  if (e == cudaSuccess) e = init_t<4>();
  if (e != cudaSuccess) return e;
  return fill_once([&](bool* done) { return table_ready(g_win_ready, done, st); },
                   [&] {
                     k_win_tables<<<(1u << MAX_JW) / 256, 256, 0, st>>>();
                     const cudaError_t l = cudaGetLastError();
                     return l ? l : cudaStreamSynchronize(st);
                   },
                   [&] { return mark_table(g_win_ready, st); });
}

cudaError_t launch_range_finish(const RangeArgs& a, cudaStream_t st) {
  k_range_finish<<<64, 128, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace cz
