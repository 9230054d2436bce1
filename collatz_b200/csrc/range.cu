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
//     32 900 (the nearest 2^i / 3^F above 1 is 2^401 / 3^253 = 1.0031).  For the
//     negative variant rho_i is subtracted: C_i < 1 gives T'^i(m) < m at once, and
//     C_i > 1 keeps T'^i(m) above m when m > F_i / (3 (1 - 1/C_i)), below 48 900
//     (3^53 / 2^84 = 1.0021).  Seeds of at least 2^16 satisfy both.
//   * T^i(n) <= C_i (n + F_i / 3), so D_i / 306 + log2(n) bounds log2 T^i(n) from
//     above to within 0.0023.
// A seed whose D is negative after a window has therefore fallen below its
// start within it.  Its stopping time is at most the steps taken and its
// excursion at most what D allowed; both are below the request's running maxima
// (the windows' limits see to that), so it can change no output and is done.
//
// The exact path.  A seed that might change an output -- D or the step count
// reaches its limit, a value could leave the words it is kept in, a seed
// below 2^16 -- is run again from its start, one run pair at a time with four limbs,
// the exact stopping time and excursion, 32 such seeds to a warp (exact_seeds).
// A value that could leave 2^128 sends the seed to the widen list, re-run with
// 6 and then 8 limbs.  Before the kernel, scouts run some of each request's
// seeds in full to give its maxima, and so the limits, a head start.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"
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
constexpr u32 RUN_MAX = 1024;             // rows of a run (10 bits of a queued seed)
constexpr u32 MIDQ = 64, SLOWQ = 64;      // queue entries per warp (31 left over + 32 new at most)
constexpr u32 SLOTS = 32;                 // runs whose seeds may be queued at a time

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

// Window tables, one per length and sign.  Entry r: T^JW(r) << 11 | m << 7 | f << 3, with f the
// odd steps and m = floor(-min D_i / 128) of the window's D_i (at most 15; 0 when none is
// negative): a seed with D < 128 m at the window's start falls below its start inside it.
constexpr u32 MIN_JW = 11, MAX_JW = 13;  // T^13(r) < 3^13 < 2^21
constexpr u32 WIN_M = 0x780u, WIN_F = 0x78u;
__device__ u32 g_win[2][MAX_JW - MIN_JW + 1][1u << MAX_JW];

__global__ void k_win_tables() {
  const u32 t = blockIdx.x * blockDim.x + threadIdx.x;
  for (u32 neg = 0; neg < 2; neg++)
    for (u32 jw = MIN_JW; jw <= MAX_JW; jw++) {
      if (t >> jw) continue;
      u32 x = t, f = 0;
      int D = 0, m = 0;
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
      }
      g_win[neg][jw - MIN_JW][t] = (x << 11) | (min((u32)(-m) >> 7, 15u) << 7) | (f << 3);
    }
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Queue a seed for the 192/256-bit re-run.
__device__ __forceinline__ void widen_seed(const RangeArgs& A, u32 req, u32 n0, u32 n1, u32 n2) {
  const u32 wi = atomicAdd(A.widen_count, 1u);
  if (wi < A.widen_cap) {
    A.widen[wi] = WidenEntry{req, n0, n1, n2};
    atomicAdd(&A.recs[req].widened, 1ull);
  } else {
    atomicOr(&A.recs[req].errors, ERR_WIDEN_FULL);
    atomicAdd(&A.recs[req].failures, 1ull);
  }
}

// ------------------------------------------------------------------
// The exact path: up to 32 seeds, one per lane, from their starts.
// ------------------------------------------------------------------
struct ExactSeed {
  u32 st;      // stopping time
  u128 E;      // excursion
  bool ok;     // fell below its start
  bool widen;  // a value reached 2^119
  bool cycle;  // negative variant: came back to its start
  bool cap;    // ST_CAP steps
};

// Runs the seeds of all lanes together (lanes with have = false idle): odd runs
// of at most 7 steps and even runs of at most 31, on 64-bit values in the steps
// in which every lane's value is below 2^59 (an odd run then stays below 2^64),
// else on 128 bits.  Warp-uniform.
__device__ __forceinline__ ExactSeed exact_run(u128 n, bool have, bool neg) {
  ExactSeed R;
  R.st = 0;
  R.ok = R.widen = R.cycle = R.cap = false;
  const u64 n0 = (u64)n, n1 = (u64)(n >> 64);
  u64 E0 = n0, E1 = n1;
  const u64 one = neg ? 1ull : ~0ull;  // from a run state to the value it stands for
  u64 v0 = n0 - one, v1 = n1 + (neg ? (n0 == 0 ? ~0ull : 0ull) : (v0 == 0 ? 1ull : 0ull));
  bool alive = have;
  while (__any_sync(FULL, alive)) {
    if (__all_sync(FULL, !alive || (v1 | (v0 >> 59)) == 0)) {
      // below 2^59 for every lane; a seed of 2^64 or more would have descended
      const u32 a = ctz32((u32)v0 | 0x80u);
      const u64 x = (v0 >> a) * pow3_le7(a) + one;
      const u32 b = ctz32((u32)x | 0x80000000u);
      const u64 w = x >> b;
      const bool fell = alive & (b != 0) & ((w < n0) | (n1 != 0));
      if (alive & (E1 == 0) & (x > E0)) E0 = x;
      if (alive) R.st += fell ? a : a + b;
      if (fell) {
        u32 s = 1;
        while ((x >> s) >= n0 && n1 == 0) s++;  // ends at b
        R.st += s;
        R.ok = true;
        alive = false;
      }
      if (neg && alive && w == n0 && n1 == 0) {
        R.cycle = true;
        alive = false;
      }
      v0 = alive ? w - one : v0;
    } else if (alive) {
      u128 v = ((u128)v1 << 64) | v0;
      const u32 a = ctz32((u32)v | 0x80u);
      v = (v >> a) * pow3_le7(a);
      if ((u32)(v >> 96) >= OVF3) {
        R.widen = true;
        alive = false;
      } else {
        const u128 x = neg ? v + 1 : v - 1;
        if (x > (((u128)E1 << 64) | E0)) {
          E0 = (u64)x;
          E1 = (u64)(x >> 64);
        }
        const u32 b = ctz32((u32)x | 0x80000000u);
        const u128 w = x >> b;
        if (b != 0 && w < n) {
          u32 s = 1;
          while ((x >> s) >= n) s++;
          R.st += a + s;
          R.ok = true;
          alive = false;
        } else if (neg && w == n) {
          R.cycle = true;
          alive = false;
        } else {
          R.st += a + b;
          v = neg ? w - 1 : w + 1;
          v0 = (u64)v;
          v1 = (u64)(v >> 64);
        }
      }
    }
    if (alive && R.st > ST_CAP) {
      R.cap = true;
      alive = false;
    }
  }
  R.E = ((u128)E1 << 64) | E0;
  return R;
}

// The exact path for the warp's queued seeds e (n limbs 0..2, request), one per
// lane with have: failures, widening and errors are recorded, and of the seeds of
// one request that may raise a maximum only the best is offered (larger, or equal
// with a smaller seed).  Out of line: its registers stay out of the window loop.
static __device__ __noinline__ void exact_seeds(const RangeArgs& A, uint4 e, bool have) {
  const u32 lane = lane_id();
  const u128 n = ((u128)e.z << 64) | ((u64)e.y << 32) | e.x;
  const ExactSeed R = exact_run(n, have, A.negative != 0);
  ReqRec* rec = A.recs + e.w;
  bool ps = false, pe = false;
  u32 E[4];
#pragma unroll
  for (int i = 0; i < 4; i++) E[i] = (u32)(R.E >> (32 * i));
  if (have) {
    if (R.ok) {
      ps = R.st >= *(volatile ull*)&rec->st_key;
      pe = key_of<4>(E) >= *(volatile ull*)&rec->e_key;
    } else if (R.widen) {
      widen_seed(A, e.w, e.x, e.y, e.z);
    } else {
      if (R.cap) atomicOr(&rec->errors, ERR_ITER_CAP);
      atomicAdd(&rec->failures, 1ull);
    }
  }
  u32 pm = __ballot_sync(FULL, ps | pe);
  while (pm) {
    const u32 req = __shfl_sync(FULL, e.w, __ffs(pm) - 1);
    const bool in = (ps | pe) & (e.w == req);
    const u32 sm = __reduce_max_sync(FULL, (in & ps) ? R.st + 1 : 0u);  // 0: nobody
    u32 cs = __ballot_sync(FULL, in & ps & (R.st + 1 == sm));
    u32 ce = __ballot_sync(FULL, in & pe);
#pragma unroll
    for (int i = 3; i >= 0; i--) {  // the lanes with the largest excursion
      const u32 m = __reduce_max_sync(FULL, ((ce >> lane) & 1u) ? E[i] : 0u);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && E[i] == m);
    }
    const u32 nl[3] = {e.x, e.y, e.z};
#pragma unroll
    for (int i = 2; i >= 0; i--) {  // the smallest seed of each
      const u32 a = __reduce_min_sync(FULL, ((cs >> lane) & 1u) ? nl[i] : FULL);
      cs = __ballot_sync(FULL, ((cs >> lane) & 1u) && nl[i] == a);
      const u32 b = __reduce_min_sync(FULL, ((ce >> lane) & 1u) ? nl[i] : FULL);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && nl[i] == b);
    }
    const u32 seed[4] = {e.x, e.y, e.z, 0};
    if (cs && lane == (u32)__ffs(cs) - 1) rec_offer_st(rec, R.st, seed);
    __syncwarp();
    if (ce && lane == (u32)__ffs(ce) - 1) rec_offer_e<4>(rec, E, seed);
    __syncwarp();
    pm &= ~__ballot_sync(FULL, in);
  }
}

// ------------------------------------------------------------------
// The range kernel.
// ------------------------------------------------------------------

// A run of rows staged for a warp (warp-uniform): rows of one chunk of 64 entries
// over blocks q, q + qs, ..., or (kind 1) rows of 64 consecutive integers.
struct StagedRun {
  ull q_lo;          // kind 0: first block (low 64 bits); kind 1: first integer
  ull d_hi;          // kind 1: end (exclusive)
  u32 q_hi;          // kind 0: first block, bits 64..95
  u32 sbase, send;   // kind 0: survivor-table range
  u32 req, kind, qs, mod9, rows, valid, pad;
};

// What a queued seed's run was, to find the seed again.
struct RunSlot {
  ull q_lo;
  u32 q_hi, qs, sbase, req, kind, pad;
};

// Per-warp state in shared memory.  A queued seed: its value y = 4 T^s(n) in L
// words, P = (limit - D) << 16 | D, and meta: [5:0] entry, [10:6] slot, [20:11] row of
// the run, [31:26] windows it may still take after the next one (signed).
template <int L>
struct RangeWarp {
  uint4 mid[MIDQ];                  // L = 2: y0 y1 P meta; L = 3: y0..y2 P; L = 4: y0..y3
  u32 mid2[L == 2 ? 4 : L == 3 ? MIDQ : 2 * MIDQ];  // L = 3: meta; L = 4: P, meta
  uint4 slow[SLOWQ];                // seeds for the exact path: n limbs 0..2, request
  RunSlot slot[SLOTS];
  uint4 stage[RANGE_ITEM];          // survivor entries of the staged run (cp.async)
  ulonglong2 keys;                  // st_key, e_key of its request (cp.async)
  ulonglong2 cur;                   // the current request's keys, as last read
  RangeSeg seg;                     // cached segment
  StagedRun run[2];                 // the current run and the staged one, in turn
  ull pos, claim_hi, seg_lo, seg_hi;
  ull acc_seeds, acc_rows;          // of the current request, not yet added to its record
  u32 req;                          // the current request
  u32 pad;
};

// Shared memory of a block: window table, powers of 3, then the warps' state.
template <int L, int JW, int WARPS>
struct RangeShared {
  u32 win[1u << JW];
  uint2 cls[16];   // per f: 4 3^f, the window's change of P
  u32 last[WARPS]; // seeds each warp has left for the exact path at its end
  ull p3[42];      // 3^f
  RangeWarp<L> w[WARPS];
};

extern __shared__ __align__(16) unsigned char range_smem[];

template <int L, int JW, int WARPS>
__device__ __forceinline__ RangeShared<L, JW, WARPS>& range_shared() {
  return *reinterpret_cast<RangeShared<L, JW, WARPS>*>(range_smem);
}

// Advances to the next run (claiming rows as needed) and starts copying its
// survivor entries and its request's keys, so that they arrive while the current
// run is worked on.  Warp-uniform.  Claims are RUN_MAX rows while a warp has
// many more ahead and shrink towards the end of the launch, so that the warps
// finish together.
template <class WT>
__device__ __forceinline__ void stage_next(WT& W, StagedRun& nxt, const RangeArgs& A, u32 lane, u32 nwarps) {
  ull pos = W.pos;
  ull claim_hi = W.claim_hi;
  if (pos >= claim_hi) {
    const ull left = A.item_limit > claim_hi ? A.item_limit - claim_hi : 0;
    const u32 claim = (u32)min((ull)RUN_MAX, max(1ull, left / (4ull * nwarps)));
    ull c = 0;
    if (lane == 0) c = atomicAdd(A.item_cursor, (ull)claim);
    c = __shfl_sync(FULL, c, 0);
    if (c >= A.item_limit) {
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
  if (pos < W.seg_lo || pos >= W.seg_hi) {
    u32 lo = 0, hi = A.nsegs;  // the last segment beginning at or before pos
    while (hi - lo > 1) {
      const u32 mid = (lo + hi) >> 1;
      if (A.segs[mid].item_begin <= pos) lo = mid; else hi = mid;
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
  u32 rows = (u32)min((ull)RUN_MAX, min(claim_hi, W.seg_hi) - pos);
  StagedRun it;
  it.req = W.seg.req;
  it.kind = W.seg.kind;
  it.mod9 = W.seg.mod9;
  it.valid = 1;
  it.pad = 0;
  if (it.kind == 0) {  // segments hold fewer than 2^32 rows
    const u32 l32 = (u32)local, nq = W.seg.nq;
    const u32 chunk = l32 / nq, qi = l32 - chunk * nq;
    rows = min(rows, nq - qi);
    it.qs = W.seg.qstride ? W.seg.qstride : 1u;
    const u128 q = (((u128)W.seg.q_hi << 64) | W.seg.q_lo) + (u128)qi * it.qs;
    it.q_lo = (u64)q;
    it.q_hi = (u32)(q >> 64);
    it.sbase = W.seg.s_lo + chunk * RANGE_ITEM;
    it.send = min(it.sbase + RANGE_ITEM, W.seg.s_hi);
    it.d_hi = 0;
    const uint4* T = reinterpret_cast<const uint4*>(A.table);
#pragma unroll
    for (u32 j = 0; j < RANGE_ITEM / 32; j++) {
      const u32 idx = it.sbase + j * 32 + lane;
      if (idx < it.send) cp_async16(&W.stage[j * 32 + lane], T + idx);
    }
  } else {
    it.q_lo = W.seg.q_lo + local * DENSE_ITEM;
    it.q_hi = 0;
    it.sbase = it.send = 0;
    it.d_hi = W.seg.d_hi;
    it.qs = 0;
  }
  if (lane == 0) cp_async16(&W.keys, &A.recs[it.req].st_key);
  cp_async_commit();
  it.rows = rows;
  __syncwarp();
  if (lane == 0) {
    W.pos = pos + rows;
    nxt = it;
  }
  __syncwarp();
}

// The limits of a request's windows for the seeds of one run, from its keys.
struct RunLimits {
  int lim;   // a seed may take a window while D <= lim (0 < D); below 0: none
  int elim;  // 306 log2 of the least excursion that counts, over the run's largest seed
  int wmax;  // windows a seed may take
};

template <int L, int JW>
__device__ __forceinline__ RunLimits run_limits(ulonglong2 keys, float lgn, int s0) {
  const ull sk = keys.x, ek = keys.y;
  RunLimits R;
  // log2 of the excursion key's value (rounded down); the margins cover the float
  // arithmetic and the 0.0023 of the bound on T^i(n)
  const float lge = ek ? (float)((int)(ek >> 54) - 54) + __log2f(__ull2float_rd(ek & ((1ull << 54) - 1))) : -1.0f;
  R.elim = (int)floorf((float)DB * (lge - lgn)) - 2;
  const int lo = (int)floorf((float)DB * ((float)(32 * L - 2) - lgn)) - 2;  // values stay in L words
  R.lim = min(min(R.elim, lo), LIM_MAX) - window_slack(JW) - 1;
  const int thr = (int)min(sk, 485ull);  // D decides only below 485 steps
  R.wmax = thr - 1 >= s0 ? min((thr - 1 - s0) / JW, 31) : 0;
  return R;
}

// One window of a value y = 4 x of L words (bits 0 and 1 are arbitrary): z = 4 T^JW(x),
// Pz = P with D's change (z may be y, and Pz P).  Returns a word with bit 15 set when the seed fell below its
// start inside the window.
template <int L, int JW>
__device__ __forceinline__ u32 window(const u32* y, u32 P, u32* z, u32& Pz, const u32* s_win, const uint2* s_cls) {
  const u32 e = *reinterpret_cast<const u32*>(reinterpret_cast<const char*>(s_win) + (y[0] & (((1u << JW) - 1u) << 2)));
  const u32 low = P - (e & WIN_M);
  const uint2 c = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(s_cls) + (e & WIN_F));
  u64 t = e >> 9;  // 4 T^JW(r), and two bits of m
#pragma unroll
  for (int i = 0; i < L; i++) {
    const u32 a = (i + 1 < L) ? __funnelshift_r(y[i], y[i + 1 < L ? i + 1 : i], JW + 2) : (y[i] >> (JW + 2));
    if (i + 1 < L) {
      t += (u64)a * c.x;
      z[i] = (u32)t;
      t >>= 32;
    } else {
      z[i] = a * c.x + (u32)t;
    }
  }
  Pz = P + c.y;
  return Pz | low;
}

template <int L>
__device__ __forceinline__ void mid_store(RangeWarp<L>& W, u32 at, const u32* y, u32 P, u32 meta) {
  if (L == 2) {
    W.mid[at] = make_uint4(y[0], y[1], P, meta);
  } else if (L == 3) {
    W.mid[at] = make_uint4(y[0], y[1], y[L > 2 ? 2 : 0], P);
    W.mid2[at] = meta;
  } else {
    W.mid[at] = make_uint4(y[0], y[1], y[L > 2 ? 2 : 0], y[L > 3 ? 3 : 0]);
    reinterpret_cast<uint2*>(W.mid2)[at] = make_uint2(P, meta);
  }
}

template <int L>
__device__ __forceinline__ void mid_load(const RangeWarp<L>& W, u32 at, u32* y, u32& P, u32& meta) {
  const uint4 e = W.mid[at];
  y[0] = e.x;
  y[1] = e.y;
  if (L == 2) {
    P = e.z;
    meta = e.w;
  } else if (L == 3) {
    y[L > 2 ? 2 : 0] = e.z;
    P = e.w;
    meta = W.mid2[at];
  } else {
    y[L > 2 ? 2 : 0] = e.z;
    y[L > 3 ? 3 : 0] = e.w;
    const uint2 m = reinterpret_cast<const uint2*>(W.mid2)[at];
    P = m.x;
    meta = m.y;
  }
}

// The seed n of a queued entry, for the exact path.
template <int L>
__device__ __forceinline__ uint4 seed_of(const RangeWarp<L>& W, const RangeArgs& A, u32 meta) {
  const RunSlot s = W.slot[(meta >> 6) & 31u];
  const u32 row = (meta >> 11) & 1023u, idx = meta & 63u;
  if (s.kind) {
    const ull n = s.q_lo + (ull)row * DENSE_ITEM + idx;
    return make_uint4((u32)n, (u32)(n >> 32), 0u, s.req);
  }
  const RangeEntry e = A.table[s.sbase + idx];
  const u128 q = (((u128)s.q_hi << 64) | s.q_lo) + (u128)row * s.qs;
  const u128 n = (q << A.k) | ((u64)(e.meta & 0xFFu) << 32) | e.r_lo;
  return make_uint4((u32)n, (u32)(n >> 32), (u32)(n >> 64), s.req);
}

// Queued seeds of a warp (warp-uniform).
struct Queues {
  u32 mid, slow;
};

// Lanes with p: their queued seed (meta) goes to the slow queue.
template <int L>
__device__ __forceinline__ void push_slow(RangeWarp<L>& W, const RangeArgs& A, u32& slow, bool p, u32 meta) {
  const u32 b = __ballot_sync(FULL, p);
  if (p) W.slow[slow + __popc(b & lanemask_lt())] = seed_of<L>(W, A, meta);
  slow += __popc(b);
}

// One window for the last min(mid, 32) queued seeds.
template <int L, int JW, bool PART>
__device__ __forceinline__ void step_mid(RangeWarp<L>& W, const RangeArgs& A, u32 lane, Queues& Q, const u32* s_win,
                                         const uint2* s_cls) {
  const u32 cnt = PART ? min(Q.mid, 32u) : 32u;
  __syncwarp();
  u32 y[L], z[L], P, meta;
  Q.mid -= cnt;
  mid_load<L>(W, Q.mid + lane, y, P, meta);  // past the end (lane >= cnt): inside the queue's array
  if (PART && lane >= cnt) {                 // an idle lane: done at once
    P = 0xC000u;
    meta = 0;
  }
  const bool bad = (int)(P | meta) < 0;
  if (__any_sync(FULL, bad)) {
    push_slow<L>(W, A, Q.slow, bad, meta);
    P = bad ? 0xC000u : P;
  }
  const bool keep = !(window<L, JW>(y, P, z, P, s_win, s_cls) & 0x8000u);
  const u32 b = __ballot_sync(FULL, keep);
  if (keep) mid_store<L>(W, Q.mid + __popc(b & ((1u << lane) - 1u)), z, P, meta - (1u << 26));
  Q.mid += __popc(b);
}

// Works off the queues: until both hold fewer than 32 seeds, or (all) the window
// queue is empty.  After seeds took the exact path the current
// request's keys are read again.  Out of line: the row loop calls it rarely.
template <int L, int JW, int WARPS>
__device__ __noinline__ Queues drain(const RangeArgs& A, Queues Q, bool all) {
  RangeShared<L, JW, WARPS>& S = range_shared<L, JW, WARPS>();
  RangeWarp<L>& W = S.w[threadIdx.x >> 5];
  const u32 lane = lane_id();
  for (;;) {
    if (Q.slow >= 32u) {
      __syncwarp();
      Q.slow -= 32u;
      exact_seeds(A, W.slow[Q.slow + lane], true);
      if (A.stats && lane == 0) atomicAdd(&A.stats[1], 32ull);
      const ReqRec* r = A.recs + W.req;
      const ull sk = *(volatile const ull*)&r->st_key, ek = *(volatile const ull*)&r->e_key;
      __syncwarp();
      if (lane == 0) {
        W.cur.x = max(W.cur.x, sk);
        W.cur.y = max(W.cur.y, ek);
      }
      __syncwarp();
    } else if (Q.mid >= (all ? 1u : 32u)) {
      step_mid<L, JW, true>(W, A, lane, Q, S.win, S.cls);
    } else {
      break;
    }
  }
  return Q;
}

// drain, for a converged warp.
template <int L, int JW, int WARPS>
__device__ __forceinline__ void drain_warp(const RangeArgs& A, u32 lane, Queues& Q, bool all) {
  const Queues R = drain<L, JW, WARPS>(A, Q, all);
  Q.mid = __popc(__ballot_sync(FULL, lane < R.mid));  // (both below 32; a vote, so that they are known to be uniform)
  Q.slow = __popc(__ballot_sync(FULL, lane < R.slow));
}

// Full windows while the window queue holds a warp's worth; when seeds for the exact
// path have piled up as well, drain runs them.  Returns whether it did (the
// request's keys may then have risen).
template <int L, int JW, int WARPS>
__device__ __forceinline__ bool work_off(RangeWarp<L>& W, const RangeArgs& A, u32 lane, Queues& Q, const u32* s_win,
                                         const uint2* s_cls) {
  while (Q.mid >= 32u && Q.slow < 32u) step_mid<L, JW, false>(W, A, lane, Q, s_win, s_cls);
  if (Q.slow < 32u) return false;
  drain_warp<L, JW, WARPS>(A, lane, Q, false);
  return true;
}

template <int L>
__device__ __forceinline__ void add_step(u32* y, u64 step) {
  const u64 c = (((u64)y[1] << 32) | y[0]) + step;
  if (L > 2) {
    const u64 h = ((L > 3 ? ((u64)y[L > 3 ? 3 : 0] << 32) : 0ull) | y[L > 2 ? 2 : 0]) + (c < step ? 1u : 0u);
    y[L > 2 ? 2 : 0] = (u32)h;
    if (L > 3) y[L > 3 ? 3 : 0] = (u32)(h >> 32);
  }
  y[0] = (u32)c;
  y[1] = (u32)(c >> 32);
}

// After a window: a lane whose seed is done (bit 15 of tst) takes its next one over the
// window's outcome in y, P and rem.  Predicated moves and adds, without a branch.
template <int L>
__device__ __forceinline__ void next_if_done(u32 tst, u32* y, u32* yn, u64 step, u32& P, u32 Pn, int& rem, int rem0,
                                             int& left) {
  const u32 done = tst & 0x8000u, s0 = (u32)step, s1 = (u32)(step >> 32);
  asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q mov.b32 %0, %6;\n\t"
      "@q mov.b32 %1, %7;\n\t"
      "@q mov.b32 %2, %8;\n\t"
      "@q mov.b32 %3, %9;\n\t"
      "@q sub.s32 %4, %4, 1;\n\t}"
      : "+r"(y[0]), "+r"(y[1]), "+r"(P), "+r"(rem), "+r"(left)
      : "r"(done), "r"(yn[0]), "r"(yn[1]), "r"(Pn), "r"(rem0));
  if constexpr (L == 2) {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %4, 0;\n\t"
        "@q add.cc.u32 %0, %0, %2;\n\t"
        "@q addc.u32 %1, %1, %3;\n\t}"
        : "+r"(yn[0]), "+r"(yn[1])
        : "r"(s0), "r"(s1), "r"(done));
  } else if constexpr (L == 3) {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %6, 0;\n\t"
        "@q mov.b32 %3, %2;\n\t"
        "@q add.cc.u32 %0, %0, %4;\n\t"
        "@q addc.cc.u32 %1, %1, %5;\n\t"
        "@q addc.u32 %2, %2, 0;\n\t}"
        : "+r"(yn[0]), "+r"(yn[1]), "+r"(yn[L > 2 ? 2 : 0]), "+r"(y[L > 2 ? 2 : 0])
        : "r"(s0), "r"(s1), "r"(done));
  } else {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %8, 0;\n\t"
        "@q mov.b32 %4, %2;\n\t"
        "@q mov.b32 %5, %3;\n\t"
        "@q add.cc.u32 %0, %0, %6;\n\t"
        "@q addc.cc.u32 %1, %1, %7;\n\t"
        "@q addc.cc.u32 %2, %2, 0;\n\t"
        "@q addc.u32 %3, %3, 0;\n\t}"
        : "+r"(yn[0]), "+r"(yn[1]), "+r"(yn[L > 2 ? 2 : 0]), "+r"(yn[L > 3 ? 3 : 0]), "+r"(y[L > 2 ? 2 : 0]),
          "+r"(y[L > 3 ? 3 : 0])
        : "r"(s0), "r"(s1), "r"(done));
  }
}

// The kernel.  What bounds it: integer issue (54 warp instructions per window of 32 lanes, 1.81
// windows per seed; ALU pipe 73 % busy, shared-memory data pipe 50 %).  Against run pairs of
// two table-free steps each in their lanes (17.0 warp instructions per seed, 43.5 ms for
// 2^38 seeds at 2^40 with k = 24) it takes 4.3 instructions per seed and 8.9 ms; 2^40 seeds at 2^60
// with k = 34 went from 128.8 to 32.8 ms.  Lanes step through their own entry's blocks without
// exchanging seeds; queueing every window's survivors instead (compacted, so that
// lanes stay full) took 10.6 ms, bound by the shared-memory pipe at 16 bytes a seed and way.
// L: words of a value; JW: window length; STOP: a half-run leaves its lanes once this many
// have no seed left; WARPS per block, one block per SM.
template <int L, int JW, int STOP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) k_range(const __grid_constant__ RangeArgs A) {
  RangeShared<L, JW, WARPS>& S = range_shared<L, JW, WARPS>();
  {
    const uint4* src = reinterpret_cast<const uint4*>(g_win[A.negative ? 1 : 0][JW - MIN_JW]);
    for (u32 i = threadIdx.x; i < (1u << JW) / 4; i += WARPS * 32) cp_async16(reinterpret_cast<uint4*>(S.win) + i, src + i);
    cp_async_commit();
  }
  if (threadIdx.x < 42) {
    ull p = 1;
    for (u32 i = 0; i < threadIdx.x; i++) p *= 3;
    S.p3[threadIdx.x] = p;
    if (threadIdx.x < 16)
      S.cls[threadIdx.x] = make_uint2(4u * (u32)p, (u32)(-(DA * (int)threadIdx.x - DB * JW) * 65535));
  }
  const u32 lane = lane_id();
  RangeWarp<L>& W = S.w[threadIdx.x >> 5];
  const u32 nwarps = gridDim.x * WARPS;
  if (lane == 0) {
    W.pos = W.claim_hi = 0;
    W.seg_lo = 1;
    W.seg_hi = 0;
    W.acc_seeds = W.acc_rows = 0;
    W.req = FULL;
  }
  __syncwarp();
  stage_next(W, W.run[0], A, lane, nwarps);
  cp_async_wait_all();
  __syncthreads();

  const u32* s_win = S.win;
  const uint2* s_cls = S.cls;
  Queues Q{0, 0};
  u32 ring = 0;  // runs begun
  for (;;) {
    cp_async_wait_all();
    __syncwarp();
    const StagedRun& it = W.run[ring & 1u];
    if (__any_sync(FULL, it.valid == 0)) break;  // (votes: the compiler then knows these branches are uniform)
    const u32 slot = ring & (SLOTS - 1);
    if (ring && slot == 0) drain_warp<L, JW, WARPS>(A, lane, Q, true);  // no seed of an older run stays queued
    ring++;
    if (lane == 0) {
      const ulonglong2 keys = W.keys;
      if (it.req != W.req) {
        if (W.req != FULL) {
          if (W.acc_seeds) atomicAdd(&A.recs[W.req].seeds, W.acc_seeds);
          atomicAdd(&A.recs[W.req].items_done, W.acc_rows);
        }
        W.req = it.req;
        W.cur = keys;
        W.acc_seeds = W.acc_rows = 0;
      } else {
        W.cur = make_ulonglong2(max(W.cur.x, keys.x), max(W.cur.y, keys.y));
      }
      W.acc_rows += it.rows;
      if (it.kind == 0) W.acc_seeds += (ull)it.rows * (it.send - it.sbase);
      W.slot[slot] = RunSlot{it.q_lo, it.q_hi, it.qs, it.sbase, it.req, it.kind, 0u};
    }
    __syncwarp();
    if (__any_sync(FULL, it.kind == 0)) {
      // log2 of the run's largest seed, from above
      const u128 ql = (((u128)it.q_hi << 64) | it.q_lo) + (u128)(it.rows - 1) * it.qs + 1;
      const float lgn = (float)A.k + 1e-5f + __log2f(__fmaf_ru(__uint2float_ru((u32)(ql >> 64)), 18446744073709551616.0f,
                                                               __ull2float_ru((u64)ql)));
#pragma unroll 1
      for (u32 j = 0; j < RANGE_ITEM / 32; j++) {
        const u32 ents = it.send - it.sbase;
        if (__any_sync(FULL, j * 32 >= ents)) break;
        const bool valid = j * 32 + lane < ents;
        const uint4 e = W.stage[j * 32 + lane];
        if (__any_sync(FULL, j * 32 + 32 >= ents)) {  // the last entries of the run are read: the next run's may come
          __syncwarp();
          stage_next(W, W.run[ring & 1u], A, lane, nwarps);
        }
        // the lane's seed in the first row, and the step from row to row
        const u32 f = valid ? (e.y >> 8) & 0xFFu : 0u;
        const int emx = DB * (int)(e.y >> 24), D0 = DA * (int)f - DB * (int)A.k;
        const u64 p = S.p3[f], c = ((u64)e.w << 32) | e.z;
        u64 step = (p * it.qs) << 2;
        u32 yn[L];  // the lane's next seed; its P and rem are Pn and rem0
        if (L == 2) {
          const u64 x = (it.q_lo * p + c + (A.negative ? 1ull : ~0ull)) << 2;
          yn[0] = (u32)x;
          yn[1] = (u32)(x >> 32);
        } else {
          const u128 x = ((((u128)it.q_hi << 64) | it.q_lo) * p + c + (A.negative ? (u128)1 : ~(u128)0)) << 2;
#pragma unroll
          for (int i = 0; i < L; i++) yn[i] = (u32)(x >> (32 * i));
        }
        // Pn = (limit - D0) << 16 | D0; a negative one sends the lane's seeds to the exact path
        u32 Pn;
        int rem0;  // windows a seed may take after its first
        auto limits = [&]() {
          const RunLimits lim = run_limits<L, JW>(W.cur, lgn, (int)A.k);
          const bool small = A.k < 16 && it.q_hi == 0 && it.q_lo < (MIN_WINDOW_SEED >> A.k);
          const bool flag = small || lim.lim < D0 || emx >= lim.elim || lim.wmax < 1;
          Pn = flag ? 0x80000000u : ((u32)lim.lim << 16) - (u32)(D0 * 65535);
          rem0 = lim.wmax - 1;
        };
        limits();
        // the lane's current seed, and how many follow it (negative: the lane has none; it
        // then runs on beyond its rows, to no effect)
        u32 y[L], P = Pn;
        int rem = rem0, left = valid ? (int)it.rows - 1 : -1;
#pragma unroll
        for (int i = 0; i < L; i++) y[i] = yn[i];
        add_step<L>(yn, step);
        auto take_next = [&]() {
          P = Pn;
          rem = rem0;
#pragma unroll
          for (int i = 0; i < L; i++) y[i] = yn[i];
          add_step<L>(yn, step);
          left--;
        };
        for (;;) {
          // windows, until a seed is at a limit or STOP lanes have run out of seeds; the
          // latter is looked at after every second window
          bool stop = false;
          for (;;) {
            if (__any_sync(FULL, ((P | (u32)rem) & 0x80000000u) != 0)) break;
            u32 tst = window<L, JW>(y, P, y, P, s_win, s_cls);
            rem--;
            next_if_done<L>(tst, y, yn, step, P, Pn, rem, rem0, left);
            if (__any_sync(FULL, ((P | (u32)rem) & 0x80000000u) != 0)) break;
            tst = window<L, JW>(y, P, y, P, s_win, s_cls);
            rem--;
            next_if_done<L>(tst, y, yn, step, P, Pn, rem, rem0, left);
            stop = __popc(__ballot_sync(FULL, left < 0)) >= STOP;
            if (stop) break;
          }
          // the seeds at a limit go to the exact path (rare)
          const bool lim = (int)(P | (u32)rem) < 0;
          const bool bad = lim && left >= 0;
          if (__any_sync(FULL, bad)) {
            const u32 meta = (j * 32 + lane) | (slot << 6) | ((it.rows - 1 - (u32)left) << 11);
            push_slow<L>(W, A, Q.slow, bad, meta);
            if (Q.slow >= 32u) {
              volatile u32 keep[2 * L + 5];  // the lanes' state, so that the call leaves the loop's registers alone
#pragma unroll
              for (int i = 0; i < L; i++) {
                keep[i] = y[i];
                keep[L + i] = yn[i];
              }
              keep[2 * L] = P;
              keep[2 * L + 1] = (u32)rem;
              keep[2 * L + 2] = (u32)left;
              keep[2 * L + 3] = (u32)step;
              keep[2 * L + 4] = (u32)(step >> 32);
              drain_warp<L, JW, WARPS>(A, lane, Q, false);
#pragma unroll
              for (int i = 0; i < L; i++) {
                y[i] = keep[i];
                yn[i] = keep[L + i];
              }
              P = keep[2 * L];
              rem = (int)keep[2 * L + 1];
              left = (int)keep[2 * L + 2];
              step = ((u64)keep[2 * L + 4] << 32) | keep[2 * L + 3];
              limits();
            }
            if (bad) take_next();
          } else if (stop) {
            break;
          }
          if (left < 0 && (int)(Pn | P | (u32)rem) < 0) {  // a lane without seeds is at no limit
            P = Pn = 0xC000u;
            rem = rem0 = 1 << 20;
          }
        }
        // what the other lanes still have is queued: their current seeds, then their next ones
        for (;;) {
          const bool has = left >= 0;
          const u32 b = __ballot_sync(FULL, has);
          if (!b) break;
          if (has) {
            const u32 meta = (j * 32 + lane) | (slot << 6) | ((it.rows - 1 - (u32)left) << 11) | ((u32)(rem - 1) << 26);
            mid_store<L>(W, Q.mid + __popc(b & ((1u << lane) - 1u)), y, P, meta);
            take_next();
          }
          Q.mid += __popc(b);
          if ((Q.mid | Q.slow) >= 32u && work_off<L, JW, WARPS>(W, A, lane, Q, s_win, s_cls)) limits();
        }
      }
    } else {
      // integers below 2^k: no residue sieve, no jump
      stage_next(W, W.run[ring & 1u], A, lane, nwarps);
      const float lgn = 1e-5f + __log2f(__ull2float_ru(it.q_lo + (ull)it.rows * DENSE_ITEM));
      const u32 keep9 = A.negative ? KEEP9N : KEEP9;
      u32 seeds = 0;
#pragma unroll 1
      for (u32 t = 0; t < 2 * it.rows; t++) {
        const u32 idx = (t & 1u) * 32 + lane;
        const ull n = it.q_lo + (t >> 1) * DENSE_ITEM + idx;
        const bool in = n < it.d_hi && n >= 2 &&
                        (!it.mod9 || ((keep9 >> (u32)(n % 9u)) & 1u) || (A.negative && n == 5));
        seeds += __popc(__ballot_sync(FULL, in));
        const RunLimits lim = run_limits<L, JW>(W.cur, lgn, 0);
        const bool flag = in && (it.q_lo < MIN_WINDOW_SEED || lim.lim < 0 || lim.wmax < 1);
        const u32 meta = idx | (slot << 6) | ((t >> 1) << 11) | ((u32)(lim.wmax - 2) << 26);
        if (__any_sync(FULL, flag)) push_slow<L>(W, A, Q.slow, flag, meta);
        u32 y[L], P = (in && !flag) ? (u32)lim.lim << 16 : 0xC000u;
#pragma unroll
        for (int i = 0; i < L; i++) y[i] = i == 0 ? (u32)(n << 2) : i == 1 ? (u32)(n >> 30) : 0u;
        u32 z[L];
        const bool keep = !(window<L, JW>(y, P, z, P, s_win, s_cls) & 0x8000u);
        const u32 b = __ballot_sync(FULL, keep);
        if (keep) mid_store<L>(W, Q.mid + __popc(b & ((1u << lane) - 1u)), z, P, meta);
        Q.mid += __popc(b);
        if ((Q.mid | Q.slow) >= 32u) drain_warp<L, JW, WARPS>(A, lane, Q, false);
      }
      if (lane == 0) W.acc_seeds += seeds;
    }
  }
  drain_warp<L, JW, WARPS>(A, lane, Q, true);
  // the warps' last seeds for the exact path, together: 32 to a warp
  if (lane == 0) S.last[threadIdx.x >> 5] = Q.slow;
  __syncthreads();
  {
    u32 at = threadIdx.x, total = 0;  // this lane's seed among all
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    bool have = false;
    for (u32 i = 0; i < WARPS; i++) {
      const u32 c = S.last[i];
      if (!have && at - total < c) {
        e = S.w[i].slow[at - total];
        have = true;
      }
      total += c;
    }
    if (__any_sync(FULL, have)) {
      exact_seeds(A, e, have);
      if (A.stats && lane == 0) atomicAdd(&A.stats[1], (ull)min(32u, total - threadIdx.x));
    }
  }
  if (lane == 0 && W.req != FULL) {
    if (W.acc_seeds) atomicAdd(&A.recs[W.req].seeds, W.acc_seeds);
    atomicAdd(&A.recs[W.req].items_done, W.acc_rows);
  }
  if (A.stats && lane == 0) atomicAdd(&A.stats[0], (ull)ring);
}

// ------------------------------------------------------------------
// Wide re-run: one seed per thread with L limbs, from scratch.
// ------------------------------------------------------------------
template <int L, bool NEG>
__global__ void __launch_bounds__(128) k_range_wide(const WidenEntry* __restrict__ list, const u32* count,
                                                   u32 cap, ReqRec* recs, WidenEntry* next, u32 next_cap,
                                                   u32* next_count, u32 iter_cap) {
  const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
  const u32 n = min(*count, cap);
  const u32 lane = lane_id();
  bool ok = false;
  WidenEntry e{0, 0, 0, 0};
  Limbs<L> v, N, E;
  unsigned long long st = 0;
  if (i < n) {
    e = list[i];
#pragma unroll
    for (int j = 0; j < L; j++) N.w[j] = (j == 0) ? e.n0 : (j == 1) ? e.n1 : (j == 2) ? e.n2 : 0u;
    v = N;
    if (NEG) dec_l<L>(v); else inc_l<L>(v);  // v = n + 1, or u = n - 1 for T'
    E = N;
    u32 it = 0;
    for (;;) {
      if (v.w[L - 1] >= (1u << 19) || ++it > iter_cap) {
        if (it > iter_cap) {
          atomicOr(&recs[e.req].errors, ERR_ITER_CAP);
          atomicAdd(&recs[e.req].failures, 1ull);
        } else if (next) {
          const u32 wi = atomicAdd(next_count, 1u);
          if (wi < next_cap) {
            next[wi] = e;
          } else {
            atomicOr(&recs[e.req].errors, ERR_WIDEN_FULL);
            atomicAdd(&recs[e.req].failures, 1ull);
          }
        } else {
          atomicAdd(&recs[e.req].failures, 1ull);
        }
        break;
      }
      const u32 a = ctz32(v.w[0] | (1u << 8));
      u32 m = 1;
      for (u32 j = 0; j < a; j++) m *= 3u;
      odd_run_l<L>(v, a, m);
      st += a;
      Limbs<L> x = v;  // the value: v - 1, or u + 1 for T'
      if (NEG) inc_l<L>(x); else dec_l<L>(x);
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
        ok = true;
        break;
      }
      st += b;
      if (NEG && !limbs_lt<L>(w, N) && !limbs_lt<L>(N, w)) {  // back at the seed: a cycle
        atomicAdd(&recs[e.req].failures, 1ull);
        break;
      }
      v = w;
      if (NEG) dec_l<L>(v); else inc_l<L>(v);
    }
  }
  u32 pm = __ballot_sync(FULL, ok);
  while (pm) {
    const u32 leader = __ffs(pm) - 1;
    if (lane == leader) {
      const u32 seed[4] = {e.n0, e.n1, e.n2, 0};
      rec_offer_st(recs + e.req, st, seed);
      rec_offer_e<L>(recs + e.req, E.w, seed);
    }
    pm &= pm - 1;
  }
}

// ------------------------------------------------------------------
// Threshold scouts, launched before k_range.  A request's keys start at zero,
// and under zero limits every seed takes the exact path.  Warp (i, s) runs 32
// seeds of request i's scout segment (row s) in full and raises the request's
// keys to the largest stopping time and excursion among them.  These are seeds
// the request checks, so the keys stay lower bounds of its maxima, and k_range
// still offers them (values equal to a threshold pass every test).
// ------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_range_scout(const __grid_constant__ RangeArgs A,
                                                     const u32* __restrict__ first_seg, u32 nreq, u32 subs) {
  const u32 wi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = lane_id();
  if (wi >= nreq * subs) return;  // warp-uniform
  const u32 si = first_seg[wi / subs], row = wi % subs;
  if (si >= A.nsegs) return;  // a request without seeds
  const RangeSeg g = A.segs[si];
  if (g.local0_lo | g.local0_hi) return;  // not the segment's first row
  const ull rows = g.kind == 0 ? (ull)g.nq * g.ipq : (g.d_hi - g.q_lo) / DENSE_ITEM;
  if (row && row >= rows / 8) return;  // an eighth of a small segment is enough
  const bool neg = A.negative != 0;
  const u32 keep9 = neg ? KEEP9N : KEEP9;
  // this lane's seed: entry lane of the row, or integer d_lo + 64 row + lane
  bool have = false;
  u128 n = 2;
  if (g.kind == 0) {
    const u32 chunk = row % g.ipq, qi = row / g.ipq;
    const u32 idx = g.s_lo + chunk * RANGE_ITEM + lane;
    if (qi < g.nq && idx < g.s_hi) {
      const RangeEntry e = A.table[idx];
      const u128 q = (((u128)g.q_hi << 64) | g.q_lo) + (u128)qi * (g.qstride ? g.qstride : 1u);
      n = (q << A.k) | ((u64)(e.meta & 0xFFu) << 32) | e.r_lo;
      have = true;
    }
  } else {
    const ull m = g.q_lo + 64ull * row + lane;
    if (m < g.d_hi && m >= 2 && (!g.mod9 || ((keep9 >> (u32)(m % 9u)) & 1u))) {
      n = m;
      have = true;
    }
  }
  const ExactSeed R = exact_run(n, have, neg);
  u32 sig = R.ok ? R.st : 0u;
  u32 E[4];
#pragma unroll
  for (int i = 0; i < 4; i++) E[i] = (u32)(R.E >> (32 * i));
  ull ekey = R.ok ? key_of<4>(E) : 0ull;
  sig = __reduce_max_sync(FULL, sig);
#pragma unroll
  for (u32 d = 16; d; d >>= 1) ekey = max(ekey, (ull)__shfl_xor_sync(FULL, ekey, d));
  if (lane == 0) {
    if (sig) atomicMax(&A.recs[g.req].st_key, (ull)sig);
    if (ekey) atomicMax(&A.recs[g.req].e_key, ekey);
  }
}

// ------------------------------------------------------------------
// Launchers.
// ------------------------------------------------------------------

// (window length JW, STOP, warps per block).  Measured on B200, 2^36 seeds: at 2^40 (two
// words, k = 24) 2.47 ms for variant 0, 2.48 for 1, 2.53 for 2, 2.56 for 3 (JW 12), 2.62 for 4
// (JW 11), 2.53 for 5, 2.62 for 6, 3.17 for 7 (16 warps); at 2^60 (three words, k = 34) 5.17,
// 5.15, 5.32, 5.09, 5.20, 5.04, 5.34, 6.53.  Longer windows (JW 14, a 64 KB table) measured
// as JW 13 and lost bits of the table's m.
#define CZ_RANGE_VARIANTS(X)                                                                       \
  X(0, 13, 20, 32) X(1, 13, 16, 32) X(2, 13, 24, 32) X(3, 12, 20, 32) X(4, 11, 20, 32) X(5, 13, 20, 28) \
  X(6, 13, 20, 24) X(7, 13, 20, 16)

int range_variants() { return 8; }
int range64_variants() { return 8; }
uint32_t range64_max_seed_bits() { return 48; }

// FNV-1a of the variant table's parameters: part of the autotuner's cache key, so that a
// choice cached for another table is not applied to this one.
uint32_t range_variant_rev() {
  static const int p[] = {
#define X(id, jw, c1, wp) id, jw, c1, wp,
      CZ_RANGE_VARIANTS(X)
#undef X
  };
  uint32_t h = 2166136261u;
  for (int x : p) h = (h ^ (uint32_t)x) * 16777619u;
  return h;
}

template <int L>
static cudaError_t launch_t(const RangeArgs& a, int variant, u32 grid, cudaStream_t st) {
  switch (variant) {
#define X(id, jw, c1, wp)                                                                               \
  case id:                                                                                              \
    k_range<L, jw, c1, wp><<<grid, wp * 32, sizeof(RangeShared<L, jw, wp>), st>>>(a);            \
    break;
    CZ_RANGE_VARIANTS(X)
#undef X
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_range(const RangeArgs& a, int words, int variant, u32 sm_count, cudaStream_t st) {
  const u32 grid = (u32)std::max<unsigned long long>(1, std::min<unsigned long long>(sm_count, a.item_limit));
  switch (words) {
    case 2: return launch_t<2>(a, variant, grid, st);
    case 3: return launch_t<3>(a, variant, grid, st);
    case 4: return launch_t<4>(a, variant, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int L>
static cudaError_t init_t() {
  cudaError_t e = cudaSuccess;
#define X(id, jw, c1, wp)                                                                                   \
  if (e == cudaSuccess)                                                                                     \
    e = cudaFuncSetAttribute(k_range<L, jw, c1, wp>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                             (int)sizeof(RangeShared<L, jw, wp>));
  CZ_RANGE_VARIANTS(X)
#undef X
  return e;
}

// Opts every range kernel into its dynamic shared memory and fills the window tables.
cudaError_t range_init(cudaStream_t st) {
  cudaError_t e = init_t<2>();
  if (e == cudaSuccess) e = init_t<3>();
  if (e == cudaSuccess) e = init_t<4>();
  if (e != cudaSuccess) return e;
  k_win_tables<<<(1u << MAX_JW) / 256, 256, 0, st>>>();
  e = cudaGetLastError();
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

cudaError_t launch_range_scout(const RangeArgs& a, const u32* first_seg, u32 nreq, cudaStream_t st) {
  if (!nreq) return cudaSuccess;
  const u32 subs = std::max(1u, std::min(512u, 1024u / nreq));
  k_range_scout<<<(nreq * subs + 3) / 4, 128, 0, st>>>(a, first_seg, nreq, subs);
  return cudaGetLastError();
}

cudaError_t launch_range_wide(const WidenEntry* list, const u32* count, u32 cap, int limbs, ReqRec* recs,
                              WidenEntry* next, u32 next_cap, u32* next_count, u32 iter_cap, cudaStream_t st,
                              bool negative) {
  const u32 grid = (cap + 127) / 128;
  if (limbs == 6) {
    if (negative)
      k_range_wide<6, true><<<grid, 128, 0, st>>>(list, count, cap, recs, next, next_cap, next_count, iter_cap);
    else
      k_range_wide<6, false><<<grid, 128, 0, st>>>(list, count, cap, recs, next, next_cap, next_count, iter_cap);
  } else {
    if (negative)
      k_range_wide<8, true><<<grid, 128, 0, st>>>(list, count, cap, recs, nullptr, 0, nullptr, iter_cap);
    else
      k_range_wide<8, false><<<grid, 128, 0, st>>>(list, count, cap, recs, nullptr, 0, nullptr, iter_cap);
  }
  return cudaGetLastError();
}

}  // namespace cz
