// cases_win.cu -- Step 2 + Step 3 (collatz_cudav7.cu compute_kernel, cu:185-411) for N <= 52,
// with the checkpoints' run pairs taken from a table.
//
// A checkpoint is two run pairs [odd run <= 8, even run <= 31]; the hash is the XOR of
// v = T^i(n) + 1 at every checkpoint, and a seed stops at its first checkpoint with v < n
// (cu:280-405).  The low 13 bits of v fix the runs that end inside 12 steps, so one look-up takes
// two pairs for 93 % of values, else one (then the next look-up, in a second table,
// takes the checkpoint's other pair), else none (0.3 %: the pair's runs are counted).  With s steps, f
// of them odd, v -> (v >> s) 3^f + t: for x = v - 1 = q 2^s + r, T^s(x) = q 3^f + T^s(r), and v >> s is q,
// or q + 1 when r = 2^s - 1, where T^s(r) + 1 - 3^f = 0.
//
// Stopping times and excursions are only bounded on the way.  A seed whose value
// reaches 1/256 of the line's maximum excursion (a look-up's odd runs raise it by less than
// 1.5^12 = 130) or a bound below 2^71 (case_limits.h), or whose look-ups could hold as many steps as the line's longest
// stopping time, is queued and run again from its start, pair by pair with four limbs:
// overflow reports, exact maxima, its hash (exact_batch).  No other seed can change a
// maximum, report an overflow or reach the checkpoint cap.
#include <cuda_runtime.h>

#include <algorithm>

#include "case_limits.h"
#include "common.cuh"
#include "fill_once.h"
#include "kernels.h"
#include "tables.h"

namespace cz {

constexpr u32 WQ = 1024;       // queue entries per warp (>= 31 + 570 survivors of one pair)
constexpr u32 WR = 32;         // pair slots per warp (a queue of < 32 entries spans < 32 pairs)
constexpr u32 WWARPS = 32;     // per block, one block per SM
constexpr u32 WCLAIM = 16;     // pairs per claim while many remain
constexpr int WGROUP = 4;      // look-ups between two looks at the lanes
constexpr int WREFILL = 20;    // lanes without a next seed that call for a refill
constexpr u32 CP_BITS = 13;    // low bits of a look-up
constexpr int IDLE_CNT = 1 << 30;

// Entries, [0] before a checkpoint's first pair, [1] before its second: t << 12 | (1: a first pair was
// taken) << 10 | (1: at a checkpoint) << 9 | f << 5 | s; s = 0: no pair ends.
constexpr u32 CP_HALF = 1u << 10, CP_DONE = 1u << 9, CP_F = 0xFu << 5;
__device__ u32 g_cp[2][1u << CP_BITS];
__device__ u32 g_cp_ready;  // 1: the tables are filled

__global__ void k_cp_tables() {
  const u32 m = blockIdx.x * blockDim.x + threadIdx.x;  // low bits of v
  if (m >> CP_BITS) return;
  const u32 r = (m - 1u) & ((1u << CP_BITS) - 1u);
  for (u32 half = 0; half < 2; half++) {
    u32 x = r, known = CP_BITS, s = 0, f = 0, pairs = 0;
    while (pairs < 2u - half) {
      u32 y = x, k = known, a = 0, b = 0;
      while (a < 8 && k && (y & 1u)) {
        y = y + (y >> 1) + 1u;
        a++;
        k--;
      }
      if (k == 0) break;  // the run may go on
      while (k && !(y & 1u)) {
        y >>= 1;
        b++;
        k--;
      }
      if (k == 0) break;
      x = y;
      known = k;
      s += a + b;
      f += a;
      pairs++;
    }
    u32 t = r & ((1u << s) - 1u);
    if (t == (1u << s) - 1u) {
      t = 0;
    } else {
      for (u32 i = 0; i < s; i++) t = (t & 1u) ? t + (t >> 1) + 1u : t >> 1;
      t++;
    }
    const bool done = pairs + half == 2;
    g_cp[half][m] = (t << 12) | ((!done && pairs + half == 1) ? CP_HALF : 0u) | (done ? CP_DONE : 0u) | (f << 5) | s;
  }
}

struct CwWarp {
  uint2 slow[64];             // seeds for the exact path: pair, a
  unsigned short q[WQ];       // (slot << 10) | a
  uint4 ring[WR][3];          // base0..1, number0..2, 3^f limbs 0..2, limits, pair, line, limbs above those
                              // kept (2: of the base, 1: of the values only; the pair's seeds then all go to the
                              // exact path)
};

struct CwShared {
  u32 tab[2][1u << CP_BITS];
  u32 p3[16];
  CwWarp w[WWARPS];
};

static_assert(sizeof(CwShared) <= MAX_BLOCK_SMEM, "shared memory of a block");

extern __shared__ __align__(16) unsigned char cw_smem[];

__device__ __forceinline__ u32 lds32(u32 at) {
  u32 v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
  return v;
}

// The queued seeds of all lanes with have, from their starts to their last checkpoints:
// the reference's checkpoint structure with four limbs.
template <bool MULTI>
__device__ __forceinline__ void exact_batch(const CasesArgs& A, uint2 e, bool have) {
  const u32 lane = lane_id();
  const u32* P = A.pairs + 8ull * e.x;
  const u32 a10 = e.y;
  const u32 b3 = P[3];
  const u32 line = MULTI ? b3 >> 8 : 0u;
  ReqRec* rec = A.rec + line;
  u32 bi = (A.bigindex >= 0) ? (u32)A.bigindex : (MULTI ? (b3 & 0xFFu) : b3);
  const bool cpu = bi >= 16u;
  u32 f = A.tpo + bi;
  if (f >= POW3_COUNT) f = POW3_COUNT - 1;
  const u64 n = (((u64)P[1] << 32) | P[0]) | ((u64)a10 << A.mbi);
  const u32 n0 = (u32)n, n1 = (u32)(n >> 32), n2 = P[2];
  u64 t = (u64)a10 * A.pow3[4u * f] + P[4];
  u32 v0 = (u32)t;
  t = (u64)a10 * A.pow3[4u * f + 1] + P[5] + (t >> 32);
  u32 v1 = (u32)t;
  t = (u64)a10 * A.pow3[4u * f + 2] + P[6] + (t >> 32);
  u32 v2 = (u32)t;
  u32 v3 = a10 * A.pow3[4u * f + 3] + P[7] + (u32)(t >> 32);
  const ull sk = *(volatile ull*)&rec->st_key;
  u32 E[4];  // the excursion threshold, then the seed's maximum
  key_decode<4>(*(volatile ull*)&rec->e_key, E);
  const u32 nbl = bitlen96(n0, n1, n2);
  u32 st = A.mbi, sig = 0, hash = 0, iters = 0;
  bool found = false, ovf = false, evalid = false, alive = have, good = false;
  auto candidate = [&]() {  // x = v - 1 against the maximum so far
    const u32 x0 = v0 - 1, x1 = v1 - (v0 == 0), x2 = v2 - ((v0 | v1 | v2) == 0), x3 = v3 - ((v0 | v1 | v2) == 0);
    if (x3 > E[3] || (x3 == E[3] && !lt96c(x0, x1, x2, E[0], E[1], E[2]))) {
      E[0] = x0;
      E[1] = x1;
      E[2] = x2;
      E[3] = x3;
      evalid = true;
    }
  };
  candidate();  // E candidate T^(N-A)(n)
#pragma unroll 1
  while (__any_sync(FULL, alive)) {
    if (alive) {
#pragma unroll 1
      for (int half = 0; half < 2; half++) {
        const u32 a = ctz32(v0 | (1u << 8));
        odd_run4(v0, v1, v2, v3, a, pow3_le8(a));
        st += a;
        if (v3 >= 16u && !(half == 1 && cpu && v3 == 16u && (v0 | v1 | v2) == 0u)) {
          // v >= 2^100 (cu:295, 334); search3 tests > on the second (cu:702)
          const ull i = atomicAdd(A.overflow_count, 1ull);
          if (i < A.overflow_cap) {
            A.overflow[4 * i + 0] = n0;
            A.overflow[4 * i + 1] = n1;
            A.overflow[4 * i + 2] = n2;
            A.overflow[4 * i + 3] = line;
          }
          if (MULTI) atomicAdd(&rec->items_done, 1ull);  // the line's overflow reports
          ovf = true;
          v0 = 2;
          v1 = v2 = v3 = 0;
        } else if (!found && !ovf) {
          candidate();
        }
        v0 -= 1;
        const u32 b = ctz32(v0 | 0x80000000u);
        const u32 w0 = __funnelshift_r(v0, v1, b), w1 = __funnelshift_r(v1, v2, b);
        const u32 w2 = __funnelshift_r(v2, v3, b), w3 = v3 >> b;
        if (!(found | ovf) & (b != 0) & (w3 == 0) & lt96c(w0, w1, w2, n0, n1, n2)) {
          // first descent inside this run: smallest i with (v-1) >> i < n
          sig = st + first_below(v0, v1, v2, v3, n0, n1, n2, nbl);
          found = true;
        }
        st += b;
        v0 = w0 + 1;
        v1 = w1;
        v2 = w2;
        v3 = w3;
        add_carry3(v1, v2, v3, (v0 == 0) & (b != 0));  // carry of the +1 (cu:310-318)
      }
      hash ^= v0;  // cu:359
      iters++;
      const bool done = (v3 == 0) & lt96c(v0, v1, v2, n0, n1, n2);  // cu:362-365
      if (done || iters >= A.iter_cap) {
        alive = false;
        good = done && !ovf;
        if (!done) {
          atomicOr(&rec->errors, ERR_ITER_CAP);
          atomicAdd(&rec->failures, 1ull);
        }
      }
    }
  }
  if (have) atomicXor(&rec->hash, hash);
  const u32 sigma = found ? sig : st;
  const bool ps = good && sigma >= sk, pe = good && evalid;
  u32 pm = __ballot_sync(FULL, ps | pe);
#pragma unroll 1
  while (pm) {  // of one line's seeds that may raise a maximum, the best is offered
    const u32 ln = __shfl_sync(FULL, line, __ffs(pm) - 1);
    const bool in = (ps | pe) & (line == ln);
    const u32 sm = __reduce_max_sync(FULL, (in & ps) ? sigma + 1 : 0u);
    u32 cs = __ballot_sync(FULL, in & ps & (sigma + 1 == sm));
    u32 ce = __ballot_sync(FULL, in & pe);
#pragma unroll
    for (int i = 3; i >= 0; i--) {  // the lanes with the largest excursion
      const u32 m = __reduce_max_sync(FULL, ((ce >> lane) & 1u) ? E[i] : 0u);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && E[i] == m);
    }
#pragma unroll
    for (int i = 2; i >= 0; i--) {  // the smallest seed of each
      const u32 nl = i == 2 ? n2 : i ? n1 : n0;
      const u32 s = __reduce_min_sync(FULL, ((cs >> lane) & 1u) ? nl : FULL);
      cs = __ballot_sync(FULL, ((cs >> lane) & 1u) && nl == s);
      const u32 x = __reduce_min_sync(FULL, ((ce >> lane) & 1u) ? nl : FULL);
      ce = __ballot_sync(FULL, ((ce >> lane) & 1u) && nl == x);
    }
    const u32 seed[4] = {n0, n1, n2, 0u};
#pragma unroll 1
    for (u32 kind = 0; kind < 2; kind++) {
      const u32 set = kind ? ce : cs;
      const bool lead = set != 0 && lane == (u32)__ffs(set) - 1;
      const ull key = kind ? key_of<4>(E) : (ull)sigma;
      if (lead) atomicMax(kind ? &rec->e_key : &rec->st_key, key);
      rec_offer_vote<true>(rec, lead, kind, key, sigma, E, seed);
    }
    pm &= ~__ballot_sync(FULL, in);
  }
}

// Lane state: v (0: idle; a fixed point of the look-ups that leaves the hash alone), n, the seed's
// hash so far, the largest v in the limit's units and that limit, the look-ups left, the address of the
// table for its next look-up; and the lane's next seed, so that a refill serves most lanes.
// Bound by issue (77 % busy, the ALU 75 %): 18.8 warp instructions per seed against 49.7 with
// the runs counted in 64-bit pairs; a seed takes about six look-ups, so that half the
// instructions hand seeds to lanes.  555.7 M seeds of one line (27 10 8 183 0 0): 28.6 -> 11.9 ms,
// 2048 lines: 14.2 -> 6.5 ms.  Groups of 3 look-ups 9.9 ms, of 2 10.6; a refill at 26 lanes 9.7; without
// the next seed in the lane 10.1; 24 warps with 80 registers 10.1.
// UNIT: the limits' unit, or 0 for A.unit.
template <bool MULTI, u32 UNIT>
__global__ void __launch_bounds__(WWARPS * 32, 1) k_cases_win(const __grid_constant__ CasesArgs A) {
  CwShared& S = *reinterpret_cast<CwShared*>(cw_smem);
  const u32 unit = UNIT ? UNIT : A.unit;
  for (u32 i = threadIdx.x; i < (2u << CP_BITS); i += WWARPS * 32) (&S.tab[0][0])[i] = (&g_cp[0][0])[i];
  if (threadIdx.x < 16) {
    u32 p = 1;
#pragma unroll 1
    for (u32 i = 0; i < threadIdx.x; i++) p *= 3u;
    S.p3[threadIdx.x] = p;
  }
  const u32 lane = lane_id();
  CwWarp& W = S.w[threadIdx.x >> 5];
  W.ring[lane][2].z = 0;
  __syncthreads();
  const u32 tab = (u32)__cvta_generic_to_shared(&S.tab[0][0]), p3 = (u32)__cvta_generic_to_shared(S.p3);
  const u32 mbi = A.mbi;
  // warp-uniform state
  u32 qhead = 0, qcount = 0, ring_seq = 0, ns = 0, warp_seeds = 0;
  u32 pc = 0, pc_end = 0;  // claimed pairs
  u32 wline = 0;           // MULTI: the line whose seeds warp_seeds counts
  bool exhausted = false, last = false, end = false;  // no more pairs, none in the queue, none in the lanes
  // lane state
  u32 v0 = 0, v1 = 0, v2 = 0, n0 = 0, n1 = 0, hs = 0, hash = 0, mx = 0, hi = 1, hb = tab, pair = FULL;
  u32 w0 = 0, w1 = 0, w2 = 0, m0 = 0, m1 = 0, npair = 0, na10 = 0, nlim = 0, nline = 0, a10 = 0;  // the next seed (w = 0: none)
  u32 hline = 0;  // MULTI: the line of the lane's seed and of hash
  int cnt = IDLE_CNT;

  for (;;) {
    if (ns >= 32u || (end && ns)) {
      // ---- the exact path (the lanes' state is put away around it) ----
      volatile u32 keep[23];
      keep[21] = a10;
      keep[22] = na10;
      keep[0] = v0;
      keep[1] = v1;
      keep[2] = v2;
      keep[3] = n0;
      keep[4] = n1;
      keep[5] = hs;
      keep[6] = hash;
      keep[7] = mx;
      keep[8] = hi;
      keep[9] = hb;
      keep[10] = pair;
      keep[11] = w0;
      keep[12] = w1;
      keep[13] = w2;
      keep[14] = m0;
      keep[15] = m1;
      keep[16] = npair;
      keep[17] = nlim;
      keep[18] = nline;
      keep[19] = hline;
      keep[20] = (u32)cnt;
      __syncwarp();
      const u32 c = min(ns, 32u);
      ns -= c;
      const bool have = lane < c;
      const uint2 e = W.slow[ns + (have ? lane : 0u)];
      exact_batch<MULTI>(A, e, have);
      __syncwarp();
      {  // the lines' maxima may have risen
        const ReqRec* r = A.rec + W.ring[lane][2].z;
        W.ring[lane][2].x = line_limits(*(volatile const ull*)&r->st_key, *(volatile const ull*)&r->e_key, mbi, A.iter_cap, unit);
      }
      __syncwarp();
      v0 = keep[0];
      v1 = keep[1];
      v2 = keep[2];
      n0 = keep[3];
      n1 = keep[4];
      hs = keep[5];
      hash = keep[6];
      mx = keep[7];
      hi = keep[8];
      hb = keep[9];
      pair = keep[10];
      w0 = keep[11];
      w1 = keep[12];
      w2 = keep[13];
      m0 = keep[14];
      m1 = keep[15];
      npair = keep[16];
      nlim = keep[17];
      nline = keep[18];
      hline = keep[19];
      cnt = (int)keep[20];
      a10 = keep[21];
      na10 = keep[22];
      continue;
    }
    if (end) break;
    const u32 lack = __ballot_sync(FULL, (w0 | w1 | w2) == 0);
    const u32 nlack = __popc(lack);
    {
      // ---- refill the queue and give lanes without one their next seed ----
      while (__any_sync(FULL, qcount < nlack && !exhausted)) {
        if (__any_sync(FULL, pc >= pc_end)) {
          const u32 claim = ((ull)pc + (ull)WCLAIM * gridDim.x * WWARPS < A.npairs) ? WCLAIM : 1u;
          u32 p0 = 0;
          if (lane == 0) p0 = atomicAdd(A.pair_counter, claim);
          pc = __shfl_sync(FULL, p0, 0);
          pc_end = (pc < A.npairs) ? min(A.npairs, pc + claim) : pc;
        }
        const u32 p = pc++;
        if (__any_sync(FULL, p >= A.npairs)) {
          exhausted = true;
          break;
        }
        // Step 2 (cu:198-235): sieve words for this pair
        const u32* P = A.pairs + 8ull * p;
        const u32 pw = (lane < 8) ? P[lane] : 0u;
        const u32 b0 = __shfl_sync(FULL, pw, 0), b1 = __shfl_sync(FULL, pw, 1);
        const u32 b2 = __shfl_sync(FULL, pw, 2), b3 = __shfl_sync(FULL, pw, 3);
        const u32 m0 = __shfl_sync(FULL, pw, 4), n3 = __shfl_sync(FULL, pw, 7);
        const u32 pline = MULTI ? (b3 >> 8) : 0u;
        const ReqRec* prec = A.rec + pline;
        const u32 lim = line_limits(*(volatile const ull*)&prec->st_key, *(volatile const ull*)&prec->e_key, mbi, A.iter_cap, unit);
        const u32 bi = (A.bigindex >= 0) ? (u32)A.bigindex : (MULTI ? (b3 & 0xFFu) : b3);
        u32 f = A.tpo + bi;
        if (f >= POW3_COUNT) f = POW3_COUNT - 1;
        const u32 red = ((b0 % 9u) + 4u * (b1 % 9u) + 7u * (b2 % 9u)) % 9u;  // 2^32 = 4, 2^64 = 7 (mod 9)
        u32 word = A.mod9[red * 32u + lane];
        if (__any_sync(FULL, bi < 16u)) {
          const u32 idx = (A.magic[bi] * m0) & ((1u << 24) - 1);
          const u32* row = A.bv + (size_t)bi * BV_WORDS + (idx >> 5);
          const u32 lo = row[lane];
          u32 up = __shfl_down_sync(FULL, lo, 1);
          if (lane == 31) up = row[32];
          word &= __funnelshift_r(lo, up, idx & 31u);
        }
        u32 total;
        const u32 excl = warp_excl_scan(__popc(word), &total);
        if (__any_sync(FULL, total != 0)) {
          const u32 slot = ring_seq & (WR - 1);
          ring_seq++;
          const u32 rv = __shfl_sync(FULL, pw, lane < 2 ? lane : lane + 2);  // base0..1, number0..2
          u32* R = reinterpret_cast<u32*>(W.ring[slot]);
          if (lane < 5) R[lane] = rv;
          if (lane >= 5 && lane < 8) R[lane] = A.pow3[4u * f + (lane - 5)];
          if (lane == 8) R[8] = lim;
          if (lane == 9) R[9] = p;
          if (lane == 10) R[10] = pline;
          if (lane == 11) R[11] = b2 ? 2u : (n3 | A.pow3[4u * f + 3]) != 0;
          if (MULTI && __any_sync(FULL, pline != wline)) {  // seeds are counted per warp until the line changes
            if (lane == 0 && warp_seeds) atomicAdd(&A.rec[wline].seeds, (ull)warp_seeds);
            warp_seeds = 0;
            wline = pline;
          }
          u32 pos = qhead + qcount + excl;
          while (word) {
            const u32 j = ctz32(word);
            word &= word - 1;
            W.q[pos & (WQ - 1)] = (unsigned short)((slot << 10) | (lane * 32u + j));
            pos++;
          }
          qcount += total;
          warp_seeds += total;
          if (!MULTI && __any_sync(FULL, warp_seeds >= 1u << 30)) {
            if (lane == 0) atomicAdd(&A.rec->seeds, (ull)warp_seeds);
            warp_seeds = 0;
          }
        }
        __syncwarp();
      }
      const u32 take = min(nlack, qcount);
      const u32 rank = __popc(lack & lanemask_lt());
      if ((w0 | w1 | w2) == 0 && rank < take) {
        const u32 q = W.q[(qhead + rank) & (WQ - 1)];
        const uint4 r0 = W.ring[q >> 10][0], r1 = W.ring[q >> 10][1], r2 = W.ring[q >> 10][2];
        const u32 a = q & 1023u;
        const u64 n = (((u64)r0.y << 32) | r0.x) | ((u64)a << mbi);  // n = base | a << (N-A)  (cu:241-260)
        m0 = (u32)n;
        m1 = (u32)(n >> 32);
        u64 t = (u64)a * r1.y + r0.z;  // v = number + a * 3^f  (cu:262-278)
        w0 = (u32)t;
        t = (u64)a * r1.z + r0.w + (t >> 32);
        w1 = (u32)t;
        t = (u64)a * r1.w + r1.x + (t >> 32);
        // (0, which would read as none, and 2^80 and beyond: to the exact path)
        w2 = ((t >> 32) | r2.w) != 0 || (w0 | w1 | (u32)t) == 0 ? FULL : (u32)t;
        nlim = r2.x;
        npair = r2.y;
        na10 = a;
        nline = r2.z;
        if (n < 3 && r2.w != 2u) {  // v < n can never hold: the reference would loop forever
          atomicOr(&A.rec[nline].errors, ERR_SEED_SMALL);
          w0 = w1 = w2 = 0;
        }
      }
      qhead = (qhead + take) & (WQ - 1);
      qcount -= take;
      last = __any_sync(FULL, exhausted && qcount == 0);
      end = __all_sync(FULL, (w0 | w1 | w2) == 0 && pair == FULL && last);
      if (end) continue;
      __syncwarp();
    }
    // ---- look-ups (Step 3, cu:280-405) ----
    for (;;) {
      u32 e = 0;
#pragma unroll
      for (int i = 0; i < WGROUP; i++) {
        u32 at, fa;
        asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(at) : "r"(v0 & ((1u << CP_BITS) - 1u)), "r"(A.four), "r"(hb));
        e = lds32(at);
        asm("mad.hi.u32 %0, %1, %2, %3;" : "=r"(fa) : "r"(e & CP_F), "r"(A.p29), "r"(p3));  // p3 + 4 f
        const u32 m = lds32(fa);
        u64 w = (u64)__funnelshift_r(v0, v1, e) * m + (e >> 12);
        v0 = (u32)w;
        w = (u64)__funnelshift_r(v1, v2, e) * m + (w >> 32);
        v1 = (u32)w;
        v2 = (v2 >> (e & 31u)) * m + (u32)(w >> 32);
        asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(hb) : "r"(e & CP_HALF), "r"(A.p5), "r"(tab));
        mx = max(mx, __funnelshift_r(v1, v2, unit));
        // at a checkpoint: the hash; below n: idle
        asm("{\n\t.reg .pred p, q;\n\t.reg .u32 t;\n\t.reg .u64 v, n;\n\t"
            "and.b32 t, %3, 0x200;\n\t"
            "setp.ne.u32 p, t, 0;\n\t"
            "@p xor.b32 %2, %2, %0;\n\t"
            "mov.b64 v, {%0, %1};\n\t"
            "mov.b64 n, {%4, %5};\n\t"
            "setp.eq.and.u32 p, %6, 0, p;\n\t"
            "setp.lt.and.u64 q, v, n, p;\n\t"
            "@q mov.b32 %0, 0;\n\t"
            "@q mov.b32 %1, 0;\n\t}"
            : "+r"(v0), "+r"(v1), "+r"(hs)
            : "r"(e), "r"(n0), "r"(n1), "r"(v2));
      }
      cnt -= WGROUP;
      const bool stall = (e & 31u) == 0 && (v0 | v1 | v2) != 0;
      if (__any_sync(FULL, stall)) {
        if (stall) {  // the pair's runs, counted
          u32 v3 = 0;
          const u32 a = ctz32(v0 | (1u << 8));
          odd_run4(v0, v1, v2, v3, a, S.p3[a]);
          v0 -= 1;
          const u32 b = ctz32(v0 | 0x80000000u);
          v0 = __funnelshift_r(v0, v1, b) + 1;
          v1 = __funnelshift_r(v1, v2, b);
          v2 >>= b;
          add_carry3(v1, v2, v3, (v0 == 0) & (b != 0));
          cnt -= 4;  // (at most 39 steps)
          mx = max(mx, __funnelshift_r(v1, v2, unit));
          if (hb != tab) {
            hs ^= v0;
            if (v2 == 0 && (((u64)v1 << 32) | v0) < (((u64)n1 << 32) | n0)) v0 = v1 = 0;
          }
          hb = hb != tab ? tab : tab + (4u << CP_BITS);
        }
        __syncwarp();
      }
      const bool bad = (mx >= hi || cnt < 0) && pair != FULL;
      const u32 b = __ballot_sync(FULL, bad);
      if (__any_sync(FULL, bad)) {
        if (bad) {
          W.slow[ns + __popc(b & lanemask_lt())] = make_uint2(pair, a10);
          v0 = v1 = v2 = hs = 0;
        }
        ns += __popc(b);
        __syncwarp();
      }
      if ((v0 | v1 | v2) == 0) {  // the lane's next seed
        hash ^= hs;
        hs = 0;
        hb = tab;
        if (MULTI && nline != hline && (w0 | w1 | w2)) {  // the lane's XORs so far belong to the previous line
          if (hash) atomicXor(&A.rec[hline].hash, hash);
          hash = 0;
          hline = nline;
        }
        v0 = w0;
        v1 = w1;
        v2 = w2;
        n0 = m0;
        n1 = m1;
        const bool none = (w0 | w1 | w2) == 0;
        pair = none ? FULL : npair;
        a10 = na10;
        mx = v2 >> unit ? FULL : __funnelshift_r(v1, v2, unit);
        hi = nlim & 0xFFFFFFu;
        cnt = none ? IDLE_CNT : (int)(nlim >> 24);
        w0 = w1 = w2 = 0;
      }
      if (ns >= 32u) break;
      const u32 o = __ballot_sync(FULL, last ? pair == FULL : (w0 | w1 | w2) == 0);
      if ((int)__popc(o) >= (last ? 32 : WREFILL)) break;
    }
  }

  // ---- warp totals ----
  if (MULTI) {
    if (hash) atomicXor(&A.rec[hline].hash, hash);
  } else {
#pragma unroll
    for (u32 d = 16; d; d >>= 1) hash ^= __shfl_xor_sync(FULL, hash, d);
    if (lane == 0) atomicXor(&A.rec->hash, hash);
  }
  if (lane == 0 && warp_seeds) atomicAdd(&A.rec[MULTI ? wline : 0].seeds, (ull)warp_seeds);
}

// Lines of N >= 45 have the largest unit: it is compiled in there (2048 lines of N = 45 took 7.73 ms with
// the unit from the arguments and 7.61 so).
constexpr u32 MAX_UNIT = 16;

cudaError_t cases_win_init(cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (auto k : {k_cases_win<false, 0>, k_cases_win<true, 0>, k_cases_win<false, MAX_UNIT>, k_cases_win<true, MAX_UNIT>})
    if (!e) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CwShared));
  if (e) return e;
  return fill_once([&](bool* done) { return table_ready(g_cp_ready, done, st); },
                   [&] {
                     k_cp_tables<<<(1u << CP_BITS) / 256, 256, 0, st>>>();
                     const cudaError_t l = cudaGetLastError();
                     return l ? l : cudaStreamSynchronize(st);
                   },
                   [&] { return mark_table(g_cp_ready, st); });
}

cudaError_t launch_cases_win(const CasesArgs& a, u32 sm_count, cudaStream_t st) {
  const u32 grid = std::min(sm_count, std::max(1u, a.npairs));
  CasesArgs b = a;
  b.unit = line_unit(a.mbi + 10u);
  const auto k = b.unit == MAX_UNIT ? (b.multi ? k_cases_win<true, MAX_UNIT> : k_cases_win<false, MAX_UNIT>)
                                    : (b.multi ? k_cases_win<true, 0> : k_cases_win<false, 0>);
  k<<<grid, WWARPS * 32, sizeof(CwShared), st>>>(b);
  return cudaGetLastError();
}

}  // namespace cz
