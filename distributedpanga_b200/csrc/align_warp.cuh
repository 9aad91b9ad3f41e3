// Warp-cooperative wave extension: forward_wave / reverse_wave /
// Local_Alignment (lib/align.c:352-1576) with the 32 lanes of a warp
// updating the diagonals of a wave in parallel.
//
// Growth coordinates.  Both directions run one code: the reverse wave is the
// forward wave under x -> -x, y -> -y.  Diagonals, antidiagonals and trace
// marks negate with them, the lowest diagonal becomes the highest, and the
// visit order (forward hgh..low, reverse low..hgh) and the tie rules carry
// over unchanged; the bases are read from the reversed packed copies.  Only
// pebbles keep the caller's coordinates, for the trace-back.
//
// The sequential loop of the reference visits the diagonals of a wave from
// high to low and reads, for k, the previous wave's values at k-1, k, k+1.
// Every lane here reads those from the previous wave, so the new values equal
// the reference's.  What the reference accumulates in visit order is rebuilt:
//   besta / bestx       the wave's best; a diagonal is a record if it beats
//                       every higher diagonal and the best so far, so the
//                       last record is the highest diagonal with the best
//   lasta / trim*       the last record that passes the path-average and the
//                       trim tests, found going back through the records
//   aclip / bclip       the lowest diagonal that met A's end, the highest
//                       that met B's (what the reference keeps of them beyond
//                       the clip, mor*, is read only with reach set; the
//                       driver's specification has it 0)
//   pebbles             slot numbers only name pebbles, so they are taken in
//                       lane order from a global pool
//
// What the loop costs.  A wave step is a few hundred instructions on one warp
// with a dependent chain through it (neighbours, snake loads, best, prune):
// with many warps per SM it is bound by instruction fetch, with few by its
// latency, so both want few instructions in few places.  Hence one copy of
// the code for both directions (no direction tests inside), and:
//   * no match count: it is the number of ones among the 61 low bits of the
//     match history, taken only for a record;
//   * no trim tables: they (lib/align.c:222-268) ask whether every suffix of
//     1..30 history bits scores at least 0; lane i tests the suffix of i + 1
//     bits of the one record's history and a vote answers;
//   * clips, earlier records and pebble refills are branches off the path.
#pragma once
#include <stdint.h>
#include "align_core.cuh"
#include "align_share.cuh"

namespace pga {
namespace aln {

constexpr uint32_t FULL = 0xffffffffu;

// Pebble pool shared by all warps of a launch: bump allocation in chunks.
struct PebblePool {
  Pebble *cells;
  unsigned long long *next;  // next free pebble (global counter)
  int64_t cap;
};

// A diagonal's match history, head pebble and that pebble's mark.
struct __align__(16) RingCell {
  uint64_t T;
  int HA, HM;
};

// MurmurHash3's 32-bit finaliser (A. Appleby, public domain).
__device__ __forceinline__ uint32_t mix32(uint32_t h) {
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  return h ^ (h >> 16);
}

struct WarpWork {
  RingCell *C[2];  // waves by diagonal & (vcap - 1), in growth coordinates
  int *V[2];
  int *NA;         // next trace mark of each diagonal
  int vcap;
  uint16_t *points;
  int64_t point_cap;
  PebblePool pool;
  int64_t chunk_next, chunk_end;  // this warp's current pebble chunk (lane-uniform)
  int err;
  int64_t waves, cells;  // waves after the 0-wave, and their diagonals (lane-uniform counts)
  unsigned *smflag;      // per SM id: a warp there runs a long call (null: not kept)
  int long_waves;        // waves of one wave loop that make a call long (0: never)
  int flagged;           // this warp has flagged its SM
  long long la_cycles;   // SM cycles spent in Local_Alignment calls (lane-uniform)
  int *sm;                  // 128 words of this warp's shared memory
  const ShareTable *share;  // null: extensions are not shared
  unsigned pair;            // the call's contigs and orientation, for the table's keys
  const struct TaskChains *task;  // the task's chains, until its scouts are queued (null: none are)
};

constexpr int PEBBLE_CHUNK = 4096;

// Queues the scouts of the warp's task if warps are free for them (align.cu).
__device__ void scout_if_free(WarpWork &W);

// Reserve `cnt` consecutive pebbles for the warp (lane-uniform call).
__device__ __forceinline__ int64_t warp_pebbles(WarpWork &W, int cnt) {
  if (cnt == 0) return 0;
  if (W.chunk_next + cnt > W.chunk_end) {
    int64_t want = cnt > PEBBLE_CHUNK ? cnt : PEBBLE_CHUNK;
    unsigned long long base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(W.pool.next, (unsigned long long)want);
    base = __shfl_sync(FULL, base, 0);
    if ((int64_t)base + want > min(W.pool.cap, (int64_t)I32MAX)) {
      W.err |= ALN_ERR_CELLS;
      return -1;
    }
    W.chunk_next = (int64_t)base;
    W.chunk_end = (int64_t)base + want;
  }
  int64_t s = W.chunk_next;
  W.chunk_next += cnt;
  return s;
}

__device__ __forceinline__ int warp_excl_sum(int v, int lane) {
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(FULL, x, o);
    if (lane >= o) x += y;
  }
  return x - v;
}

// The antidiagonal of a diagonal outside the wave: below every real one.
constexpr int NO_WAVE = -2147483647 - 1;
constexpr uint32_t HIST_HI = 0x1fffffffu;  // the upper word of the history's 61 bits

// The match count of lib/align.c:663-668: ones among the last 61 history bits.
__device__ __forceinline__ int hist_ones(uint64_t t) {
  return __popc((uint32_t)t) + __popc((uint32_t)(t >> 32) & HIST_HI);
}

// A mismatch and `run` matches shifted into a history.
__device__ __forceinline__ uint64_t hist_step(uint64_t t, int run) {
  const int s = min(run, 63);
  return ((t << 1) << s) | ((1ull << s) - 1);
}

// Matching bases of 16 * N + 15 loaded ones a (from 2-bit shift sa) and b
// (from sb): 16 * N bases compared, 16 * N when all match.
template <int N>
__device__ __forceinline__ int match_loaded(const uint32_t (&a)[N + 1], int sa, const uint32_t (&b)[N + 1], int sb) {
  uint32_t w = 0;
  int o = 0;
#pragma unroll
  for (int i = N - 1; i >= 0; i--) {
    const uint32_t d = __funnelshift_l(a[i + 1], a[i], sa) ^ __funnelshift_l(b[i + 1], b[i], sb);
    if (i == N - 1 || d != 0) {
      w = d;
      o = 32 * i;
    }
  }
  return (o + __clz(w)) >> 1;
}

// The same of words q and r.  The words read may lie past the sequence's
// copy: the packed buffer has spare words at its end.
template <int N>
__device__ __forceinline__ int match_words(const uint32_t *q, int sq, const uint32_t *r, int sr) {
  uint32_t a[N + 1], b[N + 1];
#pragma unroll
  for (int i = 0; i <= N; i++) {
    a[i] = __ldg(q + i);
    b[i] = __ldg(r + i);
  }
  return match_loaded<N>(a, sq, b, sr);
}

// One extension (forward_wave or reverse_wave): its lane-uniform inputs and
// state, in growth coordinates.  Base i of a sequence in growth order is at
// x + off, and lim - x bases remain from x.
struct Wave {
  const uint32_t *pa, *pb;
  int offA, offB, limA, limB;
  int minp, maxp;
  int tspace, ave_path, dscore;
  int sg;    // 1 forward, -1 reverse
  int low, hgh, dif, cur;
  int besta, bestx, lasta, trima, trimx, trimd, trimha;
  int more;
  int line;  // the antidiagonal narrow_waves stops at
};

// Snake along diagonal k from x in rounds of 16 * N bases: stops at the first
// mismatch or a sequence's end.  Where x is outside the sequences
// (`go` false) it does not move, and no read leaves the buffers.
template <int N>
__device__ __forceinline__ int snake(const Wave &E, int x, int k, bool act, int mx, bool &go) {
  const int ia = x + E.offA, ib = x - k + E.offB;
  go = act && (mx | ia | ib) >= 0;
  int run = 0;
  if (go) {
    int r;
    do {
      const int qa = ia + run, qb = ib + run;
      r = match_words<N>(E.pa + (qa >> 4), (qa & 15) << 1, E.pb + (qb >> 4), (qb & 15) << 1);
      run += r;
    } while (r == 16 * N && run < mx);
    run = min(run, mx);
  }
  return run;
}

// Which end a snake that could go no further met: true B's (checked first by
// the reference's byte loop), false A's.  x is the snake's start; one that
// starts outside the sequences counts as meeting an end, B's if y is outside.
__device__ __forceinline__ bool met_b(const Wave &E, int x, int k, bool go) {
  const int ra = E.limA - x, rb = E.limB - x + k;
  return go ? rb <= ra : (x - k + E.offB < 0 || rb < (E.sg > 0 ? 0 : 1));
}

// The trim test on a record's history (New_Align_Spec's tables,
// lib/align.c:222-268, with match score 1000 - dscore and mismatch -dscore):
// every suffix of 1..30 bits scores at least 0.  The tables cut the 30 bits
// at TRIM_LEN: TABLE[low 15] >= 0 is the suffixes up to 15 bits,
// TABLE[high 15] + SCORE[low 15] >= 0 the longer ones.
struct TrimTest {
  uint32_t mask;  // this lane's suffix
  int need;       // matches it needs
  __device__ __forceinline__ TrimTest(int dscore) {
    const int lane = threadIdx.x & 31;
    mask = lane < 2 * TRIM_LEN ? (2u << lane) - 1u : 0u;
    need = lane < 2 * TRIM_LEN ? ((lane + 1) * dscore + 999) / 1000 : 0;
  }
  __device__ __forceinline__ bool operator()(uint64_t t) const {
    return __all_sync(FULL, __popc((uint32_t)t & mask) >= need);
  }
};

// The trace marks the lanes' snakes passed: one pebble each unless the path
// has it already (hm).  next / end: the warp's pebble chunk.  Returns false
// when the pool is full.
__device__ __forceinline__ bool drop_pebbles(const PebblePool &pool, const Wave &E, bool act, int k, int x, int dif, int &ha,
                                             int &hm, int &nak, int &next, int &end) {
  const int lane = threadIdx.x & 31;
  bool cross = act && x >= nak;
#pragma unroll 1
  do {
    const bool mk = cross && hm < nak;
    const uint32_t mb = __ballot_sync(FULL, mk);
    const int cnt = __popc(mb);
    if (next + cnt > end) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(pool.next, (unsigned long long)PEBBLE_CHUNK);
      base = __shfl_sync(FULL, base, 0);
      // pebble numbers are int
      if ((int64_t)base + PEBBLE_CHUNK > min(pool.cap, (int64_t)I32MAX)) return false;
      next = (int)base;
      end = next + PEBBLE_CHUNK;
    }
    if (mk) {
      const int s = next + __popc(mb & ((1u << lane) - 1u));
      *reinterpret_cast<int4 *>(pool.cells + s) = make_int4(ha, E.sg * k, dif, E.sg * nak);
      ha = s;
      hm = nak;
    }
    next += cnt;
    if (cross) nak += E.tspace;
    cross = cross && x >= nak;
  } while (__any_sync(FULL, cross));
  return true;
}

// The records before the one on diagonal kr (the higher diagonals; `passed`:
// the later ones already gave lasta), back to the last that also passes the
// trim test.  carry: the best before the wave.
__device__ __forceinline__ void earlier_records(Wave &S, int &lasta, const TrimTest &trim, bool act, int k, int c,
                                                uint64_t b, int ha, int dif, int carry, int kr, bool passed) {
  const bool good = act && c > carry && hist_ones(b) >= S.ave_path;
  while (__any_sync(FULL, good && k > kr)) {  // else none of them passes
    const bool cand = act && k > kr && c > carry;
    const int rc = __reduce_max_sync(FULL, cand ? c : NO_WAVE);
    kr = __reduce_max_sync(FULL, cand && c == rc ? k : NO_WAVE);
    const int L = __ffs(__ballot_sync(FULL, act && k == kr)) - 1;
    const uint64_t t = __shfl_sync(FULL, b, L);
    if (hist_ones(t) < S.ave_path) continue;
    if (!passed) lasta = rc;
    passed = true;
    if (trim(t)) {
      S.trima = rc;
      S.trimx = (rc + kr) >> 1;
      S.trimd = dif;
      S.trimha = __shfl_sync(FULL, ha, L);
      return;
    }
  }
}

// The records of one pass over up to 32 diagonals (lane's diagonal k at c
// with history b), none of them above the pass: the wave's best, and the last
// record that passes the path-average test and the last that also passes the
// trim test.
__device__ __forceinline__ void take_records(Wave &S, int &besta, int &lasta, const TrimTest &trim, bool act, int k,
                                             int c, uint64_t b, int ha, int dif) {
  const int rc = __reduce_max_sync(FULL, act ? c : NO_WAVE);
  if (rc <= besta) return;
  const int kr = __reduce_max_sync(FULL, act && c == rc ? k : NO_WAVE);
  const int L = __ffs(__ballot_sync(FULL, act && k == kr)) - 1;
  const uint64_t t = __shfl_sync(FULL, b, L);
  const bool pass = hist_ones(t) >= S.ave_path, tip = trim(t);
  S.bestx = (rc + kr) >> 1;
  if (pass) lasta = rc;
  if (pass && tip) {
    S.trima = rc;
    S.trimx = (rc + kr) >> 1;
    S.trimd = dif;
    S.trimha = __shfl_sync(FULL, ha, L);
  } else
    earlier_records(S, lasta, trim, act, k, c, b, ha, dif, besta, kr, pass);
  besta = rc;
}

// Whether the furthest path can still grow (neither sequence's end reached).
__device__ __forceinline__ int can_grow(const Wave &S, int besta) {
  return S.limB - besta + S.bestx != 0 && S.limA - S.bestx != 0 ? 1 : 0;
}

// What an extension shares: its record and last entry (-1: none), and the
// entry it joined (-1: none), with its best diagonal's head pebble there (the
// path most likely comes through that one).
struct Sharing {
  int rec, last, joined, guess;
  int from;   // the extension's first antidiagonal
  bool full;  // no room for more entries
};

// The first multiple of SHARE_LINE above antidiagonal a.
__device__ __forceinline__ int next_line(int a) { return (a & ~(SHARE_LINE - 1)) + SHARE_LINE; }

// A narrow wave, in the ring, whose best crossed a line (`way`: the pair,
// orientation and direction): joins the extension whose wave there was the
// same (returned), or enters it.
__device__ __noinline__ bool cross_line(const WarpWork &W, const Wave &wave, unsigned way, Sharing &io) {
  const ShareTable &X = *W.share;
  Sharing *S = &io;
  const int lane = threadIdx.x & 31;
  const int low = wave.low, hgh = wave.hgh, besta = wave.besta, bestx = wave.bestx, lasta = wave.lasta;
  const int dif = wave.dif, next = (int)W.chunk_next;
  if (besta - S->from < SHARE_MIN) return false;
  const int k = low + ((lane - low) & 31), vi = k & (W.vcap - 1);
  const bool live = k <= hgh;
  int V = NO_WAVE, HA = -1, HM = 0, NA = 0;
  uint64_t T = 0;
  if (live) {
    const RingCell c = W.C[wave.cur][vi];
    V = W.V[wave.cur][vi];
    NA = W.NA[vi];
    T = c.T;
    HA = c.HA;
    HM = c.HM;
  }
  // which diagonals have the same head pebble: the first lane with this one's
  const int pat = __ffs(__match_any_sync(FULL, live ? HA : -2 - lane)) - 1;
  // the state's key (the multipliers are the golden ratio's and a prime of xxHash)
  const uint32_t tl = (uint32_t)T, th = (uint32_t)(T >> 32) & HIST_HI;
  const uint32_t a = mix32(V + 0x9e3779b9u * (lane + 1)) + mix32(tl ^ 0x7f4a7c15u), b = mix32(th + HM) + mix32(NA ^ tl ^ pat << 16);
  const uint32_t h1 = __reduce_xor_sync(FULL, live ? mix32(a + 31 * b) : 0);
  const uint32_t h2 = __reduce_add_sync(FULL, live ? mix32(b ^ (a * 0x27d4eb2fu)) : 0);
  const uint32_t u = mix32(besta + mix32(lasta + mix32(bestx + mix32(way))));
  const unsigned long long key = ((unsigned long long)mix32(h1 + u) << 32 | mix32(h2 ^ (u + mix32(low + 37 * hgh)))) | 1;
  int val = -2;
  unsigned at = 0;
  if (lane == 0) {
    at = (unsigned)(key >> 20) & X.mask;
    for (int probe = 0; probe < SHARE_PROBES; probe++, at = (at + 1) & X.mask) {
      const unsigned long long old = atomicCAS(&X.keys[at], 0ull, key);
      if (old == 0) {
        val = -3;  // ours to write
        break;
      }
      if (old == key) {
        for (int poll = 0; poll < SHARE_POLLS && (val = *(volatile int *)&X.vals[at]) == -1; poll++) __nanosleep(100);
        break;
      }
    }
  }
  val = __shfl_sync(FULL, val, 0);
  if (val == -3) {
    int e = -1, r = S->rec;
    if (lane == 0) {
      e = (int)min(atomicAdd(X.nentry, 1u), (unsigned)X.entry_cap);
      if (e < X.entry_cap && r < 0) r = (int)min(atomicAdd(X.nrec, 1u), (unsigned)X.rec_cap);
      if (e >= X.entry_cap || r >= X.rec_cap) {
        e = -1;
        *(volatile int *)&X.vals[at] = -2;
      }
    }
    e = __shfl_sync(FULL, e, 0);
    r = __shfl_sync(FULL, r, 0);
    if (e < 0) {
      S->full = true;
      return false;
    }
    ShareEntry &E = X.entries[e];
    if (lane == 0) {
      if (S->rec < 0) X.recs[r].status = 0;
      E.rec = r;
      E.prev = S->last;
      E.low = low;
      E.hgh = hgh;
      E.besta = besta;
      E.bestx = bestx;
      E.lasta = lasta;
      E.dif = dif;
      E.mark = next;
      E.way = way;
      E.kind = SHARE_NONE;
    }
    E.V[lane] = V;
    E.HA[lane] = live ? HA : -1;
    E.HM[lane] = HM;
    E.pat[lane] = pat;
    E.NA[lane] = NA;
    E.T[lane] = T;
    S->rec = r;
    S->last = e;
    __threadfence();
    __syncwarp();
    if (lane == 0) *(volatile int *)&X.vals[at] = e;
    return false;
  }
  if (val < 0) return false;
  const ShareEntry &E = X.entries[val];
  __threadfence();
  bool same = __ldcg(&E.way) == way && __ldcg(&E.low) == low && __ldcg(&E.hgh) == hgh && __ldcg(&E.besta) == besta &&
              __ldcg(&E.bestx) == bestx && __ldcg(&E.lasta) == lasta;
  if (live)
    same = same && __ldcg(&E.V[lane]) == V && __ldcg(&E.HM[lane]) == HM && __ldcg(&E.NA[lane]) == NA &&
           __ldcg(&E.pat[lane]) == pat &&
           ((__ldcg(&E.T[lane]) ^ T) & ((1ull << 61) - 1)) == 0;
  if (!__all_sync(FULL, same)) return false;
  S->joined = val;
  S->guess = __shfl_sync(FULL, HA, (2 * bestx - besta) & 31);
  return true;
}

// ---------------------------------------------------------------------------
// Narrow waves, at most 31 diagonals: diagonal k lives in lane k mod 32, its
// state in registers, the previous wave's neighbours come by shuffle.  The
// free lane between the window's ends (like every lane outside it) holds
// NO_WAVE, so the neighbours of the ends need no range test.
//
// A long alignment is one warp's chain of these steps, so the step is laid
// out along its critical path: neighbours -> start points -> sequence words
// -> snakes -> the wave's best -> the next window.  The wave's pebbles and
// its record's tests are not on it: they are settled in the next step, while
// that step's sequence words are on their way, before the loop's end
// conditions are tested and anything of the new wave is kept.
//
// Runs until the loop ends, the next wave does not fit, the best crosses
// `line`, or the wave count reaches `stop`.  Returns 1 when the pebble pool is
// full.
//
// R: 16 * R bases are compared per round.  64 where the loop's length counts
// (a second round's words are another trip to the cache); 32 in the builds
// with many resident warps, whose limit is fetching their instructions
// (2 x 200 Mbp repeat-rich: pair phase 201 -> 196 ms).
// ---------------------------------------------------------------------------
constexpr int NARROW = 31;
constexpr int PAST_MAX = (1 << 26) - 1;  // a best further past than this takes the general record search

template <int R>
__device__ __noinline__ int narrow_waves(WarpWork &W, Wave &io, int stop) {
  const int lane = threadIdx.x & 31;
  const int lup = (lane + 1) & 31, ldn = (lane - 1) & 31;
  Wave S = io;
  const PebblePool pool = W.pool;
  const TrimTest trim(S.dscore);
  const int vmask = W.vcap - 1;
  int next = (int)W.chunk_next, end = (int)W.chunk_end;
  int ncells = 0;
  int low = S.low, hgh = S.hgh, dif = S.dif, besta = S.besta, lasta = S.lasta;
  const int line = S.line;

  // the last wave: lane's diagonal kw (if live), its furthest x, what came with it
  int V = NO_WAVE, HA = -1, HM = 0, NA = 0, X = 0, kw = low + ((lane - low) & 31);
  bool live = false;
  uint64_t T = 0;
  // its record, if any: the best rc on diagonal kr, past the best before it
  int rc = besta, kr = 0, carry = besta;
  if (kw <= hgh) {
    const RingCell c = W.C[S.cur][kw & vmask];
    V = W.V[S.cur][kw & vmask];
    NA = W.NA[kw & vmask];
    T = c.T;
    HA = c.HA;
    HM = c.HM;
  }
  // the last wave's pebbles and record; once done, doing it again changes nothing
  auto settle = [&]() {
    if (__any_sync(FULL, live && X >= NA) && !drop_pebbles(pool, S, live, kw, X, dif, HA, HM, NA, next, end)) return false;
    const int L = kr & 31;
    const uint64_t t = __shfl_sync(FULL, T, L);
    const int hr = __shfl_sync(FULL, HA, L);
    const bool tip = trim(t), rec = rc > carry, pass = rec && hist_ones(t) >= S.ave_path;
    if (rec) S.bestx = (rc + kr) >> 1;
    if (pass) lasta = rc;
    if (pass && tip) {
      S.trima = rc;
      S.trimx = (rc + kr) >> 1;
      S.trimd = dif;
      S.trimha = hr;
    } else if (rec)
      earlier_records(S, lasta, trim, live, kw, (X << 1) - kw, T, HA, dif, carry, kr, pass);
    carry = rc;
    return true;
  };
  bool full = false;
  while (true) {
    const int nlow = max(low - 1, S.minp), nhgh = min(hgh + 1, S.maxp);  // a window end is never past its border
    const int wide = nhgh - nlow;
    const int p = (lane - nlow) & 31, k = nlow + p;
    const bool act = p <= wide;

    // the furthest point each diagonal starts from
    const int vup = __shfl_sync(FULL, V, lup), vdn = __shfl_sync(FULL, V, ldn);
    const bool up = vup > max(V, vdn), dn = !up && vdn > V;
    const int x = ((up ? vup + 1 : (dn ? vdn + 1 : V + 2)) + k) >> 1;
    const int mx = min(S.limA - x, S.limB - x + k);
    const int ia = x + S.offA, ib = x - k + S.offB;
    const bool go = act && (mx | ia | ib) >= 0;
    uint32_t a[R + 1], b[R + 1];
    {
      const uint32_t *qa = S.pa + (go ? ia >> 4 : 0), *qb = S.pb + (go ? ib >> 4 : 0);
#pragma unroll
      for (int i = 0; i <= R; i++) {
        a[i] = __ldg(qa + i);
        b[i] = __ldg(qb + i);
      }
    }

    if (!settle()) {
      full = true;
      break;
    }
    if (!(S.more && lasta >= besta - TRIM_MLAG && low <= hgh && wide < NARROW && dif < stop && besta < line)) break;
    dif += 1;
    ncells += wide + 1;

    // what comes with the start points; a new end diagonal copies its
    // neighbour's trace mark
    const int sl = up ? lup : (dn ? ldn : lane);
    const int nlo = __shfl_sync(FULL, NA, low & 31), nhi = __shfl_sync(FULL, NA, hgh & 31);
    HA = __shfl_sync(FULL, HA, sl);
    HM = __shfl_sync(FULL, HM, sl);
    T = __shfl_sync(FULL, T, sl);
    NA = k < low ? nlo : (k > hgh ? nhi : NA);

    // snakes: 16 * R bases, then 32 per round
    int run = 0;
    if (go) {
      run = match_loaded<R>(a, (ia & 15) << 1, b, (ib & 15) << 1);
      if (run == 16 * R) {
        int r;
        do {
          const int qa = min(ia + run, ia + mx), qb = min(ib + run, ib + mx);
          r = match_words<2>(S.pa + (qa >> 4), (qa & 15) << 1, S.pb + (qb >> 4), (qb & 15) << 1);
          run += r;
        } while (r == 32 && run < mx);
      }
      run = min(run, mx);
    }
    const uint32_t hits = __ballot_sync(FULL, act && (!go || run == mx));
    X = x + run;
    const int c = (X << 1) - k;
    // the wave's best: how far a diagonal is past the best so far, then the
    // highest such diagonal, in one reduction
    const int past = min(max(c - besta, 0), PAST_MAX);
    const int key = __reduce_max_sync(FULL, act ? (past << 5) + p : 0);
    T = hist_step(T, run);
    live = act;
    kw = k;
    carry = besta;
    rc = besta + (key >> 5);
    kr = nlow + (key & 31);
    low = nlow;
    hgh = nhgh;
    if (key >= (PAST_MAX << 5)) {
      rc = __reduce_max_sync(FULL, act ? c : NO_WAVE);
      kr = __reduce_max_sync(FULL, act && c == rc ? k : NO_WAVE);
    }
    if (hits) {
      // snakes that reached a sequence's end clip the window
      const bool hit = hits >> lane & 1, hb = met_b(S, x, k, go);
      const int ka = __reduce_min_sync(FULL, hit && !hb ? k : I32MAX);
      const int kb = __reduce_max_sync(FULL, hit && hb ? k : NO_WAVE);
      if (rc > besta) S.bestx = (rc + kr) >> 1;
      S.more = can_grow(S, rc);
      if (ka != I32MAX) hgh = ka - 1;
      if (kb != NO_WAVE) low = kb + 1;
    }
    besta = rc;
    // WAVE_LAG pruning from either end, between the clipped ends
    const uint32_t keep = __ballot_sync(FULL, k >= low && k <= hgh && c >= besta - WAVE_LAG);
    const uint32_t kept = __funnelshift_r(keep, keep, nlow & 31);  // bit q: diagonal nlow + q
    low = nlow + __clz(__brev(kept));                              // none: low = nlow + 32, above hgh = nlow - 1
    hgh = nlow + 31 - __clz(kept);
    V = k >= low && k <= hgh ? c : NO_WAVE;
  }
  W.waves += dif - S.dif;
  W.cells += ncells;
  W.chunk_next = next;
  W.chunk_end = end;
  if (full) {
    W.err |= ALN_ERR_CELLS;
    return 1;
  }
  // (the diagonals of [low, hgh] are where they were in the last wave)
  if (kw >= low && kw <= hgh) {
    W.V[S.cur][kw & vmask] = V;
    W.C[S.cur][kw & vmask] = RingCell{T, HA, HM};
    W.NA[kw & vmask] = NA;
  }
  __syncwarp();
  S.low = low;
  S.hgh = hgh;
  S.dif = dif;
  S.besta = besta;
  S.lasta = lasta;
  io = S;
  return 0;
}

// ---------------------------------------------------------------------------
// Block waves, at most J * 31 diagonals: lane l holds the J diagonals of one
// aligned block, blocks dealt to the lanes in turn, all state in registers;
// only the blocks' edges come by shuffle.  The waves past an alignment's end
// run here: they widen by two diagonals per step until the trim lag ends the
// loop, nearly all snakes stopping at once, so a step is the fixed work per
// diagonal; a lane's J independent diagonals overlap in it where passes of 32
// through memory would follow one another.  Runs until the loop ends, the
// window narrows to BLOCK_OUT diagonals or no longer fits, or the wave count
// reaches `stop`.
// ---------------------------------------------------------------------------
constexpr int BLOCK = 4;
constexpr int BLOCK_OUT = 20;

// v[j] for a per-lane index j < J, without local memory
template <int J, class T>
__device__ __forceinline__ T pick(const T (&v)[J], int j) {
  T r = v[0];
#pragma unroll
  for (int q = 1; q < J; q++)
    if (j == q) r = v[q];
  return r;
}

template <int J>
__device__ __noinline__ int block_waves(WarpWork &W, Wave &io, int stop) {
  constexpr int LG = J == 2 ? 1 : 2;
  static_assert(J == 1 << LG, "J is 2 or 4");
  const int lane = threadIdx.x & 31;
  const int lup = (lane + 1) & 31, ldn = (lane - 1) & 31;
  Wave S = io;
  const PebblePool pool = W.pool;
  const TrimTest trim(S.dscore);
  const int vmask = W.vcap - 1;
  int next = (int)W.chunk_next, end = (int)W.chunk_end;
  int ncells = 0;
  int low = S.low, hgh = S.hgh, dif = S.dif, besta = S.besta, lasta = S.lasta;
  bool full = false;

  int V[J], HA[J], HM[J], NA[J];
  uint64_t T[J];
  int kw = ((low >> LG) + ((lane - (low >> LG)) & 31)) << LG;  // the lane's first diagonal
#pragma unroll
  for (int j = 0; j < J; j++) {
    const int k = kw + j;
    V[j] = NO_WAVE;
    HA[j] = -1;
    HM[j] = NA[j] = 0;
    T[j] = 0;
    if (k >= low && k <= hgh) {
      const RingCell c = W.C[S.cur][k & vmask];
      V[j] = W.V[S.cur][k & vmask];
      NA[j] = W.NA[k & vmask];
      T[j] = c.T;
      HA[j] = c.HA;
      HM[j] = c.HM;
    }
  }
  while (true) {
    const int nlow = max(low - 1, S.minp), nhgh = min(hgh + 1, S.maxp);
    const int wide = nhgh - nlow;
    if (!(S.more && lasta >= besta - TRIM_MLAG && low <= hgh && wide < J * NARROW && wide >= BLOCK_OUT && dif < stop))
      break;
    dif += 1;
    ncells += wide + 1;
    const int bl = nlow >> LG;
    kw = (bl + ((lane - bl) & 31)) << LG;

    // start points and what comes with them
    const int nlo = __shfl_sync(FULL, pick<J>(NA, low & (J - 1)), (low >> LG) & 31);
    const int nhi = __shfl_sync(FULL, pick<J>(NA, hgh & (J - 1)), (hgh >> LG) & 31);
    const int vup = __shfl_sync(FULL, V[0], lup), vdn = __shfl_sync(FULL, V[J - 1], ldn);
    const int hau = __shfl_sync(FULL, HA[0], lup), had = __shfl_sync(FULL, HA[J - 1], ldn);
    const int hmu = __shfl_sync(FULL, HM[0], lup), hmd = __shfl_sync(FULL, HM[J - 1], ldn);
    const uint64_t tu = __shfl_sync(FULL, T[0], lup), td = __shfl_sync(FULL, T[J - 1], ldn);
    int x[J], run[J], mx[J];
    bool act[J], go[J];
    {
      int ha[J], hm[J];
      uint64_t t[J];
#pragma unroll
      for (int j = 0; j < J; j++) {
        const int jp = j < J - 1 ? j + 1 : j, jm = j > 0 ? j - 1 : j, k = kw + j;
        const int ap = j < J - 1 ? V[jp] : vup, am = j > 0 ? V[jm] : vdn;
        const bool up = ap > max(V[j], am), dn = !up && am > V[j];
        x[j] = ((up ? ap + 1 : (dn ? am + 1 : V[j] + 2)) + k) >> 1;
        ha[j] = up ? (j < J - 1 ? HA[jp] : hau) : (dn ? (j > 0 ? HA[jm] : had) : HA[j]);
        hm[j] = up ? (j < J - 1 ? HM[jp] : hmu) : (dn ? (j > 0 ? HM[jm] : hmd) : HM[j]);
        t[j] = up ? (j < J - 1 ? T[jp] : tu) : (dn ? (j > 0 ? T[jm] : td) : T[j]);
        act[j] = k >= nlow && k <= nhgh;
        NA[j] = k < low ? nlo : (k > hgh ? nhi : NA[j]);
      }
#pragma unroll
      for (int j = 0; j < J; j++) {
        HA[j] = ha[j];
        HM[j] = hm[j];
        T[j] = t[j];
      }
    }

    // snakes: 32 bases each, then the few that go on
    bool more32 = false;
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int k = kw + j, ia = x[j] + S.offA, ib = x[j] - k + S.offB;
      mx[j] = min(S.limA - x[j], S.limB - x[j] + k);
      go[j] = act[j] && (mx[j] | ia | ib) >= 0;
      run[j] = 0;
      if (go[j]) run[j] = match_words<2>(S.pa + (ia >> 4), (ia & 15) << 1, S.pb + (ib >> 4), (ib & 15) << 1);
      more32 |= run[j] == 32 && mx[j] > 32;
    }
    if (more32) {
#pragma unroll 1
      for (int j = 0; j < J; j++) {
        int t = pick<J>(run, j);
        const int xj = pick<J>(x, j), m = pick<J>(mx, j), ia = xj + S.offA, ib = xj - kw - j + S.offB;
        for (int r = t; r == 32 && t < m; t += r)
          r = match_words<2>(S.pa + ((ia + t) >> 4), ((ia + t) & 15) << 1, S.pb + ((ib + t) >> 4),
                             ((ib + t) & 15) << 1);
#pragma unroll
        for (int q = 0; q < J; q++)
          if (q == j) run[q] = t;
      }
    }

    bool hit = false, cross = false;
    int key = 0, c[J];
#pragma unroll
    for (int j = 0; j < J; j++) {
      const int k = kw + j;
      run[j] = min(run[j], max(mx[j], 0));
      hit |= act[j] && (!go[j] || run[j] == mx[j]);
      T[j] = hist_step(T[j], run[j]);
      x[j] += run[j];
      c[j] = (x[j] << 1) - k;
      cross |= act[j] && x[j] >= NA[j];
      const int past = min(max(c[j] - besta, 0), PAST_MAX >> 2);
      if (act[j]) key = max(key, (past << 7) + (k - nlow));
    }
    if (__any_sync(FULL, cross)) {
#pragma unroll 1
      for (int j = 0; j < J; j++) {  // (one copy of the loop: few diagonals cross a mark)
        int ha = pick<J>(HA, j), hm = pick<J>(HM, j), nak = pick<J>(NA, j);
        const int k = kw + j;
        full |= !drop_pebbles(pool, S, k >= nlow && k <= nhgh, k, pick<J>(x, j), dif, ha, hm, nak, next, end);
#pragma unroll
        for (int q = 0; q < J; q++)
          if (q == j) {
            HA[q] = ha;
            HM[q] = hm;
            NA[q] = nak;
          }
      }
      if (full) break;
    }

    // the record: the highest diagonal of the wave's best
    key = __reduce_max_sync(FULL, key);
    if (key >= 128) {
      const int carry = besta;
      int rc = besta + (key >> 7), kr = nlow + (key & 127);
      if (key >= (PAST_MAX >> 2) << 7) {
        int m = NO_WAVE, mk = NO_WAVE;
#pragma unroll
        for (int j = 0; j < J; j++) m = max(m, act[j] ? c[j] : NO_WAVE);
        rc = __reduce_max_sync(FULL, m);
#pragma unroll
        for (int j = 0; j < J; j++)
          if (act[j] && c[j] == rc) mk = kw + j;
        kr = __reduce_max_sync(FULL, mk);
      }
      besta = rc;
      S.bestx = (rc + kr) >> 1;
      bool passed = false;
      while (true) {
        const int L = (kr >> LG) & 31, q = kr & (J - 1);
        const uint64_t t = __shfl_sync(FULL, pick<J>(T, q), L);
        if (hist_ones(t) >= S.ave_path) {
          if (!passed) lasta = rc;
          passed = true;
          if (trim(t)) {
            S.trima = rc;
            S.trimx = (rc + kr) >> 1;
            S.trimd = dif;
            S.trimha = __shfl_sync(FULL, pick<J>(HA, q), L);
            break;
          }
        }
        // an earlier record (a higher diagonal), if one could pass
        bool good = false;
        int m = NO_WAVE, mk = NO_WAVE;
#pragma unroll
        for (int j = 0; j < J; j++)
          if (act[j] && kw + j > kr && c[j] > carry) {
            good |= hist_ones(T[j]) >= S.ave_path;
            m = max(m, c[j]);
          }
        if (!__any_sync(FULL, good)) break;
        rc = __reduce_max_sync(FULL, m);
#pragma unroll
        for (int j = 0; j < J; j++)
          if (act[j] && kw + j > kr && c[j] == rc) mk = kw + j;
        kr = __reduce_max_sync(FULL, mk);
      }
    }

    low = nlow;
    hgh = nhgh;
    if (__any_sync(FULL, hit)) {
      // snakes that reached a sequence's end clip the window
      int ka = I32MAX, kb = NO_WAVE;
#pragma unroll
      for (int j = 0; j < J; j++)
        if (act[j] && (!go[j] || run[j] == mx[j])) {
          if (met_b(S, x[j] - run[j], kw + j, go[j])) kb = max(kb, kw + j);
          else ka = min(ka, kw + j);
        }
      ka = __reduce_min_sync(FULL, ka);
      kb = __reduce_max_sync(FULL, kb);
      S.more = can_grow(S, besta);
      if (ka != I32MAX) hgh = ka - 1;
      if (kb != NO_WAVE) low = kb + 1;
    }
    // WAVE_LAG pruning from either end, between the clipped ends
    int kmin = I32MAX, kmax = NO_WAVE;
#pragma unroll
    for (int j = 0; j < J; j++)
      if (kw + j >= low && kw + j <= hgh && c[j] >= besta - WAVE_LAG) {
        kmin = min(kmin, kw + j);
        kmax = max(kmax, kw + j);
      }
    kmin = __reduce_min_sync(FULL, kmin);
    kmax = __reduce_max_sync(FULL, kmax);
    if (kmin <= kmax) {
      low = kmin;
      hgh = kmax;
    } else
      hgh = low - 1;
#pragma unroll
    for (int j = 0; j < J; j++) V[j] = kw + j >= low && kw + j <= hgh ? c[j] : NO_WAVE;
  }
  W.waves += dif - S.dif;
  W.cells += ncells;
  W.chunk_next = next;
  W.chunk_end = end;
  if (full) {
    W.err |= ALN_ERR_CELLS;
    return 1;
  }
#pragma unroll
  for (int j = 0; j < J; j++) {
    const int k = kw + j;
    if (k >= low && k <= hgh) {
      W.V[S.cur][k & vmask] = V[j];
      W.C[S.cur][k & vmask] = RingCell{T[j], HA[j], HM[j]};
      W.NA[k & vmask] = NA[j];
    }
  }
  __syncwarp();
  S.low = low;
  S.hgh = hgh;
  S.dif = dif;
  S.besta = besta;
  S.lasta = lasta;
  io = S;
  return 0;
}

// ---------------------------------------------------------------------------
// Wide waves: the ring in memory (L1-resident at the widths that occur), 32
// diagonals per pass from the highest down.  Runs until the loop ends, the
// window has at most `least` diagonals, or the wave count reaches `stop`.
// ---------------------------------------------------------------------------
__device__ __noinline__ int wide_waves(WarpWork &W, Wave &io, int stop, int least) {
  const int lane = threadIdx.x & 31;
  Wave S = io;
  const TrimTest trim(S.dscore);
  const int vmask = W.vcap - 1;
  int next = (int)W.chunk_next, end = (int)W.chunk_end;
  const int dif0 = S.dif;
  int ncells = 0, err = 0;
  while (S.more && S.lasta >= S.besta - TRIM_MLAG) {
    if (S.hgh - S.low < least || S.dif >= stop) break;
    if (S.hgh - S.low + 5 > W.vcap) {
      err = ALN_ERR_VCAP;
      break;
    }
    const RingCell *Co = W.C[S.cur];
    RingCell *Cn = W.C[S.cur ^ 1];
    int *Vo = W.V[S.cur], *Vn = W.V[S.cur ^ 1];
    if (lane == 0) {
      // the diagonals just outside, and the trace marks of grown ends
      const bool glo = S.low > S.minp, ghi = S.hgh < S.maxp;
      Vo[(S.low - 1) & vmask] = Vo[(S.hgh + 1) & vmask] = NO_WAVE;
      if (glo) {
        Vo[(S.low - 2) & vmask] = NO_WAVE;
        W.NA[(S.low - 1) & vmask] = W.NA[S.low & vmask];
      }
      if (ghi) {
        Vo[(S.hgh + 2) & vmask] = NO_WAVE;
        W.NA[(S.hgh + 1) & vmask] = W.NA[S.hgh & vmask];
      }
    }
    __syncwarp();
    const int low = S.low - (S.low > S.minp ? 1 : 0), hgh = S.hgh + (S.hgh < S.maxp ? 1 : 0);
    S.low = low;
    S.hgh = hgh;
    S.dif += 1;
    ncells += hgh - low + 1;
    int ka = I32MAX, kb = NO_WAVE;
    for (int top = hgh; top >= low; top -= 32) {
      const int k = top - lane, vi = k & vmask;
      const bool act = k >= low;
      int c = 0, ha = -1, hm = 0, nak = 0, x = 0, mx = 0;
      uint64_t t0 = 0;
      if (act) {
        const int vup = Vo[(k + 1) & vmask], v = Vo[vi], vdn = Vo[(k - 1) & vmask];
        nak = W.NA[vi];
        const bool up = vup > max(v, vdn), dn = !up && vdn > v;
        c = up ? vup + 1 : (dn ? vdn + 1 : v + 2);
        const RingCell q = Co[(k + (up ? 1 : (dn ? -1 : 0))) & vmask];
        t0 = q.T;
        ha = q.HA;
        hm = q.HM;
        x = (c + k) >> 1;
        mx = min(S.limA - x, S.limB - x + k);
      }
      // Most snakes of a wide wave end within 16 bases and few of its passes
      // cross a trace mark: one word per round and pebbles only where there
      // are some are the fewer instructions (2 x 200 Mbp repeat-rich: pair
      // phase 196 -> 179 ms, 2 x 41 kbp 10.2 -> 9.3).
      bool go;
      const int run = snake<1>(S, x, k, act, mx, go);
      const bool hit = act && (!go || run == mx);
      const uint64_t b = hist_step(t0, run);
      x += run;
      c = (x << 1) - k;
      if (__any_sync(FULL, act && x >= nak) && !drop_pebbles(W.pool, S, act, k, x, S.dif, ha, hm, nak, next, end)) {
        err = ALN_ERR_CELLS;
        break;
      }
      if (act) {
        Vn[vi] = c;
        Cn[vi] = RingCell{b, ha, hm};
        W.NA[vi] = nak;
      }
      take_records(S, S.besta, S.lasta, trim, act, k, c, b, ha, S.dif);
      if (__any_sync(FULL, hit)) {
        const bool hb = met_b(S, x - run, k, go);
        ka = min(ka, __reduce_min_sync(FULL, hit && !hb ? k : I32MAX));
        kb = max(kb, __reduce_max_sync(FULL, hit && hb ? k : NO_WAVE));
      }
    }
    if (err) break;
    S.cur ^= 1;
    __syncwarp();
    if (ka != I32MAX || kb != NO_WAVE) {
      S.more = can_grow(S, S.besta);
      if (ka != I32MAX) S.hgh = ka - 1;
      if (kb != NO_WAVE) S.low = kb + 1;
    }
    // WAVE_LAG pruning from either end
    if (S.hgh >= S.low) {
      const int n = S.besta - WAVE_LAG;
      int nh = S.low - 1;
      for (int top = S.hgh; top >= S.low; top -= 32) {
        const int k = top - lane;
        const uint32_t keep = __ballot_sync(FULL, k >= S.low && Vn[k & vmask] >= n);
        if (keep) {
          nh = top - __ffs(keep) + 1;
          break;
        }
      }
      S.hgh = nh;
      for (int bot = S.low; bot <= nh; bot += 32) {
        const int k = bot + lane;
        const uint32_t keep = __ballot_sync(FULL, k <= nh && Vn[k & vmask] >= n);
        if (keep) {
          S.low = bot + __ffs(keep) - 1;
          break;
        }
      }
    }
  }
  __syncwarp();
  W.chunk_next = next;
  W.chunk_end = end;
  W.waves += S.dif - dif0;
  W.cells += ncells;
  if (err) {
    W.err |= err;
    return 1;
  }
  io = S;
  return 0;
}

// A trace being walked back from its tip: intervals (diffs, b-delta) in the
// free end of the trace buffer, last first -- forward ones down from the
// buffer's top, reverse ones up from its bottom.
struct TraceWalk {
  bool fwd, inner;   // inner: the reverse path of a call whose forward path has a trace
  int sg, mida, tspace, aoff;
  int64_t room;      // intervals the free end holds
  int64_t base, lim; // the extension's first pebble, and a bound of its pebbles
  int64_t n;         // intervals so far
  int last;          // the extension's entries not yet crossed, going back
  int start;         // the diagonal the path starts on
  // the interval of a reverse path that ends inside the forward path's first
  // one, which it extends
  int jd, jb;

  __device__ __forceinline__ uint32_t *slot(const WarpWork &W, int64_t i) const {
    return reinterpret_cast<uint32_t *>(W.points) + (fwd ? (W.point_cap >> 1) - 1 - i : i);
  }
  __device__ __forceinline__ void put(const WarpWork &W, int dd, int db) {
    if ((threadIdx.x & 31) == 0 && n < room) *slot(W, n) = (uint32_t)(uint16_t)dd | (uint32_t)(uint16_t)db << 16;
    n += 1;
  }
  // the b position a pebble stands for; the start pebble stands at its
  // antidiagonal's going forward
  __device__ __forceinline__ int bpos(int4 q) const { return fwd && q.x < 0 ? (mida - q.y) >> 1 : q.w - q.y; }
  __device__ __forceinline__ bool inside(int4 q) const { return !fwd && q.x < 0 && q.w % tspace != aoff; }

  // The end past the last mark: an interval of its own, or part of the one
  // before (left in dd, db).
  __device__ __forceinline__ void tip(const WarpWork &W, int4 q, int trimx, int trimy, int trimd, int &dd, int &db) {
    const int qb = bpos(q);
    dd = trimd - q.z;
    db = sg * (trimy - qb);
    if (inside(q) || qb + q.y != trimx) {
      if (inside(q) && inner) {
        jd = dd;
        jb = db;
      } else
        put(W, dd, db);
      dd = db = 0;
    } else if (qb == trimy)
      dd = db = 0;
    else if (!fwd && q.x < 0) {
      jd = dd;
      jb = db;
    }
  }
};

// How the path crosses the lines of the entries that pebble `head` is older
// than: p is the first pebble after them (kind PEBBLE), or the path's head is
// from before (HEAD), or there is no trace to share (NONE).
__device__ __noinline__ void cross_entries(const WarpWork &W, TraceWalk &T, int head, int kind, int4 p) {
  const int lane = threadIdx.x & 31;
  while (T.last >= 0) {
    ShareEntry &O = W.share->entries[T.last];
    if (head >= __ldcg(&O.mark)) return;
    const unsigned eq = __ballot_sync(FULL, __ldcg(&O.HA[lane]) == head);
    if (lane == 0) {
      O.kind = eq ? kind : SHARE_NONE;
      O.lane = __ffs(eq) - 1;
      O.after = (int)T.n;
      O.pdiag = p.y;
      O.pdiff = p.z;
      O.pmark = p.w;
    }
    T.last = __ldcg(&O.prev);
  }
}

// The walk from pebble values q (its slot's successor is q.x) to the path's
// start.  A path's pebbles lie a dozen or so slots apart, so the pointers of
// the 128 slots up to the next one come into shared memory at once (the block
// below it already on its way), one lane per pebble found there takes its
// interval, and only the hops within a block are a chain: a warp's load per
// pebble took 360 ns each.  dd, db: what the first interval has already.
// Returns an error code.
template <bool SHARE>
__device__ __noinline__ int walk_back(const WarpWork &W, TraceWalk &io, int4 q, int dd, int db) {
  constexpr int SPAN = 128;
  const int lane = threadIdx.x & 31;
  const int4 *cl = reinterpret_cast<const int4 *>(W.pool.cells);  // ptr, diag, diff, mark
  int *sm = W.sm;
  TraceWalk T = io;
  int near = I32MAX, err = 0, ahead[SPAN / 32];
  int64_t steps = 0;
  int mark = SHARE && T.last >= 0 ? __ldcg(&W.share->entries[T.last].mark) : -1;
  while (q.x >= 0) {
    const int h = q.x;
    if (h < T.base || steps > T.lim || T.n > T.room) {
      err = T.n > T.room ? ALN_ERR_POINTS : ALN_ERR_CELLS;
      break;
    }
    if (SHARE && h < mark) {
      io = T;
      cross_entries(W, io, h, SHARE_PEBBLE, q);
      T.last = io.last;
      mark = T.last >= 0 ? __ldcg(&W.share->entries[T.last].mark) : -1;
    }
    const bool have = near != I32MAX && h >= near - SPAN && h < near;
    near = have ? near - SPAN : h - (SPAN - 1);
    if (!have) {
#pragma unroll
      for (int j = 0; j < SPAN / 32; j++) ahead[j] = cl[max(near + 32 * j + lane, 0)].x;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < SPAN / 32; j++) sm[32 * j + lane] = ahead[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < SPAN / 32; j++) ahead[j] = cl[max(near - SPAN + 32 * j + lane, 0)].x;
    // the path's pebbles in the block, before the next entry's line
    const int least = max(max(near, mark), 0);
    int cnt = 0, slot = h;
    for (int cur = h; cnt < 32 && cur >= least; cnt++) {
      slot = lane == cnt ? cur : slot;
      cur = sm[cur - near];
    }
    const bool in = lane < cnt;
    const int4 p = cl[slot];
    const int pb = T.bpos(p);
    int by = __shfl_up_sync(FULL, pb, 1), bz = __shfl_up_sync(FULL, p.z, 1);
    if (lane == 0) {
      by = T.bpos(q);
      bz = q.z;
    }
    const int vd = bz - p.z + (lane == 0 ? dd : 0), vb = T.sg * (by - pb) + (lane == 0 ? db : 0);
    const bool ends = T.inner && T.inside(p);  // (the start: the last pebble at most)
    if (in && !ends && T.n + lane < T.room)
      *T.slot(W, T.n + lane) = (uint32_t)(uint16_t)vd | (uint32_t)(uint16_t)vb << 16;
    const unsigned e = __ballot_sync(FULL, in && ends);
    if (e) {
      T.jd = __shfl_sync(FULL, vd, cnt - 1);
      T.jb = __shfl_sync(FULL, vb, cnt - 1);
    }
    T.n += cnt - (e ? 1 : 0);
    steps += cnt;
    dd = db = 0;
    q.x = __shfl_sync(FULL, p.x, cnt - 1);
    q.y = __shfl_sync(FULL, p.y, cnt - 1);
    q.z = __shfl_sync(FULL, p.z, cnt - 1);
    q.w = __shfl_sync(FULL, p.w, cnt - 1);
  }
  T.start = q.y;
  io = T;
  return err ? err : (T.n > T.room ? ALN_ERR_POINTS : 0);
}

// Publishes an extension that stopped: its first n own intervals (the walk's)
// and, filled by the caller on lane 0, the rest of its record.  Returns whether
// the list had room.
__device__ __forceinline__ bool publish(const WarpWork &W, const TraceWalk &T, int rec, int status) {
  const ShareTable &X = *W.share;
  const int lane = threadIdx.x & 31;
  ShareRec &R = X.recs[rec];
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(X.nlist, (unsigned long long)T.n);
  off = __shfl_sync(FULL, off, 0);
  const bool fits = (int64_t)off + T.n <= X.list_cap;
  __syncwarp();
  if (fits)
    for (int64_t i = lane; i < T.n; i += 32) X.list[off + i] = *T.slot(W, i);
  if (lane == 0) {
    R.own = (int)T.n;
    R.off = (int64_t)off;
  }
  __threadfence();
  __syncwarp();
  if (lane == 0) *(volatile int *)&R.status = fits ? status : SHARE_FAILED;
  return fits;
}

// A joined extension's path past its join: the extensions on the way to the
// tip, their parts of the trace from the tip on into the walk's buffer.
// Returns the first pebble after the join's line (x unset) in this
// extension's wave numbers (its wave `dif` joined entry e0), what the interval
// from there has already (dd, db), and the tip; false if there is no room.
// way: W.vcap places, for the entries on the way.
__device__ __noinline__ bool gather_path(const WarpWork &W, TraceWalk &T, int *way, int e0, int dif, int4 &q, int &dd,
                                         int &db, int &tipx, int &tipy, int &tipd) {
  const ShareTable &X = *W.share;
  const int lane = threadIdx.x & 31;
  int m = 0, status = SHARE_JOINED;
  for (int e = e0; status == SHARE_JOINED; m++) {
    if (m >= W.vcap) return false;
    if (lane == 0) way[m] = e;
    const ShareRec &R = X.recs[__ldcg(&X.entries[e].rec)];
    status = __ldcg(&R.status);
    if (status == SHARE_FAILED) return false;
    if (status == SHARE_DONE) {
      tipx = __ldcg(&R.tipx);
      tipy = __ldcg(&R.tipy);
      tipd = __ldcg(&R.tipd);
    } else
      e = __ldcg(&R.entry);
  }
  __syncwarp();
  dd = db = 0;
  for (int i = m - 1; i >= 0; i--) {
    const ShareEntry &E = X.entries[way[i]];
    const ShareRec &R = X.recs[__ldcg(&E.rec)];  // the owner; q, tipd are in its wave numbers from here
    if (i < m - 1) {
      // from the pebble after the line it joined on to its head there
      const int4 head = make_int4(0, __ldcg(&R.hdiag), __ldcg(&R.hdiff), __ldcg(&R.hmark));
      T.put(W, dd + q.z - head.z, db + T.sg * (T.bpos(q) - T.bpos(head)));
      dd = db = 0;
    }
    const int after = __ldcg(&E.after);
    const int64_t off = __ldcg(&R.off);
    if (T.n + after > T.room) return false;
    for (int k = lane; k < after; k += 32) *T.slot(W, T.n + k) = __ldcg(&X.list[off + k]);
    T.n += after;
    q = make_int4(0, __ldcg(&E.pdiag), __ldcg(&E.pdiff), __ldcg(&E.pmark));
    if (i == m - 1 && after == 0) T.tip(W, q, tipx, tipy, tipd, dd, db);
    // on to the joiner's wave numbers
    const int delta = (i > 0 ? __ldcg(&X.recs[__ldcg(&X.entries[way[i - 1]].rec)].dif) : dif) - __ldcg(&E.dif);
    q.z += delta;
    tipd += delta;
  }
  __syncwarp();
  return T.n <= T.room;
}

// forward_wave (fwd) or reverse_wave of a path, out of line: one copy of the
// code serves both directions and every call.  `start` is the forward wave's
// lowest diagonal on entry and, on return, the diagonal the path starts on.
// A scout's trace is left out (its own intervals go to the share's list).
// BLOCKS: waves of 32 to 124 diagonals run in registers (block_waves), for
// launches bounded by their longest calls; without, they too run as passes
// (wide_waves), for launches bounded by throughput, where the smaller loop
// and its registers pay (four CTAs per SM, with and without: 2 x 41 kbp 11.4
// and 13.4 ms of pair phase, 2 x 200 Mbp repeat-rich 260 and 211).
// Returns 1 on a work-space overflow (W.err set).
template <bool BLOCKS, bool SHARE>
__device__ __noinline__ int extend(const bool fwd, const bool scout, WarpWork &W, const AlignSpec &spec, const Seq &A, const Seq &B,
                                   Path &P, int &start, int maxd, int mida, int minp, int maxp, int aoff) {
  const int lane = threadIdx.x & 31;
  const int tspace = spec.trace_space;
  const int vmask = W.vcap - 1;
  Pebble *cells = W.pool.cells;
  if (maxd - start + 3 > W.vcap) {
    W.err |= ALN_ERR_VCAP;
    return 1;
  }
  Wave S;
  S.pa = fwd ? A.pf : A.pr;
  S.pb = fwd ? B.pf : B.pr;
  S.offA = fwd ? 0 : A.len;
  S.offB = fwd ? 0 : B.len;
  S.limA = fwd ? A.len : 0;
  S.limB = fwd ? B.len : 0;
  S.minp = fwd ? minp : -maxp;
  S.maxp = fwd ? maxp : -minp;
  S.tspace = tspace;
  S.ave_path = spec.ave_path;
  S.dscore = spec.dscore;
  S.sg = fwd ? 1 : -1;
  S.low = fwd ? start : -maxd;
  S.hgh = fwd ? maxd : -start;
  S.dif = S.cur = 0;
  S.besta = S.lasta = S.trima = S.sg * mida;
  S.bestx = S.trimx = S.sg * ((mida + maxd) >> 1);
  S.trimd = S.trimha = 0;
  Sharing sh;
  sh.rec = sh.last = sh.joined = -1;
  sh.guess = 0;
  sh.from = S.besta;
  sh.full = false;
  // (a border would be part of the state: such calls grow alone)
  S.line = SHARE && minp == -I32MAX && maxp == I32MAX ? next_line(S.besta) : I32MAX;
  S.more = 1;
  int64_t call_base = -1;  // this call's first pebble: the reference's cells[0]

  // 0-wave: diagonals visited from the highest down
  int ka = I32MAX, kb = NO_WAVE;
  for (int top = S.hgh; top >= S.low; top -= 32) {
    const int k = top - lane;
    const bool act = k >= S.low;
    int x = 0, mark = 0, nak = 0, mx = 0;
    if (act) {
      const int x0 = (mida + S.sg * k) >> 1;
      // forward: the trace mark at or below the start is its pebble's mark;
      // reverse: the start itself, and the mark below it comes next
      const int m0 = ((x0 + (tspace - aoff) - (fwd ? 0 : 1)) / tspace - 1) * tspace + aoff;
      x = S.sg * x0;
      mark = fwd ? m0 : x;
      nak = fwd ? m0 + tspace : -m0;
      mx = min(S.limA - x, S.limB - x + k);
    }
    bool go;
    const int xs = x, run = snake<4>(S, x, k, act, mx, go);
    const bool hit = act && (!go || run == mx);
    x += run;
    const int c = (x << 1) - k;
    const int npb = act ? 1 + (x >= nak ? (x - nak) / tspace + 1 : 0) : 0;
    const int off = warp_excl_sum(npb, lane);
    const int tot = __reduce_add_sync(FULL, npb);
    const int64_t pb0 = warp_pebbles(W, tot);
    if (pb0 < 0) return 1;
    if (call_base < 0) {
      call_base = pb0;
      S.trimha = (int)pb0;
    }
    int ha = (int)pb0 + off;
    if (act) {
      *reinterpret_cast<int4 *>(cells + ha) = make_int4(-1, S.sg * k, 0, S.sg * mark);
      for (; x >= nak; nak += tspace) {
        mark = nak;
        *reinterpret_cast<int4 *>(cells + ha + 1) = make_int4(ha, S.sg * k, 0, S.sg * mark);
        ha += 1;
      }
      const int vi = k & vmask;
      W.V[0][vi] = c;
      W.C[0][vi] = RingCell{PATH_INT, ha, mark};
      W.NA[vi] = nak;
    }
    if (__any_sync(FULL, hit)) {
      const bool hb = met_b(S, xs, k, go);
      ka = min(ka, __reduce_min_sync(FULL, hit && !hb ? k : I32MAX));
      kb = max(kb, __reduce_max_sync(FULL, hit && hb ? k : NO_WAVE));
    }
    // the last record is the highest diagonal with the pass's best
    const int rc = __reduce_max_sync(FULL, act ? c : NO_WAVE);
    if (rc > S.besta) {
      const int L = __ffs(__ballot_sync(FULL, act && c == rc)) - 1;
      S.besta = S.trima = S.lasta = rc;
      S.bestx = S.trimx = __shfl_sync(FULL, x, L);
      S.trimha = __shfl_sync(FULL, ha, L);
    }
  }
  __syncwarp();
  if (ka != I32MAX || kb != NO_WAVE) {
    S.more = can_grow(S, S.besta);
    if (ka != I32MAX) S.hgh = ka - 1;
    if (kb != NO_WAVE) S.low = kb + 1;
  }

  // an extension that fails lets those that joined it go on alone
  auto give_up = [&]() {
    if (SHARE && sh.rec >= 0 && lane == 0) *(volatile int *)&W.share->recs[sh.rec].status = SHARE_FAILED;
    return 1;
  };
  const int64_t t0 = P.trace_off;
  TraceWalk T;
  T.fwd = fwd;
  T.inner = !fwd && P.tlen != 0;
  T.sg = S.sg;
  T.mida = mida;
  T.tspace = tspace;
  T.aoff = aoff;
  T.room = (fwd ? W.point_cap - t0 : t0) >> 1;
  T.base = call_base;
  const int4 *cl = reinterpret_cast<const int4 *>(cells);
  int trimx, trimy, trimd;
  const int max_waves = A.len + B.len + 1024;
grow:
  while (S.more && S.lasta >= S.besta - TRIM_MLAG) {
    // no wave to grow from, or more waves than bases: neither ends by itself
    if (S.hgh < S.low || S.dif > max_waves) {
      W.err |= ALN_ERR_VCAP;
      return give_up();
    }
    int stop = max_waves + 1;
    if (W.long_waves > 0 && !W.flagged) {
      if (S.dif + 1 >= W.long_waves) {
        // a long call: the other warps of this SM take no new task, so that it
        // runs with the SM to itself once their current tasks end
        if (lane == 0) {
          unsigned sm;
          asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
          if (sm < SM_FLAGS) atomicExch(&W.smflag[sm], 1u);
        }
        W.flagged = 1;
      } else
        stop = min(stop, W.long_waves - 1);
    }
    const int width = S.hgh - S.low + 1 + (S.low > S.minp ? 1 : 0) + (S.hgh < S.maxp ? 1 : 0);
    int r;
    if (SHARE && S.besta >= S.line && width <= NARROW) {
      S.line = next_line(S.besta);
      if (W.task) scout_if_free(W);
      if (cross_line(W, S, W.pair | (fwd ? 1u << 31 : 0u), sh)) break;
      if (sh.full) S.line = I32MAX;
    }
    if (width <= NARROW) r = narrow_waves<BLOCKS ? 4 : 2>(W, S, stop);
    else if (BLOCKS && width <= BLOCK * NARROW) r = block_waves<BLOCK>(W, S, stop);
    else r = wide_waves(W, S, stop, BLOCKS ? BLOCK * NARROW - 8 : BLOCK_OUT);
    if (r) return give_up();
  }
  __syncwarp();

  // Trace-back, from the path's tip to its start.
  T.lim = W.chunk_next - call_base + 1;
  T.n = 0;
  T.jd = T.jb = 0;
  T.last = -1;
  int err = 0;
  bool joined = false, closed = false;  // closed: its record, if any, has been published
  if (SHARE && sh.joined >= 0) {
    const ShareTable &X = *W.share;
    const ShareEntry &E = X.entries[sh.joined];
    ShareRec &R = X.recs[__ldcg(&E.rec)];
    const bool walks = sh.rec >= 0 || (scout && fwd);
    // Its own part, back from head pebble `from`.  An entry that this pebble
    // is older than has no pebble between its line and the join: what its
    // joiners would start from lies past the join, so they go on alone.
    auto walk_own = [&](int from) {
      T.n = 0;
      T.jd = T.jb = 0;
      T.last = sh.last;
      const int4 q = cl[from];
      if (T.last >= 0) cross_entries(W, T, from, SHARE_NONE, q);
      return walk_back<SHARE>(W, T, q, 0, 0);
    };
    if (walks) {
      // as it most likely is, while the owner's is on its way
      err = walk_own(sh.guess);
      if (err) {
        W.err |= err;
        return give_up();
      }
    }
    if (scout && sh.rec < 0) {  // nothing behind it for others
      start = T.start;
      return 0;
    }
    int status = 0;
    if (lane == 0)
      for (int poll = 0; poll < SHARE_POLLS && (status = *(volatile int *)&R.status) == 0; poll++) __nanosleep(200);
    status = __shfl_sync(FULL, status, 0);
    __threadfence();
    const int kind = __ldcg(&E.kind);
    if (status == 0 || status == SHARE_FAILED || kind == SHARE_NONE) {
      // go on alone (what was entered so far stays with the record, which fails)
      give_up();
      sh.rec = sh.last = sh.joined = -1;
      goto grow;
    }
    const int dif = S.dif - __ldcg(&E.dif), kc = S.low + ((__ldcg(&E.lane) - S.low) & 31);
    const int head = W.C[S.cur][kc & vmask].HA;
    const bool own = status == SHARE_DONE && __ldcg(&R.tipd) <= __ldcg(&E.dif);
    if (lane == 0) atomicAdd(X.joins + (own ? 2 : kind == SHARE_HEAD ? 1 : 0), 1u);
    if (own) {
      // the owner found nothing past this wave: the tip is this extension's own
    } else if (kind == SHARE_HEAD) {
      // the owner's tip is before the next mark
      S.trimx = S.sg * __ldcg(&R.tipx);
      S.trima = S.trimx + S.sg * __ldcg(&R.tipy);
      S.trimd = __ldcg(&R.tipd) + dif;
      S.trimha = head;
    } else {
      joined = true;
      if (walks && head != sh.guess) err = walk_own(head);
      bool listed = false;
      if (sh.rec >= 0 && !err) {
        ShareRec &O = X.recs[sh.rec];
        if (lane == 0) {
          const int4 q = cl[head];
          O.entry = sh.joined;
          O.dif = S.dif;
          O.hdiag = q.y;
          O.hdiff = q.z;
          O.hmark = q.w;
        }
        listed = publish(W, T, sh.rec, SHARE_JOINED);
        closed = true;
      }
      if (!scout && !err) {
        // the parts past the join, then this extension's own
        const int64_t own = T.n;
        int4 q;
        int dd, db;
        T.n = 0;
        if (!gather_path(W, T, W.V[S.cur ^ 1], sh.joined, S.dif, q, dd, db, trimx, trimy, trimd)) {
          sh.rec = sh.last = sh.joined = -1;  // (its record stands)
          goto grow;
        }
        q.x = head;
        T.last = -1;
        if (listed) {
          const int4 p = cl[head];
          T.put(W, dd + q.z - p.z, db + T.sg * (T.bpos(q) - T.bpos(p)));
          const int64_t off = __ldcg(&X.recs[sh.rec].off);
          if (T.n + own > T.room) err = ALN_ERR_POINTS;
          else
            for (int64_t i = lane; i < own; i += 32) *T.slot(W, T.n + i) = __ldcg(&X.list[off + i]);
          T.n += own;
        } else
          err = walk_back<SHARE>(W, T, q, dd, db);
      }
    }
  }
  if (!joined) {
    T.n = 0;
    T.jd = T.jb = 0;
    T.last = SHARE ? sh.last : -1;
    trimx = S.sg * S.trimx;
    trimy = S.sg * S.trima - trimx;
    trimd = S.trimd;
    const int4 q = cl[S.trimha];
    if (SHARE && T.last >= 0) cross_entries(W, T, S.trimha, SHARE_HEAD, q);
    int dd, db;
    T.tip(W, q, trimx, trimy, trimd, dd, db);
    err = walk_back<SHARE>(W, T, q, dd, db);
    if (SHARE && sh.rec >= 0 && !err) {
      if (lane == 0) {
        ShareRec &O = W.share->recs[sh.rec];
        O.tipx = trimx;
        O.tipy = trimy;
        O.tipd = trimd;
      }
      publish(W, T, sh.rec, SHARE_DONE);
    }
  }
  if (err) {
    W.err |= err;
    return closed ? 1 : give_up();
  }
  __syncwarp();
  const int64_t n = T.n;
  if (scout) {
    start = T.start;
    return 0;
  }
  if ((T.jd | T.jb) && lane == 0) {
    uint16_t *o = W.points + t0;
    o[0] = (uint16_t)(o[0] + T.jd);
    o[1] = (uint16_t)(o[1] + T.jb);
  }
  __syncwarp();
  {
    uint32_t *pt = reinterpret_cast<uint32_t *>(W.points);
    const int64_t src = fwd ? (W.point_cap >> 1) - n : 0, dst = fwd ? t0 >> 1 : (t0 >> 1) - n;
    for (int64_t i = 0; i < n; i += 32) {
      const int64_t j = fwd ? i + lane : n - 1 - i - lane;  // away from what is still to be read
      uint32_t v = 0;
      const bool in = i + lane < n;
      if (in) v = pt[src + j];
      __syncwarp();
      if (in) pt[dst + j] = v;
      __syncwarp();
    }
  }
  if (fwd) {
    start = T.start;
    P.aepos = trimx;
    P.bepos = trimy;
    P.diffs = trimd;
    P.tlen = (int)(2 * n);
  } else {
    P.abpos = trimx;
    P.bbpos = trimy;
    P.diffs += trimd;
    P.tlen += (int)(2 * n);
    P.trace_off -= (int)(2 * n);
  }
  return 0;
}

// A path on the complemented A (and so on reversed B coordinates) in
// forward coordinates: both intervals mirrored, and the trace-point pairs
// (diffs, b-delta) in the opposite order, the warp's lanes swapping pair q
// with pair npairs-1-q.
__device__ __forceinline__ void path_to_forward(uint16_t *trace, const Seq &A, const Seq &B, Path &P) {
  const int lane = threadIdx.x & 31;
  const int ab = P.abpos, bb = P.bbpos;
  P.abpos = A.len - P.aepos;
  P.aepos = A.len - ab;
  P.bbpos = B.len - P.bepos;
  P.bepos = B.len - bb;
  const int npairs = P.tlen >> 1;
  __syncwarp();
  for (int q = lane; q < npairs / 2; q += 32) {
    uint32_t *x = reinterpret_cast<uint32_t *>(trace) + q, *y = reinterpret_cast<uint32_t *>(trace) + (npairs - 1 - q);
    const uint32_t t = *x;
    *x = *y;
    *y = t;
  }
  __syncwarp();
}

// Local_Alignment (lib/align.c:1423-1576) on one warp.  The path is grown
// forward from the seed point (antidiagonal `anti`, diagonals [low, hgh],
// kept within `lbord` / `hbord` of them when those are set), then backward
// from the diagonal the forward pass started on.  An end that moved fewer
// than DUB_TRIM antidiagonals from `anti` did not get away from the seed:
// with both ends short the path shrinks to the midpoint of the two, without
// trace points; with one end short, that direction runs again from the end
// the other direction reached (a forward re-run keeps the reverse pass's
// start, a reverse re-run counts its differences afresh).  With `acomp` A is
// the complemented contig and the path comes back in forward coordinates.
// Returns 1 on a work-space overflow (W.err says which).
template <bool BLOCKS, bool SHARE>
__device__ __noinline__ int local_alignment_w(WarpWork &W, const AlignSpec &spec, const Seq &A, const Seq &B,
                                                 bool acomp, Path &P, int low, int hgh, int anti, int lbord,
                                                 int hbord) {
  const int maxtp = 2 * (A.len / spec.trace_space + 2);  // trace points the longest path can have
  if (2 * (int64_t)maxtp > W.point_cap) {
    W.err |= ALN_ERR_POINTS;
    return 1;
  }
  P.trace_off = maxtp;
  while (((anti - hgh) >> 1) < 0) hgh -= 1;  // no diagonal above the antidiagonal's start
  const int minp = lbord < 0 ? -I32MAX : low - lbord;
  const int maxp = hbord < 0 ? I32MAX : hgh + hbord;
  const int aoff = acomp ? A.len % spec.trace_space : 0;

  int from = low;
  if (extend<BLOCKS, SHARE>(true, false, W, spec, A, B, P, from, hgh, anti, minp, maxp, aoff)) return 1;
  const bool fwd_away = (P.aepos + P.bepos) - anti >= DUB_TRIM;
  if (extend<BLOCKS, SHARE>(false, false, W, spec, A, B, P, from, from, anti, minp, maxp, aoff)) return 1;
  const bool rev_away = anti - (P.abpos + P.bbpos) >= DUB_TRIM;

  if (!fwd_away && !rev_away) {
    P.aepos = P.abpos = (P.abpos + P.aepos) >> 1;
    P.bepos = P.bbpos = (P.bbpos + P.bepos) >> 1;
    P.tlen = 0;
  } else if (!fwd_away) {
    from = P.abpos - P.bbpos;
    P.tlen = 0;
    if (extend<BLOCKS, SHARE>(true, false, W, spec, A, B, P, from, from, P.abpos + P.bbpos, minp, maxp, aoff)) return 1;
  } else if (!rev_away) {
    from = P.aepos - P.bepos;
    const int at = P.aepos + P.bepos;
    P.tlen = 0;
    P.diffs = 0;
    if (extend<BLOCKS, SHARE>(false, false, W, spec, A, B, P, from, from, at, minp, maxp, aoff)) return 1;
  }
  if (acomp) path_to_forward(W.points + P.trace_off, A, B, P);
  return 0;
}

// A scout: a call's two extensions for those that join them.  What it cannot
// do (a full pool) its joiners do themselves.
__device__ __forceinline__ void scout_w(WarpWork &W, const AlignSpec &spec, const Seq &A, const Seq &B, bool acomp,
                                        int low, int hgh, int anti) {
  Path P;
  P.tlen = P.diffs = P.abpos = P.bbpos = P.aepos = P.bepos = 0;
  P.trace_off = 2 * (A.len / spec.trace_space + 2);
  if (2 * (int64_t)P.trace_off > W.point_cap) return;
  while (((anti - hgh) >> 1) < 0) hgh -= 1;
  const int aoff = acomp ? A.len % spec.trace_space : 0;
  int from = low;
  if (hgh < low || extend<true, true>(true, true, W, spec, A, B, P, from, hgh, anti, -I32MAX, I32MAX, aoff)) return;
  P.tlen = 0;
  extend<true, true>(false, true, W, spec, A, B, P, from, from, anti, -I32MAX, I32MAX, aoff);
}

}  // namespace aln
}  // namespace pga
