// The phase-settled exact search, shared by the whole-lattice search
// (fullgraph.cu) and the ROI searches (route.cu): one search by a team of
// CTAs.
//
// The rule (SimpleDijkstra.find_path_roi, unified_pathfinder.py:2451-2548):
// every node takes the lexicographic minimum of (float32(alt), L(u), u) over
// its in-neighbours u, alt = (L(u) + c) + pen.  Phases: every frontier node
// pulls from the in-neighbours settled before the phase; with T = a lower
// bound of the frontier's labels it is final when its label equals T or its
// float32 key is below float32((T + cin) + pen), cin being its cheapest
// in-arc from any other in-neighbour.  A settling node marks its unreached
// out-neighbours and offers its candidate labels to the next T.  A phase's
// decisions depend only on the set settled before it and on T, and any T not
// above the true minimum gives the same result (only the phase count moves).
//
// What bounds it: a phase is a chain of dependent L2 round trips and a
// barrier over the team, far from any bandwidth (a few thousand nodes a phase
// on 152 SMs).  So everything a phase needs is on the SM before it starts:
//
// * Frontier entries stay with the CTA that found them, in shared memory,
//   with their CSR row (neighbour ids, in- and out-costs).  The row of a new
//   entry is fetched while the barrier is waited for.  A carried entry costs
//   one round trip per phase: its neighbours' records.
// * A node's record is 16 bytes, read in one load: label, state, penalty.
//   Until the node settles the label's place holds its row bounds, so whoever
//   reaches it first has all of its entry without another load.
// * Reaching a node is a plain store; nodes reached twice in one phase are
//   sorted out by an atomic on the first examination, in the shadow of the
//   record loads, not by an atomic each on the critical path.
// * T, the frontier size and the flags of a phase travel in the barrier's own
//   16-byte word, which one thread per CTA polls.
// * One lane serves one arc of an entry (two in rows of 9 to 16 arcs: 64
//   entries at a time instead of 32, 10.0 -> 9.5 us a phase at 600x400x12; two
//   lanes of two arcs in rows of up to 4: 18.8 -> 16.3 at 1000x800x32, where a
//   thousand entries per SM make it a matter of instructions).
//   512 threads with 128 registers, not 1024 with 64: idle warps cost issue
//   slots and 64 registers spill (307x199x8: 6.5 -> 4.6 us a phase).  Rows
//   longer than 32 arcs, and values that ticks cannot hold, are searched by
//   the general form, kept out of line.
// * Labels are whole ticks of 2^-30 in 64-bit integers.  This part has two
//   FP64 lanes per SM, so an FP64 instruction of a warp takes 16 clocks of it:
//   in doubles the 18 of an examination were 4.4 us of a phase (600x400x12
//   fell from 13.9 to 9.3 us a phase, 1000x800x32 from 46 to 28).  Ticks
//   are exact wherever the doubles are: costs and penalties of 2^-7 or more
//   (or 0) are multiples of 2^-30, and below 2^22 their double sums do not
//   round.  A search that meets any other value goes on in doubles from the
//   phase in which it did (go_over).
// * A CTA with more entries than its share sends new ones to a list in global
//   memory that the next phase deals over the team (see plan()).
#pragma once
#include "common.cuh"

namespace ogr_phase {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr unsigned long long kNone = ~0ull;

struct __align__(16) Rec {
  unsigned long long lab;   // label once settled (ticks, or a double's bits); before that
                            // {row start, row length}
  int32_t sp;      // 0 unreached, 1 reached, 2 + the phase in which it settled; multi-source:
                   // | kTgt, | kSeed
  float pen;       // node penalty of this search
};

// One barrier of the team: a = arrivals (bits 0-9), destination settled (10),
// surplus entries (11-31, each CTA's share of the field at most kMostOut: at
// that, the counter in global memory tells), next frontier's entries (32-63);
// t = ~T, taken by max so that an all-zero slot is the identity.  T = 0 after
// the first phase says that a CTA met a value ticks cannot hold.
struct __align__(16) Slot {
  unsigned long long a;
  unsigned long long t;
};
constexpr unsigned long long kArrive = 1ull, kDst = 1ull << 10, kOut = 1ull << 11, kCount = 1ull << 32;
constexpr unsigned long long kArriveMask = 0x3ffull;
constexpr unsigned kOutMask = 0x1fffff, kMostOut = 2047;
constexpr int kMostEntries = 1 << 14;        // (with rows of up to 32 arcs they ask for fewer than 2^20 places)
constexpr int kMaxTeam = 1023;      // CTAs of a team
constexpr int kStInexact = 100;    // Outcome::status: to go on in doubles (go_over)
constexpr int kFirstOver = 6;      // first phase of a search that does (a multiple of 2 and of 3)

// Control words of a team in global memory, zero before a search.
struct Ctl {
  alignas(128) Slot slot[4];
  alignas(128) int32_t err;        // a CTA gave up waiting
  alignas(128) int32_t nov[3];     // surplus entries by phase mod 3
  int32_t kept;                    // frontier of a search that goes over to doubles
};

constexpr int32_t kTgt = 1 << 30, kSeed = 1 << 29, kSpMask = kSeed - 1;

__device__ __forceinline__ Rec ld_rec(const Rec* p) {
  const int4 q = __ldcg(reinterpret_cast<const int4*>(p));
  Rec r;
  r.lab = ((unsigned long long)(unsigned)q.y << 32) | (unsigned)q.x;
  r.sp = q.z;
  r.pen = __int_as_float(q.w);
  return r;
}

__device__ __forceinline__ void st_rec(Rec* p, unsigned long long lab, int32_t sp, float pen) {
  __stcg(reinterpret_cast<int4*>(p), make_int4((int)(unsigned)lab, (int)(unsigned)(lab >> 32), sp, __float_as_int(pen)));
}

// ---- labels in ticks of 2^-30 ---------------------------------------------
constexpr unsigned kBitsLow = 0x3c000000u, kBitsHigh = 0x4a800000u, kBitsInf = 0x7f800000u;   // 2^-7, 2^22, +inf
constexpr unsigned long long kTickLimit = 1ull << 52;

// Whether a cost (or +inf) or penalty is a whole number of ticks below 2^22.
__device__ __forceinline__ bool tick_exact(float c) {
  const unsigned b = __float_as_uint(c);
  return b == 0u || (b >= kBitsLow && b < kBitsHigh) || b == kBitsInf;
}

__device__ __forceinline__ bool tick_finite(float c) { return tick_exact(c) && __float_as_uint(c) != kBitsInf; }

// Ticks of a value that passes tick_finite.
__device__ __forceinline__ unsigned long long ticks(float c) {
  const unsigned b = __float_as_uint(c);
  // the shift is at most 28: one wide multiply instead of a 64-bit shift
  return b < kBitsLow ? 0ull : (unsigned long long)((b & 0x7fffffu) | 0x800000u) * (1u << (((b >> 23) - 120u) & 31u));
}

// The largest tick count that rounds (to nearest even) to the same float32
// as x: two labels have one float32 key iff the larger is not above the
// smaller's round_hi.
__device__ __forceinline__ unsigned long long round_hi(unsigned long long x) {
  const int e = 40 - __clzll((long long)(x | 1ull));   // bits below the 24 that a float32 keeps
  if (e <= 0) return x;
  const unsigned long long half = 1ull << (e - 1);
  const unsigned long long r = (x + half - 1ull + ((x >> e) & 1ull)) >> e;
  // r = 2^24 is the next binade's first value: its upper neighbour is twice as far
  return (r << e) + (r == (1ull << 24) ? half << 1 : half - (r & 1ull));
}

// Label of a seed given as a double (kFix): false if ticks cannot hold it.
__device__ __forceinline__ bool seed_ticks(double c, unsigned long long* out) {
  const double x = c * 1073741824.0;
  if (!(x >= 0.0 && x < (double)kTickLimit)) return false;
  const unsigned long long n = (unsigned long long)x;
  *out = n;
  return (double)n == x;
}

template <bool kFix>
__device__ __forceinline__ double label_value(unsigned long long lab) {
  return kFix ? (double)lab * (1.0 / 1073741824.0) : __longlong_as_double((long long)lab);
}

// What a search is given.  Node ids are 0..R-1 in tie order; in an ROI search
// (kRoi) they index roi[] and g2r maps global ids back (-1 outside).
struct Problem {
  int32_t R;
  int32_t src, dst;                // -1: multi-source
  const int32_t* indptr;
  const int32_t* indices;
  const int32_t* rev;
  const float* cost;               // cost of each arc
  const float* rcost;              // cost of each arc's reverse, or NULL (then cost[rev])
  const int32_t* roi;
  const int32_t* g2r;
  Rec* rec;
  int32_t* par;
  int32_t* claim;                  // == sid: the node has its entry
  int32_t sid;
  int4* ov[2];                     // surplus lists of {node, row start, row length, penalty}, by phase
  const double* mseed;             // multi-source: cost of each node marked kSeed
  Ctl* ctl;
  int rank, nranks;                // this CTA and the CTAs of the team
  bool want_stats;
};

// What it found (the same in every CTA of the team).
struct Outcome {
  int status;                      // OGR_OK with found, OGR_NO_PATH, or an error
  bool found;                      // single source: dst settled; multi-source: frontier exhausted
  bool exhausted;                  // the frontier ran out before dst
  int phases;                      // (kStInexact: the last two are the phase to be taken back, and the look at its end)
  unsigned long long ld;           // label of dst (as in Rec)
  unsigned long long examined;     // entries this CTA examined
  long long wait, clocks;          // clocks thread 0 spent waiting, and in all
};

// Shared memory of one CTA: the control words, then as many entries as fit
// with their rows of A arcs.
struct Head {
  // what the phase is to do, written by thread 0 between two phases
  struct __align__(16) Plan {
    unsigned long long T;
    int verdict;                   // kGo, or how the search ends
    int nloc, ncarr, n;            // entries: here, of these carried, with the share of the surplus list
    int head, avail;               // free ring: next place, places to be given
  } plan;
  unsigned long long a, t;         // the barrier's word, as thread 0 read it
  unsigned long long ld;           // label of dst, once settled
  unsigned long long wmin[kWarps];
  // entries carried (bits 0-11) and places asked for (12-31: the count may run
  // over where none are given, with kMostEntries or more) in a phase
  unsigned push[2];
  unsigned tail;                   // free ring: end
  int inexact, nov_out, dst_hit, ok;
  int res[3];
  // bounds of the search: polls of a wait, settle phases (thread 0 sets and
  // reads them; in registers of all threads they were spilled)
  unsigned spin;
  int max_phase;
  int first;                       // general form: the first phase, 0 or kFirstOver
};

template <int A>
struct Body {
  static constexpr int kS = A == 4 ? 3072 : A == 8 ? 1792 : A == 16 ? 1024 : 512;
  int4 ent[kS];                    // {node, row start, row length | kTgt | kSeed | unclaimed << 31, penalty}
  int32_t rid[kS * A];             // neighbour, in-cost and out-cost of each arc
  float rin[kS * A];
  float rout[kS * A];
  uint16_t carr[2][kS];            // entries carried into this phase and the next
  uint16_t fresh[2][kS];           // entries new in this phase and the next (their rows are fetched in between)
  uint16_t freel[kS];              // ring of free entries
};
constexpr size_t kHeadBytes = (sizeof(Head) + 127) & ~(size_t)127;
constexpr size_t smax(size_t a, size_t b) { return a > b ? a : b; }
constexpr size_t kSmemBytes =
    kHeadBytes + smax(smax(sizeof(Body<4>), sizeof(Body<8>)), smax(sizeof(Body<16>), sizeof(Body<32>)));
static_assert(kSmemBytes <= 227 * 1024, "one CTA's shared memory");

enum { kGo = 0, kFound, kFoundEarly, kEmpty, kCapped, kInexactSeen, kTimedOut };

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
  const unsigned hi = __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32));
  const unsigned lo = __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0xffffffffu);
  return ((unsigned long long)hi << 32) | lo;
}

__device__ __forceinline__ void ld_slot(const Slot* p, unsigned long long& a, unsigned long long& t) {
  asm volatile(
      "{\n\t.reg .b128 q;\n\tld.acquire.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
      : "=l"(a), "=l"(t)
      : "l"(p)
      : "memory");
}

__device__ __forceinline__ void clear_slot(const Problem& pr, int k) {
  Slot* s = &pr.ctl->slot[k & 3];
  s->a = 0ull;
  s->t = 0ull;
}

// Thread 0: hand in this CTA's word for barrier k (after a __syncthreads that
// follows the phase's writes).  Alone in its team a CTA keeps the word.
__device__ __forceinline__ void arrive(const Problem& pr, Head& sm, int k, unsigned long long add,
                                       unsigned long long tmin) {
  if (pr.nranks == 1) {
    sm.a = add;
    sm.t = ~tmin;
    return;
  }
  Slot* s = &pr.ctl->slot[k & 3];
  if (tmin != kNone) asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(&s->t), "l"(~tmin) : "memory");
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(&s->a), "l"(add) : "memory");
}

// Thread 0: wait for barrier k and take its word.  The wait is bounded:
// sm.ok = 0 once any CTA of the team gave up.
__device__ __forceinline__ void await(const Problem& pr, Head& sm, int k, unsigned long long& a,
                                      unsigned long long& t) {
  if (pr.nranks == 1) {
    a = sm.a;
    t = sm.t;
    return;
  }
  const Slot* s = &pr.ctl->slot[k & 3];
  const unsigned want = (unsigned)pr.nranks;
  unsigned it = 0;
  while (true) {
    ld_slot(s, a, t);
    if ((unsigned)(a & kArriveMask) >= want) return;
    ++it;
    if (it > sm.spin || ((it & 63) == 0 && *(const volatile int32_t*)&pr.ctl->err)) {
      atomicExch(&pr.ctl->err, 1);
      sm.ok = 0;
      return;
    }
    if (it > 256) __nanosleep(32);
  }
}

// The same, the word left in sm.a / sm.t.
__device__ __forceinline__ void await(const Problem& pr, Head& sm, int k) {
  unsigned long long a = 0, t = 0;
  await(pr, sm, k, a, t);
  sm.a = a;
  sm.t = t;
}

// The phases of one search.  Before the call: rec of every node holds
// {row start, row length}, sp 0 (targets kTgt, seeds 1 | kSeed) and its
// penalty; the leader's first entries (src, or the seeds: claimed) lie in surplus list 0 with their count in
// nov[0], all of it ordered before this call in every CTA of the team by the
// caller's barrier k0, whose word (count, T) the caller left in sm.a / sm.t.
// Uses barriers k0 + 1, k0 + 2, ..., of which the first two have clear words
// on entry; on return k0 + phases and the next have (unless found early).
//
// kGen = false: rows of at most L * K arcs, K per lane, labels in ticks.
// kGen = true: any rows (read in global memory by L lanes), labels in doubles.
template <int L, int K, bool kGen, bool kMulti, bool kRoi>
__device__ __forceinline__ Outcome run_phases(const Problem& pr, Head& sm, Body<L * K>& bd, int k0) {
  typedef unsigned long long u64;
  constexpr int kA = L * K;
  constexpr int kS = Body<kA>::kS;
  constexpr int kPer = 32 / L;                 // entries per warp at a time
  constexpr int kGroups = kThreads / L;        // entries per CTA at a time
  constexpr unsigned kAll = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sl = lane & (L - 1);
  const unsigned gmask = (L == 32 ? kAll : (1u << (L & 31)) - 1u) << (lane & ~(L - 1));
  const unsigned below = (1u << lane) - 1u;
  const float kInf = __int_as_float(0x7f800000);
  Rec* __restrict__ rec = pr.rec;
  Outcome out{};
  for (int i = tid; i < kS; i += kThreads) bd.freel[i] = (uint16_t)i;
  // thread 0's view of the search between phases
  bool dst_done = false;
  u64 ld = 0;
  int head = 0;
  const unsigned team = (unsigned)pr.nranks, per_team = team > 1 ? (unsigned)((1ull << 32) / team) : 0;
  const float share = 1.0f / (float)team;
  auto plan = [&](int phase, int b3, int nf, int nk, float carried, u64 word, u64 tbits) {
    // (word, tbits: the barrier's.  The whole team waits for this; with the
    // word taken through shared memory and three divisions it was 540 clocks.)
    const u64 T = ~tbits;
    const unsigned total = (unsigned)(word >> 32);
    int verdict = kGo;
    if (!kMulti && !dst_done && (word & kDst)) {
      dst_done = true;
      if (!sm.dst_hit) sm.ld = __ldcg(&rec[pr.dst].lab);
      ld = sm.ld;
      if (!pr.want_stats) verdict = kFoundEarly;
    }
    if (verdict == kGo) {
      if (total == 0)
        verdict = dst_done || kMulti ? kFound : kEmpty;
      else if (dst_done && T > ld)
        verdict = kFound;
      else if (phase > sm.max_phase)
        verdict = kCapped;
    }
    if (!kGen && phase > 0 && T == 0) verdict = kInexactSeen;
    int n = nf + nk;
    unsigned nov = (unsigned)(word >> 11) & kOutMask;
    if (nov) {
      if (nov >= kMostOut) nov = (unsigned)__ldcg(&pr.ctl->nov[b3]);
      if (nov > (unsigned)pr.rank) {
        // ceil((nov - rank) / team); the high product is the floor or one less
        const unsigned x = nov - (unsigned)pr.rank + team - 1, d = team > 1 ? __umulhi(x, per_team) : x;
        n += (int)(x - d * team >= team ? d + 1 : d);
      }
    }
    // The places given to new entries: the most entries that the CTA should
    // have in the next phase, less those it will carry (the same share of its n
    // as of the last phase's).  Entries beyond them are dealt over the team.
    // A round of kGroups entries costs the same whether full or not (600x400x12:
    // 5,500 clocks one, 10,000 two, 14,800 three), and the last CTA's rounds are
    // the phase: the average is rounded up to whole rounds.  A phase that takes
    // surplus in is longer for everyone, so only every other one evens out
    // finer than that; of a thin frontier all new entries go, to spread it.
    // us a phase at 600x400x12 / 307x199x8 / 1000x800x32, ROIs of 14,000 nodes:
    // 7.6 / 3.9 / 16.3, 3.57.  Evened out every phase 7.8 / 4.3 / 16.9, 3.9; all
    // of a phase's new entries sent away by CTAs a quarter above the average
    // 8.3 / 4.0 / 18.3, 3.6; limits a fifth higher 7.8 / 4.0 / 17.3, 3.6.
    const bool deal = (phase & 1) != 0;
    const float avg = (float)total * share;
    float room = 1e6f;
    if (team > 1) {
      const float unit = (float)(deal ? kGroups / 8 : kGroups);
      room = unit * ceilf(avg / unit) - (float)n * carried;
      if (deal && avg < (float)(kGroups / 8)) room = n > kGroups / 4 ? 0.0f : 1e6f;
    }
    head += nf;
    if (kGen || verdict != kInexactSeen) sm.plan.T = T;     // (else that of the phase to be taken back)
    sm.plan.verdict = verdict;
    sm.plan.nloc = nf + nk;
    sm.plan.ncarr = nk;
    sm.plan.n = n;
    sm.plan.head = head;
    sm.plan.avail = n < kMostEntries ? min(sm.tail - head, (unsigned)fmaxf(room, 0.0f)) : 0;
  };
  if (tid == 0) {
    sm.push[0] = sm.push[1] = 0;
    sm.tail = kS;
    sm.nov_out = 0;
    sm.dst_hit = 0;
    sm.inexact = 0;
    plan(kGen ? sm.first : 0, 0, 0, 0, 0.0f, sm.a, sm.t);
  }
  __syncthreads();
  const long long c_start = clock64();
  int phase = kGen ? sm.first : 0, b3 = 0;           // b3 = phase mod 3
  int verdict;
  while ((verdict = sm.plan.verdict) == kGo) {
    const u64 T = sm.plan.T;
    const int nloc = sm.plan.nloc, ncarr = sm.plan.ncarr, n = sm.plan.n;
    const int hd = sm.plan.head, av = sm.plan.avail;
    const int q = phase & 1, bn = b3 == 2 ? 0 : b3 + 1;
    if (tid == 0 && pr.rank == 0) {
      // every CTA is past its reads of these: they serve the next phase's
      // pushes and the barrier after the next two
      pr.ctl->nov[bn == 2 ? 0 : bn + 1] = 0;
      clear_slot(pr, k0 + phase + 3);
    }
    u64 tmin = kNone;
    for (int base = warp * kPer; base < n; base += kWarps * kPer) {
      const int idx = base + lane / L;
      const bool valid = idx < n, loc = idx < nloc;
      int slot = 0;
      int4 en = make_int4(-2, 0, 0, 0);
      if (loc) {
        slot = idx < ncarr ? bd.carr[q][idx] : bd.fresh[q][idx - ncarr];
        en = bd.ent[slot];
      } else if (valid) {
        en = __ldcg((q ? pr.ov[1] : pr.ov[0]) + pr.rank + (int64_t)(idx - nloc) * pr.nranks);
      }
      const int32_t v = en.x, f0 = en.y, deg = en.z & (kMulti ? kSpMask : 0x7fffffff);
      const bool unclaimed = en.z < 0;
      const float pv = __int_as_float(en.w);
      int old = 0;
      if (unclaimed && sl == 0) old = atomicExch(&pr.claim[v], pr.sid);
      const bool vt = kMulti && valid && (en.z & kTgt), vs = kMulti && valid && (en.z & kSeed);
      double msd = 0.0;
      if (vs) msd = __ldcg(&pr.mseed[v]);
      // this lane's arcs (the general form takes them one by one), and the
      // records they name
      int32_t u[K];
      float ci[K], co[K];
      Rec r[K];
      int32_t uf[K];               // multi-source: u's kTgt (it relaxes nothing) and kSeed
      auto fetch = [&](int j, int f) {       // in global memory
        const int32_t e = f0 + f;
        u[j] = pr.indices[e];
        if (kRoi) u[j] = pr.g2r[u[j]];
        ci[j] = pr.rcost ? pr.rcost[e] : pr.cost[pr.rev[e]];
        co[j] = pr.cost[e];
        if (!kGen && !(tick_exact(ci[j]) && tick_exact(co[j]))) sm.inexact = 1;
      };
      auto load = [&](int j) {
        if (!kRoi || u[j] >= 0) {
          r[j] = ld_rec(&rec[u[j]]);
          if (kMulti) {
            uf[j] = r[j].sp & ~kSpMask;
            r[j].sp &= kSpMask;
          }
        }
      };
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int f = sl + j * L;
        r[j].sp = -1;              // no neighbour
        uf[j] = 0;
        if (!kGen && f < deg) {
          if (loc) {
            const int at = slot * kA + f;
            u[j] = bd.rid[at];
            ci[j] = bd.rin[at];
            co[j] = bd.rout[at];
          } else {
            fetch(j, f);
          }
          load(j);
        }
      }
      // Pull.  In ticks alt is the candidate through a settled neighbour's arc;
      // through any other arc it is the least that may yet come that way, and
      // v is final if its key's class ends below all of those.
      u64 alt[K], mx = kNone, hi = 0;
      unsigned open = 0;           // arcs of the second kind
      u64 gx = kNone, gl = kNone;  // general form: the lane's best candidate, its relaxer
      int32_t gu = 0x7fffffff;
      float cin = kInf, mn = kInf, m32 = kInf;
      const u64 pt = !kGen && tick_finite(pv) ? ticks(pv) : 0ull;
      const double pd = kGen ? (double)pv : 0.0;
      if (!kGen) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const bool in = r[j].sp >= 0 && ci[j] < kInf && !(kMulti && (uf[j] & kTgt));
          const bool done = in && (unsigned)(r[j].sp - 2) < (unsigned)phase;      // settled before this phase
          alt[j] = (done ? r[j].lab : T) + (ticks(ci[j]) + pt);
          if (done) mx = alt[j] < mx ? alt[j] : mx;
          if (!done) {
            if (in) open |= 1u << j;
          }
          if (!in) alt[j] = kNone;
        }
      } else {
        for (int f = sl; f < deg; f += L) {
          r[0].sp = -1;
          fetch(0, f);
          load(0);
          if (r[0].sp < 0 || (kMulti && (uf[0] & kTgt))) continue;
          if ((unsigned)(r[0].sp - 2) >= (unsigned)phase) {
            cin = fminf(cin, ci[0]);
            continue;
          }
          const double x = (__longlong_as_double((long long)r[0].lab) + (double)ci[0]) + pd;
          const float a32 = __double2float_rn(x);
          if (a32 < mn || (a32 < kInf && a32 == mn && (r[0].lab < gl || (r[0].lab == gl && u[0] < gu)))) {
            mn = a32;
            gx = ogr_dbits(x);
            gl = r[0].lab;
            gu = u[0];
          }
        }
        m32 = mn;
      }
      // the group's least key, then the tie rule among equal keys: the
      // relaxer with the least (label, id).  In ticks two candidates have one
      // key iff the larger is not above the smaller's round_hi.
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) {
        if (!kGen) {
          const u64 ox = __shfl_xor_sync(kAll, mx, o);
          mx = ox < mx ? ox : mx;
        } else {
          m32 = fminf(m32, __shfl_xor_sync(kAll, m32, o));
          cin = fminf(cin, __shfl_xor_sync(kAll, cin, o));
        }
      }
      bool tied;
      if (!kGen) {
        hi = mx != kNone ? round_hi(mx) : 0ull;
#pragma unroll
        for (int j = 0; j < K; ++j)
          if (!((open >> j) & 1) && alt[j] <= hi && (gx == kNone || r[j].lab < gl || (r[j].lab == gl && u[j] < gu))) {
            gx = alt[j];
            gl = r[j].lab;
            gu = u[j];
          }
        tied = gx != kNone;
      } else {
        tied = gx != kNone && mn == m32;
      }
      const unsigned eq = __ballot_sync(kAll, tied) & gmask;
      int w = eq ? __ffs(eq) - 1 : lane;
      if (__any_sync(kAll, (eq & (eq - 1)) != 0)) {
        u64 xl = tied ? gl : kNone;
        int32_t xu = tied ? gu : 0x7fffffff;
#pragma unroll 1
        for (int o = L / 2; o > 0; o >>= 1) {
          const u64 ol = __shfl_xor_sync(kAll, xl, o);
          const int32_t ou = __shfl_xor_sync(kAll, xu, o);
          if (ol < xl || (ol == xl && ou < xu)) { xl = ol; xu = ou; }
        }
        const unsigned win = __ballot_sync(kAll, tied && gl == xl && gu == xu) & gmask;
        w = win ? __ffs(win) - 1 : lane;
      }
      u64 lv = __shfl_sync(kAll, gx, w);
      int32_t bu = __shfl_sync(kAll, gu, w);
      if (v == pr.src) {
        lv = 0ull;
        m32 = 0.0f;
        hi = 0ull;
        bu = -1;
      }
      if (vs) {
        // a seed's own start comes before every relaxation: it loses only to
        // a strictly smaller float32 value
        if (!kGen) {
          u64 s = 0;
          if (!seed_ticks(msd, &s) || !tick_finite(pv)) sm.inexact = 1;
          s += pt;
          if (lv == kNone || s <= hi) {
            lv = s;
            hi = round_hi(s);
            bu = -1;
          }
        } else {
          const double s = msd + pd;
          const float s32 = __double2float_rn(s);
          if (!(m32 < s32)) {
            lv = ogr_dbits(s);
            m32 = s32;
            bu = -1;
          }
        }
      }
      const int lost = __shfl_sync(kAll, unclaimed && old == pr.sid ? 1 : 0, lane & ~(L - 1));
      const bool mine = valid && lost == 0;
      bool final;
      if (!kGen) {
        if (mine && lv > kTickLimit) sm.inexact = 1;
        bool late = false;         // an open arc's bound within the class (hi may be a seed's)
#pragma unroll
        for (int j = 0; j < K; ++j) late |= ((open >> j) & 1) && alt[j] <= hi;
        final = (__ballot_sync(kAll, late) & gmask) == 0 || lv == T;
      } else {
        final = lv == T || m32 < __double2float_rn((__longlong_as_double((long long)T) + (double)cin) + pd);
      }
      const bool settle = mine && lv != kNone && final;
      const bool carry = mine && !settle;
      if (sl == 0) {
        if (settle) {
          st_rec(&rec[v], lv, (phase + 2) | (kMulti ? en.z & (kTgt | kSeed) : 0), pv);
          pr.par[v] = bu;
          if (v == pr.dst) {
            sm.dst_hit = 1;
            sm.ld = lv;
          }
        } else if (carry) {
          tmin = lv < tmin ? lv : tmin;
          if (loc && unclaimed) bd.ent[slot].z = en.z & 0x7fffffff;
        }
      }
      // Offer the labels of the open neighbours, mark and push the unreached
      // ones.  Carried entries keep their place; new ones (and carried surplus
      // entries) take a free one, or go to the surplus list; entries that
      // leave free theirs.  One turn for all arcs of a lane: its places are
      // counted out once, by two lanes side by side.
      const bool expand = settle && !vt;
      bool self = carry && sl == 0, leaves = loc && !carry && sl == 0;
      int f = sl;
      do {                         // the general form goes round once per arc
        if (kGen) {
          r[0].sp = -1;
          if (expand && f < deg) {
            fetch(0, f);
            load(0);
          }
        }
        bool push[K];
        unsigned mt[K];
        int nt = 0;
        const bool keep = self && loc;
#pragma unroll
        for (int j = 0; j < K; ++j) {
          push[j] = false;
          // open: not settled before this phase (whether it settles in this
          // one must not matter: T is the same whatever the timing)
          if (expand && r[j].sp >= 0 && (unsigned)(r[j].sp - 2) >= (unsigned)phase) {
            u64 ly = kNone;
            if (!kGen) {
              // (whoever reaches u first checks its penalty)
              if (co[j] < kInf) ly = lv + (ticks(co[j]) + ticks(r[j].pen));
            } else {
              const double y = (__longlong_as_double((long long)lv) + (double)co[j]) + (double)r[j].pen;
              if (__double2float_rn(y) < kInf) ly = ogr_dbits(y);
            }
            tmin = ly < tmin ? ly : tmin;
            push[j] = ly != kNone && r[j].sp == 0;
          }
          mt[j] = __ballot_sync(kAll, push[j] || (j == 0 && self && !loc));
          nt += __popc(mt[j]);
        }
        const unsigned mk = __ballot_sync(kAll, keep), mg = __ballot_sync(kAll, leaves);
        if (nt | mk | mg) {
          unsigned p = 0;
          if (lane < 2)
            p = atomicAdd(lane == 0 ? &sm.push[q] : &sm.tail,
                          lane == 0 ? ((unsigned)nt << 12) + (unsigned)__popc(mk) : (unsigned)__popc(mg));
          // (a row of the general form has any length)
          if (kGen && lane == 0 && p >= (1u << 31)) atomicSub(&sm.push[q], (unsigned)nt << 12);
          const unsigned t = __shfl_sync(kAll, p, 1);
          p = __shfl_sync(kAll, p, 0);
          if (leaves) bd.freel[(t + __popc(mg & below)) % (unsigned)kS] = (uint16_t)slot;
          if (keep) bd.carr[q ^ 1][(p & 0xfffu) + __popc(mk & below)] = (uint16_t)slot;
          int at0 = (int)(p >> 12);
#pragma unroll
          for (int j = 0; j < K; ++j) {
            const int at = at0 + __popc(mt[j] & below);
            at0 += __popc(mt[j]);
            bool surplus = false;
            int4 ne = en;
            if ((mt[j] >> lane) & 1) {
              if (push[j]) {
                if (!kGen && !tick_finite(r[j].pen)) sm.inexact = 1;
                const int32_t flags = kMulti ? uf[j] : 0;
                __stcg(&rec[u[j]].sp, 1 | flags);
                ne = make_int4(u[j], (int)(unsigned)r[j].lab, (int)(unsigned)(r[j].lab >> 32) | flags,
                               __float_as_int(r[j].pen));
              }
              if (at < av) {
                const int s = bd.freel[(unsigned)(hd + at) % (unsigned)kS];
                bd.fresh[q ^ 1][at] = (uint16_t)s;
                int4 e = ne;
                if (push[j]) e.z |= 0x80000000;
                bd.ent[s] = e;
              } else {
                // on the surplus list every node stands once: claimed here
                surplus = !push[j] || atomicExch(&pr.claim[u[j]], pr.sid) != pr.sid;
              }
            }
            if (av - at0 < 0) {    // (some of this turn's places are beyond those free)
              const unsigned ms = __ballot_sync(kAll, surplus);
              if (ms) {
                int b = 0;
                if (lane == 0) {
                  b = atomicAdd(&pr.ctl->nov[bn], __popc(ms));
                  atomicAdd(&sm.nov_out, __popc(ms));
                }
                b = __shfl_sync(kAll, b, 0);
                if (surplus) __stcg((q ? pr.ov[0] : pr.ov[1]) + b + __popc(ms & below), ne);
              }
            }
          }
        }
        self = leaves = false;
        f += L;
      } while (kGen && __any_sync(kAll, expand && f < deg));
    }
    tmin = warp_min_u64(tmin);
    if (lane == 0) sm.wmin[warp] = tmin;
    __syncthreads();
    // the phase's writes are done: hand in, fetch the new entries' rows, wait
    const unsigned pushed = sm.push[q];
    const int nf = min((int)(pushed >> 12), av), nk = (int)(pushed & 0xfffu);
    if (warp == 0) {
      u64 t = warp_min_u64(lane < kWarps ? sm.wmin[lane] : kNone);
      if (lane == 0) {
        const unsigned nout = (unsigned)sm.nov_out;
        if (!kGen && sm.inexact) t = 0;
        arrive(pr, sm, k0 + phase + 1,
               kArrive + (sm.dst_hit ? kDst : 0ull) + kOut * (nout < kMostOut ? nout : kMostOut) +
                   kCount * (u64)(nout + (unsigned)(nf + nk)),
               t);
      }
    }
    const int solo = pr.nranks == 1 ? 0 : 1;   // thread 0's warp waits if there is a team
    if (!kGen && warp >= solo) {
      for (int i = (tid - 32 * solo) / L; i < nf; i += (kThreads - 32 * solo) / L) {
        const int s = bd.fresh[q ^ 1][i];
        const int f0 = bd.ent[s].y, deg = bd.ent[s].z & (kMulti ? kSpMask : 0x7fffffff);
        int32_t u[K];
        float ci[K], co[K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
          if (sl + j * L >= deg) continue;
          const int32_t e = f0 + sl + j * L;
          u[j] = pr.indices[e];
          ci[j] = pr.rcost ? pr.rcost[e] : pr.cost[pr.rev[e]];
          co[j] = pr.cost[e];
        }
#pragma unroll
        for (int j = 0; j < K; ++j) {
          if (sl + j * L >= deg) continue;
          if (kRoi) u[j] = pr.g2r[u[j]];
          if (!(tick_exact(ci[j]) && tick_exact(co[j]))) sm.inexact = 1;
          const int at = s * kA + sl + j * L;
          bd.rid[at] = u[j];
          bd.rin[at] = ci[j];
          bd.rout[at] = co[j];
        }
      }
    }
    if (tid == 0) {
      const long long c0 = clock64();
      sm.ok = 1;
      u64 a = 0, t = 0;
      const float carried = n > 0 ? __fdividef((float)nk, (float)n) : 0.5f;
      await(pr, sm, k0 + phase + 1, a, t);
      out.wait += clock64() - c0;
      if (sm.ok)
        plan(phase + 1, bn, nf, nk, carried, a, t);
      else
        sm.plan.verdict = kTimedOut;
      sm.push[q ^ 1] = 0;
      out.examined += (u64)n;
      sm.nov_out = 0;
    }
    __syncthreads();
    ++phase;
    b3 = bn;
  }
  out.status = verdict == kEmpty         ? OGR_NO_PATH
               : verdict == kCapped      ? OGR_ERR_ITER_CAP
               : verdict == kTimedOut    ? OGR_ERR_TIMEOUT
               : verdict == kInexactSeen ? kStInexact
                                         : OGR_OK;
  out.found = verdict == kFound || verdict == kFoundEarly;
  out.exhausted = verdict == kEmpty;
  // a search that stops on dst did no work in its last phase
  out.phases = (verdict == kFoundEarly || verdict == kTimedOut ? phase : phase + 1) - (kGen ? sm.first : 0);
  out.clocks = clock64() - c_start;
  out.ld = sm.ld;
  return out;
}

// The forms that are rarely needed, out of line.
template <int L, int K, bool kGen, bool kMulti, bool kRoi>
__device__ __noinline__ void run_rare(const Problem* ppr, char* smem, int k0, Outcome* out) {
  const Problem pr = *ppr;
  Head& sm = *reinterpret_cast<Head*>(smem);
  Body<L * K>& bd = *reinterpret_cast<Body<L * K>*>(smem + kHeadBytes);
  *out = run_phases<L, K, kGen, kMulti, kRoi>(pr, sm, bd, kGen ? k0 - sm.first : k0);
}

// The longest row that is searched in ticks.
constexpr int kMaxRow = 32;

// The search with L lanes of K arcs per entry if the rows (of at most max_deg
// arcs) allow it, else in the form that takes them; labels in ticks, or (only
// and always in the general form) in doubles.  A kernel holds one form inline
// and is launched by the lattice's longest row (ogr_full::row_for): with all
// four in it, chosen by max_deg, registers spilled and every search was 5 to
// 16 % slower; with the larger ones out of line still 2 to 11 %.
template <int L, int K, bool kMulti, bool kRoi>
__device__ __forceinline__ Outcome run_search(const Problem& pr, char* smem, int k0, int max_deg, bool in_ticks) {
  if (in_ticks && max_deg <= L * K) {
    Head& sm = *reinterpret_cast<Head*>(smem);
    Body<L * K>& bd = *reinterpret_cast<Body<L * K>*>(smem + kHeadBytes);
    return run_phases<L, K, false, kMulti, kRoi>(pr, sm, bd, k0);
  }
  Outcome o;
  const Problem p = pr;
  if (!in_ticks)
    run_rare<16, 1, true, kMulti, kRoi>(&p, smem, k0, &o);
  else
    run_rare<32, 1, false, kMulti, kRoi>(&p, smem, k0, &o);
  return o;
}

// A search that met a value ticks cannot hold (out: its outcome, k0: barriers
// it has used) goes on in doubles from the start of phase p, in which it did:
// what settled before stays settled, its label converted (exact, being below
// 2^52 ticks).  The frontier at p is entered in surplus list 0: what p settled,
// the seeds, and every reached node with a neighbour settled before p that
// relaxes it.  A node that only p reached is unreached again, for its neighbour
// may not settle in doubles.  (Other CTAs convert at the same time; the test of
// a neighbour says the same before and after.)  This CTA's nodes are first,
// first + step, ....  Uses claim stamp sid + 1; *k0 is brought up to date.
//
// Out of line, and called once, so that the search in ticks keeps its
// registers.  Two long searches of 600x400x12 whose labels pass 2^22 late took
// 16.6 ms begun anew in doubles, and 9.9 this way.
template <bool kMulti, bool kRoi>
__device__ __noinline__ void go_over(const Problem* ppr, char* smem, int* k0, int64_t first, int64_t step, Outcome* out) {
  Problem pr = *ppr;
  Head& sm = *reinterpret_cast<Head*>(smem);
  const int tid = threadIdx.x;
  const bool leader = pr.rank == 0 && tid == 0;
  const int p = out->phases - 2, b = *k0;
  const unsigned long long T = sm.plan.T;
  pr.sid += 1;
  for (int64_t i = first; i < pr.R; i += step) {
    const Rec x = ld_rec(&pr.rec[i]);
    const int32_t s = kMulti ? x.sp & kSpMask : x.sp, flags = kMulti ? x.sp & ~kSpMask : 0;
    if (s == 0) continue;
    if (s >= 2 && s - 2 < p) {
      st_rec(&pr.rec[i], ogr_dbits(label_value<true>(x.lab)), 2 | flags, x.pen);
      continue;
    }
    const int32_t g = kRoi ? pr.roi[i] : (int32_t)i, f0 = pr.indptr[g], f1 = pr.indptr[g + 1];
    bool in = s >= 2 || (flags & kSeed);
    for (int32_t e = f0; e < f1 && !in; ++e) {
      const int32_t u = kRoi ? pr.g2r[pr.indices[e]] : pr.indices[e];
      if (u < 0) continue;
      const int32_t sp = __ldcg(&pr.rec[u].sp), su = kMulti ? sp & kSpMask : sp;
      in = su >= 2 && su - 2 < p && !(kMulti && (sp & kTgt)) &&
           (pr.rcost ? pr.rcost[e] : pr.cost[pr.rev[e]]) < __int_as_float(0x7f800000);
    }
    __stcg(reinterpret_cast<int4*>(&pr.rec[i]), make_int4(f0, f1 - f0, (in ? 1 : 0) | flags, __float_as_int(x.pen)));
    if (in) {
      pr.claim[i] = pr.sid;
      __stcg(&pr.ov[0][atomicAdd(&pr.ctl->kept, 1)], make_int4((int)i, f0, (f1 - f0) | flags, __float_as_int(x.pen)));
    }
  }
  __syncthreads();
  if (tid == 0) {
    sm.ok = 1;
    sm.first = kFirstOver;
    sm.max_phase = max(sm.max_phase - p, 0) + kFirstOver;
    if (leader) clear_slot(pr, b + 2);       // the last two barriers' words are used ones
    arrive(pr, sm, b, kArrive, kNone);
    await(pr, sm, b);
    unsigned long long a = kArrive, t = kNone;
    if (leader) {
      clear_slot(pr, b + 3);
      const int n = __ldcg(&pr.ctl->kept);
      pr.ctl->nov[0] = n;
      pr.ctl->nov[1] = 0;
      pr.ctl->nov[2] = 0;
      if (!kMulti && __ldcg(&pr.rec[pr.dst].sp) >= 2) a += kDst;
      a += kOut * (unsigned long long)(n < (int)kMostOut ? n : (int)kMostOut) + kCount * (unsigned long long)n;
      // T of phase p bounds its labels; above 2^53 their two sums may have rounded
      t = ogr_dbits((double)(T > kTickLimit ? (T - 16) & ~15ull : T) * (1.0 / 1073741824.0));
    }
    if (sm.ok) {
      arrive(pr, sm, b + 1, a, t);
      await(pr, sm, b + 1);
    }
  }
  __syncthreads();
  const int ok = sm.ok;
  __syncthreads();
  if (!ok) {
    out->status = OGR_ERR_TIMEOUT;
    out->found = out->exhausted = false;
    *k0 = b + 2;
    return;
  }
  const unsigned long long examined = out->examined;
  const long long wait = out->wait, clocks = out->clocks;
  run_rare<16, 1, true, kMulti, kRoi>(&pr, smem, b + 1, out);
  *k0 = b + 1 + out->phases;
  out->phases += p;
  out->examined += examined;
  out->wait += wait;
  out->clocks += clocks;
}

// Statistics of a finished search, added by this CTA for the nodes first,
// first + step, ...: rows scanned and nodes popped by the heap search before
// dst (exhausted or multi-source: by the time it runs empty).
template <bool kMulti, bool kRoi>
__device__ __forceinline__ void count_work(const Problem& pr, const Outcome& o, int64_t first, int64_t step, unsigned long long* stats) {
  unsigned long long arcs = 0, pops = 0;
  for (int64_t i = first; i < pr.R; i += step) {
    const int32_t r = (int32_t)i;
    const Rec x = ld_rec(&pr.rec[r]);
    if ((kMulti ? x.sp & kSpMask : x.sp) < 2) continue;
    if (kMulti) {
      ++pops;
      if (x.sp & kTgt) continue;
    } else {
      if (!(o.exhausted || x.lab < o.ld || (x.lab == o.ld && r < pr.dst))) continue;
      ++pops;
    }
    const int32_t g = kRoi ? pr.roi[r] : r;
    arcs += (unsigned long long)(pr.indptr[g + 1] - pr.indptr[g]);
  }
  arcs = (unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)arcs);
  pops = (unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)pops);
  if ((threadIdx.x & 31) == 0 && pops) {
    atomicAdd(&stats[0], arcs);
    atomicAdd(&stats[1], pops);
  }
}

// Walks the parents from node c into out[0..], last node first, by one warp;
// returns the nodes written, *end the node the walk stopped at (-1: at the
// start of the path).  Paths run straight for long stretches, so the lanes
// guess the next 31 parents at the last step's stride and a run of right
// guesses costs one round trip (a walk of 350 parents took 144 us node by
// node).
__device__ inline int walk_parents(const int32_t* par, int32_t c, int32_t R, int limit, int32_t* out, int32_t* end) {
  const int lane = threadIdx.x & 31;
  int len = 0;
  int32_t delta = 0;
  while (c != -1 && len < limit) {
    const int64_t gl = (int64_t)c + (int64_t)lane * delta;
    const bool in = gl >= 0 && gl < R;
    const int32_t g = in ? (int32_t)gl : -2;
    const int32_t p = in ? __ldcg(&par[g]) : -3;
    const int32_t before = __shfl_up_sync(0xffffffffu, p, 1);
    const unsigned good = __ballot_sync(0xffffffffu, lane == 0 || (in && before == g));
    const int run = min(good == 0xffffffffu ? 32 : __ffs(~good) - 1, limit - len);
    if (lane < run) out[len + lane] = g;
    len += run;
    const int32_t last = __shfl_sync(0xffffffffu, g, run - 1);
    c = __shfl_sync(0xffffffffu, p, run - 1);
    delta = c - last;
  }
  *end = c;
  return len;
}

}  // namespace ogr_phase
