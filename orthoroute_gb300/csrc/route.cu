// A6–A8: per-net ROI extraction, exact ROI shortest path, backtrace, and the
// commit / rip-up scatter.  A team of CTAs owns one net's search (phases.cuh).
//
// ROI (extract_roi_bfs, unified_pathfinder.py:2257-2384): level-synchronous
// bidirectional BFS.  Within one wave step the reference's marks are a set
// function of the frontier (unseen -> wave mark, other wave -> 3 and
// "met"), so claiming nodes with atomics yields the same seen set,
// meeting depth and early stop.  The ROI is then compacted in ascending
// global id order (np.where) by scanning the BFS bounding box, and truncated
// to max_roi_nodes with the reference's must-keep swap.  The BFS does not read
// costs, so a routing pass extracts the ROIs of all its nets in parallel on
// many SMs before the sequential part starts (roi_batch_kernel).
//
// Search (SimpleDijkstra.find_path_roi, :2451-2548): phases.cuh on the ROI's
// nodes, by a team of CTAs.  One SM searched an ROI in phases of 11 to 22 us
// (a few hundred to two thousand entries to examine in each); a team shares
// them out, so a phase costs little more than its chain of round trips and
// the team's barrier.
//
// ogr_route_pass runs the reference's per-net sequence (_route_all,
// :7949-8449: rip-up, ROI search, one larger-ROI retry while the pass has
// fallbacks left, commit) for a whole ordered list of nets in one launch,
// with every net's current path kept in a device-resident store.
#include <atomic>

#include "common.cuh"
#include "fullgraph.cuh"
#include "phases.cuh"
#include "roibox.h"

namespace {

using ogr_phase::kThreads;
using ogr_phase::kWarps;
constexpr int kSub = 16;                       // lanes per node (ROI BFS)
constexpr int kBfsThreads = 768;               // of the kernel that only extracts ROIs, one per CTA
constexpr int kClusterThreads = 512;           // of a cluster's CTA that extracts one ROI

// Accepted and kept for callers (ogr_search_lanes); the search fits its lanes
// to the lattice's rows, and results never depended on it.
thread_local int g_search_lanes = 4;

// Nets a disjoint-ROI window may skip over to take later disjoint ones
// (ogr_window_lookahead; 0 = consecutive nets only).
thread_local int g_window_look = 8;

constexpr int kMaxViaNodes = 4096;
constexpr int kMaxSkip = 16;                   // nets a window may skip over (look-ahead)
// CTAs of one ROI search (fewer where a window's members share the SMs): half
// the SMs, so that two jobs' searches fit side by side.  A team's phase of an
// ROI of 50,000 nodes on 600x400x12: 8.7 us with 8 CTAs, 6.5 with 16, 5.3
// with 32, 4.5 with 76 and with 152; ROIs of 14,000 nodes: 4.4, 3.9, 3.8, 3.7.
constexpr int kTeam = 76;
constexpr int kLoneNodes = 512;                // below it one CTA

// Control words of one search slot, kept between searches (sid) or zero at
// the start of each (team).
struct SlotCtl {
  ogr_phase::Ctl team;
  int32_t sid;               // searches so far: the claim stamp
  int32_t merr;              // multi-source: a bad or repeated seed / target
};

// A search slot: the ROI's node arrays, the global->ROI map, and (route
// workspace only) the BFS.
struct Ws {
  int32_t* seen;
  int32_t* g2r;
  int32_t* q[4];             // BFS queues; the search's first surplus list lies over them
  int32_t* roi;
  ogr_phase::Rec* rec;
  int32_t* par;
  int32_t* claim;
  int32_t nclaim;            // nodes that claim[] has words for
  int4* ov[2];
  SlotCtl* ctl;
  char* win1;                // control block of a pass without windows
  int64_t* result;           // [0] status, [1] path length, [2] fallbacks used, [3] ROI size
  int64_t qcap;
  unsigned spin;             // bounds of a search: polls of a wait, settle phases (0: what R allows)
  int32_t max_phases;
};

// Seeds and targets of a multi-source multi-sink search
// (find_path_multisource_multisink, unified_pathfinder.py:2550-2659), global
// ids with FP64 costs, mapped to ROI-indexed arrays inside the search.
struct MultiSeeds {
  const int32_t* seeds;
  const double* seed_cost;
  int32_t nseeds;
  const int32_t* targets;
  const double* target_cost;
  int32_t ntargets;
  double* init;    // [R] seed cost before the node penalty, kNoTerm bits for other nodes
  double* tcost;   // [R] target cost, kNoTerm bits for other nodes
};
constexpr unsigned long long kNoTerm = 0x7ff8deadbeef0001ull;

__host__ __device__ constexpr size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

constexpr size_t kWin1Bytes = 4096;

// Bytes of a route workspace for n nodes.
__host__ __device__ constexpr size_t ws_bytes_for(size_t n) {
  return 5 * round256(4 * n) + 3 * round256(16 * n) + round256(sizeof(SlotCtl)) +
         kWin1Bytes + round256(64);
}

__host__ inline size_t ws_layout(int32_t N, char* base, Ws* w) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = base ? base + off : nullptr;
    off += round256(bytes);
    return p;
  };
  const size_t n = (size_t)N;
  Ws t{};
  t.seen = (int32_t*)take(4 * n);
  t.g2r = (int32_t*)take(4 * n);
  t.roi = (int32_t*)take(4 * n);
  t.par = (int32_t*)take(4 * n);
  t.claim = (int32_t*)take(4 * n);
  t.nclaim = N;
  t.rec = (ogr_phase::Rec*)take(16 * n);
  t.ov[0] = (int4*)take(16 * n);
  t.ov[1] = (int4*)take(16 * n);
  for (int i = 0; i < 4; ++i) t.q[i] = (int32_t*)t.ov[0] + i * n;   // the queues are free while the search runs
  t.ctl = (SlotCtl*)take(sizeof(SlotCtl));
  t.win1 = take(kWin1Bytes);
  t.result = (int64_t*)take(64);
  t.qcap = (int64_t)n;
  t.spin = ogr_full::wait_limit();
  t.max_phases = ogr_full::phase_limit();
  if (w) *w = t;
  return off;
}

// A search-only slot for the window pass: the global->ROI map and ROI-sized
// arrays (the ROI comes from the batched extraction, so no BFS state).
__host__ __device__ inline size_t ws_slot_layout(int32_t N, int32_t Rmax, char* base, Ws* w) {
  const size_t n = (size_t)N, r = (size_t)Rmax;
  const size_t sz[7] = {4 * n, 16 * r, 4 * r, 4 * r, 16 * r, 16 * r, sizeof(SlotCtl)};
  char* p[7];
  size_t off = 0;
  for (int i = 0; i < 7; ++i) {
    p[i] = base ? base + off : nullptr;
    off += round256(sz[i]);
  }
  if (w) {
    Ws t{};
    t.g2r = (int32_t*)p[0];
    t.rec = (ogr_phase::Rec*)p[1];
    t.par = (int32_t*)p[2];
    t.claim = (int32_t*)p[3];
    t.nclaim = Rmax;
    t.ov[0] = (int4*)p[4];
    t.ov[1] = (int4*)p[5];
    t.ctl = (SlotCtl*)p[6];
    *w = t;
  }
  return off;
}

// A BFS-only slot for the batched ROI extraction: seen[N] + 4 queues.
struct BfsSlot {
  int32_t* seen;
  int32_t* q[4];
  int64_t qcap;
};

__host__ inline size_t bfs_slot_bytes(int32_t N, int64_t qcap) {
  return round256(4 * (size_t)N) + 4 * round256(4 * (size_t)qcap);
}

__host__ __device__ inline BfsSlot bfs_slot_at(char* base, int32_t N, int64_t qcap) {
  BfsSlot s;
  size_t off = 0;
  s.seen = (int32_t*)(base + off);
  off += round256(4 * (size_t)N);
  for (int i = 0; i < 4; ++i) {
    s.q[i] = (int32_t*)(base + off);
    off += round256(4 * (size_t)qcap);
  }
  s.qcap = qcap;
  return s;
}

// Per-stage cycle counters of the ROI searches (a tracing aid, read with
// ogr_search_profile; thread 0 of a team's first CTA): [0] BFS waves, [1] ROI
// compaction, [2] search init, [3] phases, [4] of these waiting for the team,
// [5] rip-up and commit, [6] window formation (CTA 0 of a pass), [7] statistics
// + backtrace, [8] cleanup, [9] searches, [10] phases, [11] BFS
// waves run, [12] ROI nodes, [13] entries examined, [14] ROIs taken from the
// batched extraction, [15] searches that left the form of their kernel (longer
// rows, or values that ticks cannot hold).
__device__ unsigned long long g_stage[16];

struct Shared {
  int s_cnt[32];
  int s_off[32];
  int nq[4];
  int seen_count;
  int met;
  int flags[3];    // of a BFS wave
  int overflow;
  int bx0, bx1, by0, by1;
  int pos_src, pos_dst;
  int R;
  int status;
};

struct StageClock {
  long long t;
  __device__ void start() { t = clock64(); }
  __device__ void mark(int k) {
    if (threadIdx.x == 0) {
      const long long now = clock64();
      atomicAdd(&g_stage[k], (unsigned long long)(now - t));
      t = now;
    }
  }
};

// ---- ROI extraction ---------------------------------------------------------
// Cuts the ROI of sh.R nodes in out[0..out_cap) to max_roi_nodes; sh.pos_src /
// sh.pos_dst are the terminals' positions.  Thread 0; sh.status =
// OGR_ERR_CAPACITY when a queue overflowed or out is too small.
__device__ void roi_finish(Shared& sh, const ogr_net_args& a, int32_t* out, int32_t out_cap) {
  if (threadIdx.x != 0) return;
  const int32_t src = a.src, dst = a.dst;
  int R = sh.R;
  if (R > a.max_roi_nodes) {
    // Must-keep swap (extract_roi_bfs :2359-2379): the positions of src/dst
    // in ascending order; each one beyond the cut swaps with slot 0 / 1.
    int kp[2];
    int32_t kn[2];
    int nk = 0;
    if (src == dst) {
      kp[0] = sh.pos_src; kn[0] = src; nk = 1;
    } else {
      const bool s_first = sh.pos_src < sh.pos_dst;
      kp[0] = s_first ? sh.pos_src : sh.pos_dst; kn[0] = s_first ? src : dst;
      kp[1] = s_first ? sh.pos_dst : sh.pos_src; kn[1] = s_first ? dst : src;
      nk = 2;
    }
    for (int k = 0; k < nk; ++k)
      if (kp[k] >= a.max_roi_nodes) out[k] = kn[k];
    R = a.max_roi_nodes;
  }
  sh.R = R;
  if (sh.overflow || R > out_cap) sh.status = OGR_ERR_CAPACITY;
  atomicAdd(&g_stage[12], (unsigned long long)R);
}

// Shared memory of a BFS: the mail of a cluster's CTAs, two queues (this wave's
// and the next one's), then the marks of the box around both terminals, two
// bits a cell (1: seen from src, 2: from dst; both: where the waves met).
constexpr int kBfsCtas = 8;                    // CTAs of a cluster that extracts one ROI
struct BfsMail {
  int4 in[2][kBfsCtas];                        // from each CTA: nodes for this one, new nodes, flags
  int out[kBfsCtas];                           // nodes found so far for each CTA
};
constexpr int kBfsQ = 8192;
constexpr int kBfsSeg = kBfsQ / kBfsCtas;      // of a queue, one CTA's finds
constexpr size_t kBfsHead = 512;
constexpr size_t kBfsBitsAt = kBfsHead + 2 * kBfsQ * sizeof(int32_t);
constexpr int kBfsWords = (int)((ogr_phase::kSmemBytes - kBfsBitsAt) / 4);
static_assert(sizeof(BfsMail) <= kBfsHead && 2 * kBfsQ <= 16384, "mail and queues");
constexpr int kMet = 1, kLeft = 2, kOverflow = 4;

// Another CTA's copy of a variable in shared memory.
__device__ __forceinline__ unsigned peer_addr(const void* p, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
// *addr |= bit if on; the word before (all ones if not on).
__device__ __forceinline__ unsigned peer_or(unsigned addr, unsigned bit, bool on) {
  unsigned old;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.u32 %0, 0xffffffff;\n"
      " @p atom.relaxed.cluster.shared::cluster.or.b32 %0, [%1], %2;\n}"
      : "=r"(old) : "r"(addr), "r"(bit), "r"((unsigned)on) : "memory");
  return old;
}
__device__ __forceinline__ unsigned peer_ld(unsigned addr) {
  unsigned v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void peer_st(unsigned addr, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void peer_st(unsigned addr, int4 v) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ int peer_add(unsigned addr, int v) {
  int old;
  asm volatile("atom.relaxed.cluster.shared::cluster.add.s32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ void peer_min(unsigned addr, int v) {
  int old;
  asm volatile("atom.relaxed.cluster.shared::cluster.min.s32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void peer_max(unsigned addr, int v) {
  int old;
  asm volatile("atom.relaxed.cluster.shared::cluster.max.s32 %0, [%1], %2;" : "=r"(old) : "r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
// The CTA that keeps a word of the marks, whose queue its cells go to.
__device__ __forceinline__ unsigned bfs_owner(int wd) { return ((unsigned)wd * 0x9e3779b1u) >> 29; }
static_assert(kBfsCtas == 8, "three bits of the hash");

// Bidirectional BFS from src/dst on a box in shared memory; writes the ROI
// (ascending id, truncated with the must-keep swap) into out[0..out_cap) and
// its size into sh.R.  False: the search left the box (the caller takes
// roi_build_large).
//
// Both terminals' waves go on together.  A cell that both find in one step
// goes to one queue only: the ROI is what either has seen, the cell's
// neighbours are found by whichever has it, and the step at which the waves
// meet is the same (the second of two marks of a cell tells).
//
// A step is two dependent round trips (row bounds, row) and the marks, which
// never leave the SM; the lanes of a node wait for their row together.  With
// the marks as compare-and-swaps in global memory (a third round trip and an
// atomic per arc) an ROI of 50,000 nodes on 600x400x12 took 1,352 us and its
// compaction 250; one terminal's wave after the other 550 and 55.
//
// kCluster: by the kBfsCtas CTAs of a cluster.  A word of the marks has an
// owner, whose copy counts; the others' copies only spare them asking twice.
// Whoever marks a cell first sends it to its owner's queue, and the counts of
// what was sent cross with the flags at the end of the step.  The same ROI
// then takes 237 us and 18 (8 CTAs of 512 threads, 4 lanes a node; 8 lanes:
// 277; 1,024 threads: 217, but 14,000 nodes 106 instead of 90; one CTA 165).
// Owners by column, which keeps most marks in their CTA, were no faster.
template <bool kCluster, int kLanes, int kArcs>
__device__ bool roi_build_box(Shared& sh, const ogr_graph& g, const ogr_net_args& a, int32_t* const* q, int64_t qcap,
                              int32_t* out, int32_t out_cap, char* smem, StageClock& clk, int rank) {
  constexpr int kNodes = 32 / kLanes;          // a warp's nodes at a time
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int32_t src = a.src, dst = a.dst, plane = nx * ny;
  const int32_t* __restrict__ indptr = g.indptr;
  const int32_t* __restrict__ indices = g.indices;
  const OgrDiv by_plane((unsigned)(nx * ny)), by_nx((unsigned)nx);
  BfsMail& mail = *reinterpret_cast<BfsMail*>(smem);
  int32_t* sq = reinterpret_cast<int32_t*>(smem + kBfsHead);
  unsigned* marks = reinterpret_cast<unsigned*>(smem + kBfsBitsAt);
  auto coord = [&](int32_t v, int& x, int& y, int& z) {
    z = (int)by_plane((unsigned)v);
    const unsigned r = (unsigned)v - (unsigned)z * by_plane.d;
    y = (int)by_nx(r);
    x = (int)(r - (unsigned)y * by_nx.d);
  };
  int sx, sy, sz, dx, dy, dz;
  coord(src, sx, sy, sz);
  coord(dst, dx, dy, dz);
  const ogr_box::Box box = ogr_box::fit(nx, ny, nz, sx, sy, dx, dy, a.bfs_max_depth, kBfsWords);
  if (box.words == 0) return false;
  const int X0 = box.x0, Y0 = box.y0, BW = box.w, BH = box.h, RW = box.row, NW = box.words;
  for (int i = tid; i < NW; i += nt) marks[i] = 0u;
  if (tid < kBfsCtas) {
    mail.out[tid] = 0;
    mail.in[0][tid] = make_int4(kCluster && rank == 0 && tid == 0 ? 2 : 0, 0, 0, 0);
  }
  if (tid == 0) {
    sq[0] = src;
    sq[1] = (int32_t)((unsigned)dst | 0x80000000u);
    sh.nq[0] = 2;                              // (wave w takes nq[w % 3] entries, sets flags[w % 3])
    sh.nq[1] = sh.nq[2] = 0;
    sh.flags[0] = sh.flags[1] = sh.flags[2] = 0;
    sh.overflow = 0;
    sh.pos_src = -1;
    sh.pos_dst = -1;
    sh.bx0 = min(sx, dx); sh.bx1 = max(sx, dx);
    sh.by0 = min(sy, dy); sh.by1 = max(sy, dy);
  }
  __syncthreads();
  if (tid == 0) {
    const int xs = sx - X0, xd = dx - X0;
    if (src != dst) marks[(sz * BH + (sy - Y0)) * RW + (xs >> 4)] |= 1u << (2 * (xs & 15));
    marks[(dz * BH + (dy - Y0)) * RW + (xd >> 4)] |= 2u << (2 * (xd & 15));
  }
  int depth = 0, meet = -1, par = 0, slot = 0;
  int64_t seen = src != dst ? 2 : 1;
  int64_t total = 2;
  int lx0 = 1 << 30, lx1 = -1, ly0 = 1 << 30, ly1 = -1;
  if constexpr (kCluster) cluster_sync(); else __syncthreads();
  while (depth < a.bfs_max_depth && total > 0) {
    const int nslot = slot == 2 ? 0 : slot + 1;
    int n, before[kBfsCtas];                   // cluster: entries before each CTA's segment
    if constexpr (kCluster) {
      n = 0;
#pragma unroll
      for (int k = 0; k < kBfsCtas; ++k) {
        before[k] = n;
        n += mail.in[par][k].x;
      }
    } else {
      n = (int)total;
      if (tid == 0) {                          // (both last read two waves ago)
        sh.nq[nslot == 2 ? 0 : nslot + 1] = 0;
        sh.flags[nslot] = 0;
      }
    }
    int flags = 0;
    for (int base = warp * kNodes; base < n; base += nw * kNodes) {
      const int i = base + lane / kLanes;
      int32_t u = 0, f = 0, f1 = 0;
      unsigned mark = 1;
      if (i < n) {
        int at = i;
        if constexpr (kCluster) {
          int k = 0, b = 0;
#pragma unroll
          for (int c = 1; c < kBfsCtas; ++c)
            if (i >= before[c]) { k = c; b = before[c]; }
          at = k * kBfsSeg + i - b;
        }
        int32_t x;
        if (kCluster || at < kBfsQ) x = sq[par * kBfsQ + at];
        else x = at < qcap ? q[par][at] : q[par + 2][at - qcap];
        mark = 1u + ((unsigned)x >> 31);
        u = x & 0x7fffffff;
        f = indptr[u] + lane % kLanes;
        f1 = indptr[u + 1];
      }
      // (in the shadow of the row bounds' load)
      int ux, uy, uz;
      coord(u, ux, uy, uz);
      const int32_t ur = u - uz * plane;
      const int ubx = ux - X0, uby = uy - Y0;
      while (__any_sync(0xffffffffu, f < f1)) {
        int32_t v[kArcs];
        int wd[kArcs];
        unsigned old[kArcs];
        int cx[kArcs], cy[kArcs];
#pragma unroll
        for (int j = 0; j < kArcs; ++j) {
          const int32_t e = f + kLanes * j;
          v[j] = e < f1 && !(g.blocked != nullptr && g.blocked[e]) ? indices[e] : -1;
        }
#pragma unroll
        for (int j = 0; j < kArcs; ++j) {
          // the next cell, or another layer of the same one
          const int32_t d = v[j] - u;
          int bx = ubx, by = uby;
          const int z = (int)by_plane((unsigned)max(v[j], 0));
          const int32_t r = v[j] - z * plane;
          if (r != ur) {
            if (d == 1 || d == -1) bx += d;
            else if (d == nx || d == -nx) by += d > 0 ? 1 : -1;
            else bx = -1;          // (an arc of no lattice: the caller takes the large form)
            if ((unsigned)(bx + X0) >= (unsigned)nx || (unsigned)(by + Y0) >= (unsigned)ny) bx = -1;
          }
          if (v[j] >= 0 && ((unsigned)bx >= (unsigned)BW || (unsigned)by >= (unsigned)BH)) {
            flags |= kLeft;
            v[j] = -1;
          }
          cx[j] = bx;
          cy[j] = by;
          wd[j] = v[j] >= 0 ? (z * BH + by) * RW + (bx >> 4) : 0;
          old[j] = v[j] >= 0 ? *(volatile unsigned*)&marks[wd[j]] : 0xffffffffu;
        }
#pragma unroll
        for (int j = 0; j < kArcs; ++j) {
          const unsigned bit = mark << (2 * (cx[j] & 15));
          bool on = !(old[j] & bit);
          if constexpr (kCluster) {
            const unsigned o = bfs_owner(wd[j]);
            if (on && o != (unsigned)rank) on = !(atomicOr(&marks[wd[j]], bit) & bit);
            old[j] = peer_or(peer_addr(&marks[wd[j]], o), bit, on);
          } else if (on) {
            old[j] = atomicOr(&marks[wd[j]], bit);
          }
        }
#pragma unroll
        for (int j = 0; j < kArcs; ++j) {
          const unsigned cell = old[j] >> (2 * (cx[j] & 15)) & 3u;
          const bool fresh = cell == 0;
          if (cell == 3u - mark) flags |= kMet;
          const int32_t x = (int32_t)((unsigned)v[j] | (mark - 1u) << 31);
          if constexpr (kCluster) {
            if (fresh) {
              const unsigned o = bfs_owner(wd[j]);
              const int p = atomicAdd(&mail.out[o], 1);
              if (p < kBfsSeg) peer_st(peer_addr(&sq[(par ^ 1) * kBfsQ + rank * kBfsSeg + p], o), x);
              else flags |= kLeft;             // (more than a queue holds)
            }
          } else {
            if (fresh) {
              lx0 = min(lx0, cx[j]); lx1 = max(lx1, cx[j]);
              ly0 = min(ly0, cy[j]); ly1 = max(ly1, cy[j]);
            }
            const unsigned m = __ballot_sync(0xffffffffu, fresh);
            if (m) {
              int p = 0;
              if (lane == 0) p = atomicAdd(&sh.nq[nslot], __popc(m));
              p = __shfl_sync(0xffffffffu, p, 0) + __popc(m & ((1u << lane) - 1u));
              if (fresh) {
                if (p < kBfsQ) sq[(par ^ 1) * kBfsQ + p] = x;
                else if (p < qcap) q[par ^ 1][p] = x;
                else if (p < 2 * qcap) q[(par ^ 1) + 2][p - qcap] = x;
                else flags |= kOverflow;
              }
            }
          }
        }
        f += kLanes * kArcs;
      }
    }
    flags = __reduce_or_sync(0xffffffffu, flags);
    if (lane == 0 && flags) atomicOr(&sh.flags[slot], flags);
    __syncthreads();
    if constexpr (kCluster) {
      if (tid < kBfsCtas) {
        const int mine = mail.out[tid];
        const int all = __reduce_add_sync((1u << kBfsCtas) - 1u, mine);
        mail.out[tid] = 0;
        peer_st(peer_addr(&mail.in[par ^ 1][rank], tid), make_int4(min(mine, kBfsSeg), all, sh.flags[slot], 0));
        if (tid == 0) sh.flags[nslot] = 0;
      }
      cluster_sync();
      total = 0;
      flags = 0;
      for (int k = 0; k < kBfsCtas; ++k) {
        const int4 x = mail.in[par ^ 1][k];
        total += x.y;
        flags |= x.z;
      }
    } else {
      total = sh.nq[nslot];
      flags = sh.flags[slot];
    }
    par ^= 1;
    slot = nslot;
    seen += total;
    ++depth;
    if (tid == 0 && rank == 0) atomicAdd(&g_stage[11], 1ull);
    if (flags & kLeft) return false;           // (the same in every thread, and in every CTA)
    if ((flags & kMet) && meet < 0) meet = depth;
    if (flags & kOverflow) { if (tid == 0) sh.overflow = 1; break; }
    if (meet >= 0 && depth >= meet + a.bfs_halo) break;
    if ((double)seen > a.bfs_stop_count) break;
  }
  if constexpr (!kCluster) {
    lx0 = __reduce_min_sync(0xffffffffu, lx0);
    lx1 = __reduce_max_sync(0xffffffffu, lx1);
    ly0 = __reduce_min_sync(0xffffffffu, ly0);
    ly1 = __reduce_max_sync(0xffffffffu, ly1);
    if (lane == 0 && lx1 >= 0) {
      atomicMin(&sh.bx0, X0 + lx0); atomicMax(&sh.bx1, X0 + lx1);
      atomicMin(&sh.by0, Y0 + ly0); atomicMax(&sh.by1, Y0 + ly1);
    }
  }
  __syncthreads();
  if (rank == 0) clk.mark(0);
  // Ordered compaction (ascending global id) of the words within `depth` cells
  // of the terminals' rectangle (beyond it nothing is marked): each CTA, in it
  // each warp, owns a contiguous run of them; count, scan the counts, then write.
  // Only positions below out_cap are stored; those of src and dst are recorded.
  const int cy0 = max(0, min(sy, dy) - Y0 - depth), cy1 = min(BH - 1, max(sy, dy) - Y0 + depth);
  const int cx0 = max(0, min(sx, dx) - X0 - depth) >> 4, cx1 = min(BW - 1, max(sx, dx) - X0 + depth) >> 4;
  const OgrDiv by_rw((unsigned)(cx1 - cx0 + 1)), by_bh((unsigned)(cy1 - cy0 + 1));
  const int words = (int)(by_rw.d * by_bh.d) * nz;
  // layer, row and column of the box of the i-th of these words
  auto place = [&](int i, int& z, int& y, int& c) {
    const unsigned row = by_rw((unsigned)i), zz = by_bh(row);
    z = (int)zz;
    y = cy0 + (int)(row - zz * by_bh.d);
    c = cx0 + (int)((unsigned)i - row * by_rw.d);
  };
  auto cells = [&](int i) -> unsigned {        // the low bit of each seen cell
    int z, y, c;
    place(i, z, y, c);
    const int at = (z * BH + y) * RW + c;
    unsigned w;
    if constexpr (kCluster) w = peer_ld(peer_addr(&marks[at], bfs_owner(at)));
    else w = marks[at];
    return (w | w >> 1) & 0x55555555u;
  };
  const int share = kCluster ? ((words + kBfsCtas - 1) / kBfsCtas + 31) & ~31 : words;
  const int c0 = kCluster ? min(words, rank * share) : 0, c1 = min(words, c0 + share);
  const int per = ((c1 - c0 + nw - 1) / nw + 31) & ~31;
  const int w0 = c0 + warp * per, w1 = min(c1, w0 + per);
  int cnt = 0;
#pragma unroll 4
  for (int i = w0 + lane; i < w1; i += 32) cnt += __popc(cells(i));
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) sh.s_cnt[warp] = cnt;
  __syncthreads();
  if (tid < 32) {
    const int c = tid < nw ? sh.s_cnt[tid] : 0;
    int x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    sh.s_off[tid] = x - c;
    x = __shfl_sync(0xffffffffu, x, 31);
    if (tid == 0) sh.R = x;
    if constexpr (kCluster)
      if (tid < kBfsCtas) peer_st(peer_addr(&mail.in[par ^ 1][rank], tid), make_int4(x, 0, 0, 0));
  }
  __syncthreads();
  int off = sh.s_off[warp];
  if constexpr (kCluster) {
    cluster_sync();
    int all = 0;
    for (int k = 0; k < kBfsCtas; ++k) {
      if (k == rank) off += all;
      all += mail.in[par ^ 1][k].x;
    }
    if (tid == 0) sh.R = all;
  }
  for (int i0 = w0; i0 < w1; i0 += 32) {
    const unsigned word = i0 + lane < w1 ? cells(i0 + lane) : 0u;
    unsigned some = __ballot_sync(0xffffffffu, word != 0u);
    some = (some | some >> 1) & 0x55555555u;   // two words, 32 cells, at a time
    while (some) {
      const int k = __ffs(some) - 1 + (lane >> 4);
      some &= some - 1;
      const bool in = __shfl_sync(0xffffffffu, word, k) >> (2 * (lane & 15)) & 1u;
      const unsigned b = __ballot_sync(0xffffffffu, in);
      if (in) {
        int z, y, c;
        place(i0 + k, z, y, c);
        const int pos = off + __popc(b & ((1u << lane) - 1u));
        const int32_t gid = z * plane + (Y0 + y) * nx + X0 + 16 * c + (lane & 15);
        if (pos < out_cap) out[pos] = gid;
        if constexpr (kCluster) {
          if (gid == src) peer_st(peer_addr(&sh.pos_src, 0), pos);
          if (gid == dst) peer_st(peer_addr(&sh.pos_dst, 0), pos);
        } else {
          if (gid == src) sh.pos_src = pos;
          if (gid == dst) sh.pos_dst = pos;
        }
      }
      off += __popc(b);
    }
  }
  if constexpr (kCluster) cluster_sync();
  __syncthreads();
  if (rank == 0) roi_finish(sh, a, out, out_cap);
  __syncthreads();
  if (rank == 0) clk.mark(1);
  return true;
}

// The same BFS for boxes that shared memory cannot hold, on seen[] (all zero on
// entry, restored to zero on exit) with queues of qcap entries; writes the ROI (ascending id,
// truncated with the must-keep swap) into out[0..out_cap) and its size into
// sh.R.  sh.status = OGR_ERR_CAPACITY when a queue overflowed.
//
// kCluster: by the kBfsCtas CTAs of a cluster, the counts and flags in the
// first one's sh (400x300x20, two ROIs of 200,000 nodes: 4.3 ms; by the
// first CTA alone 19.3; by one of 1,024 threads, before there was a box to try
// first, 9.5).
template <bool kCluster>
__device__ __noinline__ void roi_build_large(Shared& sh, const ogr_graph& g, const ogr_net_args& a, int32_t* seen, int32_t* const* q,
                          int64_t qcap, int32_t* out, int32_t out_cap, char* smem, StageClock& clk, int rank) {
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  const int ctas = kCluster ? kBfsCtas : 1;
  const int sl = tid & (kSub - 1), grp = (rank * nt + tid) / kSub, groups = ctas * nt / kSub;
  const int nx = g.nx, nz = g.nz;
  const int32_t plane = nx * g.ny;
  const int32_t src = a.src, dst = a.dst;
  const int32_t* __restrict__ indptr = g.indptr;
  const int32_t* __restrict__ indices = g.indices;
  auto sync_all = [&]() {
    if constexpr (kCluster) cluster_sync();
    else __syncthreads();
  };
  // a word of the first CTA's sh
  auto get = [&](int& x) -> int {
    if constexpr (kCluster) return (int)peer_ld(peer_addr(&x, 0));
    else return x;
  };
  auto add = [&](int& x, int v) -> int {
    if constexpr (kCluster) return peer_add(peer_addr(&x, 0), v);
    else return atomicAdd(&x, v);
  };
  auto lower = [&](int& x, int v) {
    if constexpr (kCluster) peer_min(peer_addr(&x, 0), v);
    else atomicMin(&x, v);
  };
  auto raise = [&](int& x, int v) {
    if constexpr (kCluster) peer_max(peer_addr(&x, 0), v);
    else atomicMax(&x, v);
  };
  if (tid == 0 && rank == 0) {
    seen[src] = 1;
    seen[dst] = 2;
    q[0][0] = src;
    q[2][0] = dst;
    sh.nq[0] = 1;
    sh.nq[2] = 1;
    sh.seen_count = (src != dst) ? 2 : 1;
    sh.overflow = 0;
    const int sy = (src % plane) / nx, sx = (src % plane) % nx;
    const int dy = (dst % plane) / nx, dx = (dst % plane) % nx;
    sh.bx0 = min(sx, dx); sh.bx1 = max(sx, dx);
    sh.by0 = min(sy, dy); sh.by1 = max(sy, dy);
    sh.met = 0;
    sh.pos_src = -1;
    sh.pos_dst = -1;
  }
  sync_all();
  int depth = 0, meet = -1;
  int cur_s = 0, cur_d = 2;
  while (depth < a.bfs_max_depth && (get(sh.nq[cur_s]) > 0 || get(sh.nq[cur_d]) > 0)) {
    for (int wave = 0; wave < 2; ++wave) {
      const int cur = wave == 0 ? cur_s : cur_d;
      const int nxt = cur ^ 1;
      const int32_t mark = wave == 0 ? 1 : 2;
      if (tid == 0 && rank == 0) sh.nq[nxt] = 0;
      sync_all();
      const int n = (int)min((int64_t)get(sh.nq[cur]), qcap);
      const int32_t* qc = q[cur];
      int32_t* qn = q[nxt];
      int local_met = 0, local_new = 0, local_ovf = 0;
      int lx0 = 1 << 30, lx1 = -1, ly0 = 1 << 30, ly1 = -1;
      for (int i = grp; i < n; i += groups) {
        const int32_t u = __ldcg(&qc[i]);
        const int32_t e1 = indptr[u + 1];
        for (int32_t e = indptr[u] + sl; e < e1; e += kSub) {
          if (g.blocked != nullptr && g.blocked[e]) continue;
          const int32_t v = indices[e];
          const int32_t old = atomicCAS(&seen[v], 0, mark);
          if (old == 0) {
            // (one count for the lanes that are here together)
            const unsigned here = __activemask();
            const int first = __ffs(here) - 1;
            int pos = 0;
            if (lane == first) pos = add(sh.nq[nxt], __popc(here));
            pos = __shfl_sync(here, pos, first) + __popc(here & ((1u << lane) - 1u));
            if (pos < qcap) qn[pos] = v; else local_ovf = 1;
            ++local_new;
            const int32_t r = v % plane;
            const int vy = r / nx, vx = r % nx;
            lx0 = min(lx0, vx); lx1 = max(lx1, vx);
            ly0 = min(ly0, vy); ly1 = max(ly1, vy);
          } else if (old != mark) {
            seen[v] = 3;
            local_met = 1;
          }
        }
      }
      __syncwarp();
      local_new = __reduce_add_sync(0xffffffffu, local_new);
      local_met = __reduce_or_sync(0xffffffffu, local_met);
      local_ovf = __reduce_or_sync(0xffffffffu, local_ovf);
      lx0 = __reduce_min_sync(0xffffffffu, lx0);
      lx1 = __reduce_max_sync(0xffffffffu, lx1);
      ly0 = __reduce_min_sync(0xffffffffu, ly0);
      ly1 = __reduce_max_sync(0xffffffffu, ly1);
      if (lane == 0) {
        if (local_met) raise(sh.met, 1);
        if (local_ovf) raise(sh.overflow, 1);
        if (local_new) {
          add(sh.seen_count, local_new);
          lower(sh.bx0, lx0); raise(sh.bx1, lx1);
          lower(sh.by0, ly0); raise(sh.by1, ly1);
        }
      }
      sync_all();
      if (wave == 0) cur_s = nxt; else cur_d = nxt;
    }
    ++depth;
    if (tid == 0 && rank == 0) atomicAdd(&g_stage[11], 2ull);
    if (get(sh.met) && meet < 0) meet = depth;
    if (meet >= 0 && depth >= meet + a.bfs_halo) break;
    if ((double)get(sh.seen_count) > a.bfs_stop_count) break;
    if (get(sh.overflow)) break;
  }
  sync_all();
  if (rank == 0) clk.mark(0);
  // Ordered compaction over the bounding box (ascending global id): each CTA,
  // in it each warp, owns a contiguous segment; count, scan the counts, then write.  Only
  // positions below out_cap are stored; those of src and dst are recorded.
  const int bx0 = get(sh.bx0), by0 = get(sh.by0);
  const int W = get(sh.bx1) - bx0 + 1, H = get(sh.by1) - by0 + 1;
  const int32_t area = W * H;
  const int32_t V = area * nz;
  const int32_t share = kCluster ? ((V + ctas - 1) / ctas + 31) & ~31 : V;
  const int32_t c0 = kCluster ? min((int64_t)V, (int64_t)rank * share) : 0, c1 = min((int64_t)V, (int64_t)c0 + share);
  const int32_t seg = (((c1 - c0 + nw - 1) / nw) + 31) & ~31;
  const int32_t w0 = c0 + min((int64_t)(c1 - c0), (int64_t)warp * seg), w1 = min((int64_t)c1, (int64_t)w0 + seg);
  auto gid_of = [&](int32_t i) -> int32_t {
    const int z = i / area;
    const int32_t rem = i - z * area;
    const int y = by0 + rem / W;
    const int x = bx0 + rem % W;
    return z * plane + y * nx + x;
  };
  int cnt = 0;
  for (int32_t b = w0; b < w1; b += 32) {
    const int32_t i = b + lane;
    const bool f = i < w1 && __ldcg(&seen[gid_of(i)]) != 0;
    cnt += __popc(__ballot_sync(0xffffffffu, f));
  }
  if (lane == 0) sh.s_cnt[warp] = cnt;
  __syncthreads();
  if (warp == 0) {
    const int c = lane < nw ? sh.s_cnt[lane] : 0;
    int x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < nw) sh.s_off[lane] = x - c;
    x = __shfl_sync(0xffffffffu, x, 31);
    if (lane == 31) sh.R = x;
    if constexpr (kCluster) {
      BfsMail& mail = *reinterpret_cast<BfsMail*>(smem);
      if (lane < kBfsCtas) peer_st(peer_addr(&mail.in[0][rank], lane), make_int4(x, 0, 0, 0));
    }
  }
  sync_all();
  int off = sh.s_off[warp];
  if constexpr (kCluster) {
    const BfsMail& mail = *reinterpret_cast<const BfsMail*>(smem);
    int all = 0;
    for (int k = 0; k < kBfsCtas; ++k) {
      if (k == rank) off += all;
      all += mail.in[0][k].x;
    }
    if (tid == 0) sh.R = all;
  }
  for (int32_t b = w0; b < w1; b += 32) {
    const int32_t i = b + lane;
    int32_t gid = 0;
    bool f = false;
    if (i < w1) {
      gid = gid_of(i);
      f = __ldcg(&seen[gid]) != 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, f);
    if (f) {
      const int pos = off + __popc(m & ((1u << lane) - 1));
      if (pos < out_cap) out[pos] = gid;
      if constexpr (kCluster) {
        if (gid == src) peer_st(peer_addr(&sh.pos_src, 0), pos);
        if (gid == dst) peer_st(peer_addr(&sh.pos_dst, 0), pos);
      } else {
        if (gid == src) sh.pos_src = pos;
        if (gid == dst) sh.pos_dst = pos;
      }
    }
    off += __popc(m);
  }
  sync_all();
  if (rank == 0) roi_finish(sh, a, out, out_cap);
  // restore seen[] to zero over the bounding box
  for (int32_t i = c0 + tid; i < c1; i += nt) seen[gid_of(i)] = 0;
  __syncthreads();
  if (rank == 0) clk.mark(1);
}

__device__ void roi_build(Shared& sh, const ogr_graph& g, const ogr_net_args& a, int32_t* seen, int32_t* const* q,
                          int64_t qcap, int32_t* out, int32_t out_cap, char* smem, StageClock& clk) {
  if (roi_build_box<false, 2, 6>(sh, g, a, q, qcap, out, out_cap, smem, clk, 0)) return;
  __syncthreads();
  roi_build_large<false>(sh, g, a, seen, q, qcap, out, out_cap, smem, clk, 0);
}

// The same by a cluster of kBfsCtas CTAs (rank: this one's); the result is in
// the first one's sh.
__device__ void roi_build_cluster(Shared& sh, const ogr_graph& g, const ogr_net_args& a, const Ws& w, int32_t* out,
                                  int32_t out_cap, char* smem, int rank) {
  StageClock clk;
  clk.start();
  if (threadIdx.x == 0) sh.status = OGR_OK;
  __syncthreads();
  if (roi_build_box<true, 4, 4>(sh, g, a, w.q, w.qcap, out, out_cap, smem, clk, rank)) return;
  __syncthreads();
  roi_build_large<true>(sh, g, a, w.seen, w.q, w.qcap, out, out_cap, smem, clk, rank);
}

// ---- the search on a given ROI ---------------------------------------------------
// What a team searches: roi[0..R) in ROI order (= tie order); with full the
// ROI is the whole lattice in id order.  The path (global ids, src first) goes
// to path_out.
//
// With ms the search is the reference's multi-source multi-sink form: every
// seed starts with label seed_cost + penalty and no parent (a first relaxation
// that later ones must beat in float32), targets are settled but never
// expanded, the search runs until nothing is left, and the result is the
// settled target with the least (label + target cost), first in pop order
// (label, ROI index) among equals.
struct RoiJob {
  const ogr_graph* g;
  const ogr_state* st;
  const ogr_net_args* a;
  const Ws* w;
  const int32_t* roi;
  int32_t R;
  const float* roi_pen;      // ROI-local penalty, or NULL: the state's
  const MultiSeeds* ms;
  int32_t* path_out;
  int32_t path_cap;
  unsigned long long* stats;
  int rank, nranks;
};

// One team's search.  Every CTA of the team calls it with the slot's team
// words zero; *status_out / *len_out are the result in the first thread of the
// team (elsewhere the status may lack what the backtrace finds, or a wait that
// another CTA gave up).
template <int L, int K, bool kMulti>
__device__ __noinline__ void roi_search(const RoiJob* jp, char* smem, int* status_out, int* len_out) {
  using namespace ogr_phase;
  const RoiJob job = *jp;
  const ogr_graph& g = *job.g;
  const ogr_state& st = *job.st;
  const ogr_net_args& a = *job.a;
  const Ws& w = *job.w;
  Head& sm = *reinterpret_cast<Head*>(smem);
  const int tid = threadIdx.x;
  const bool full = a.full_graph != 0, leader = job.rank == 0 && tid == 0;
  const int32_t R = job.R;
  const int step = job.nranks * kThreads, first = job.rank * kThreads + tid;
  long long t0 = clock64();
  auto mark = [&](int k) {
    if (leader) {
      const long long now = clock64();
      atomicAdd(&g_stage[k], (unsigned long long)(now - t0));
      t0 = now;
    }
  };
  int32_t* roi_w = w.roi;
  const int32_t* roi = full ? roi_w : job.roi;
  int32_t sid = __ldcg(&w.ctl->sid) + 1;
  const bool wrap = sid < 1 || sid == 0x7fffffff;
  if (wrap) {
    // the stamps begin again: of all nodes, not of this ROI's alone
    sid = 1;
    for (int r = first; r < w.nclaim; r += step) w.claim[r] = 0;
  }
  Problem pr{};
  pr.R = R;
  pr.indptr = g.indptr;
  pr.indices = g.indices;
  pr.rev = g.rev;
  pr.cost = st.total_cost;
  pr.rcost = st.rcost;
  pr.roi = roi;
  pr.g2r = w.g2r;
  pr.rec = w.rec;
  pr.par = w.par;
  pr.claim = w.claim;
  pr.ov[0] = w.ov[0];
  pr.ov[1] = w.ov[1];
  pr.mseed = kMulti ? job.ms->init : nullptr;
  pr.ctl = &w.ctl->team;
  pr.rank = job.rank;
  pr.nranks = job.nranks;
  if (tid == 0) {
    sm.spin = w.spin;
    sm.max_phase = w.max_phases > 0 ? min(w.max_phases, 2 * R + 4) : 2 * R + 4;
    sm.first = 0;
  }
  // With statistics requested the search goes on after dst is settled until
  // every node with a label <= L(dst) is settled (T > L(dst)): the IN bound
  // can settle dst before cheaper nodes, which the heap pops earlier.
  pr.want_stats = job.stats != nullptr;
  Outcome o{};
  bool fix = true;
  pr.sid = sid;
  int md = 0;
  for (int r = first; r < R; r += step) {
    const int32_t gid = full ? r : roi[r];
    if (full) roi_w[r] = r;
    w.g2r[gid] = r;
    const int32_t f0 = g.indptr[gid], f1 = g.indptr[gid + 1];
    md = max(md, f1 - f0);
    const float pen = job.roi_pen ? job.roi_pen[r] : ogr_node_penalty(st, a, gid);
    __stcg(reinterpret_cast<int4*>(&w.rec[r]), make_int4(f0, f1 - f0, 0, __float_as_int(pen)));
    if (kMulti) {
      job.ms->init[r] = __longlong_as_double((long long)kNoTerm);
      job.ms->tcost[r] = __longlong_as_double((long long)kNoTerm);
    }
  }
  md = __reduce_max_sync(0xffffffffu, md);
  if ((tid & 31) == 0) sm.wmin[tid >> 5] = (unsigned long long)md;
  __syncthreads();
  if (tid == 0) {
    sm.ok = 1;
    for (int i = 1; i < kWarps; ++i) md = max(md, (int)sm.wmin[i]);
    arrive(pr, sm, 0, kArrive, ~(unsigned long long)md);
    await(pr, sm, 0);
    sm.res[2] = (int)sm.t;
    sm.res[0] = 0;               // first entries
    sm.res[1] = 0;               // bad seeds or targets
    sm.wmin[0] = kNone;          // their least label
  }
  __syncthreads();
  const int max_deg = sm.res[2];
  const int ready = sm.ok;
  if (max_deg > kMaxRow) fix = false;
  if (leader && max_deg > L * K) atomicAdd(&g_stage[15], 1ull);
  int32_t rs = -1, rd = -1;
  if (!kMulti && ready) {
    rs = __ldcg(&w.g2r[a.src]);
    rd = __ldcg(&w.g2r[a.dst]);
  }
  const bool none = !kMulti && (rs < 0 || rd < 0 || rs == rd);
  pr.src = rs;
  pr.dst = rd;
  auto enter = [&](int32_t r, int at, int32_t flags) {
    const int32_t gid = roi[r], f0 = g.indptr[gid];
    w.claim[r] = pr.sid;
    w.ov[0][at] = make_int4(r, f0, (g.indptr[gid + 1] - f0) | flags, __float_as_int(__ldcg(&w.rec[r].pen)));
  };
  if (ready && job.rank == 0) {
    if constexpr (kMulti) {
      // Seeds and targets outside the ROI are dropped (as the reference
      // does); a repeated seed or target id is an argument error.
      const MultiSeeds& ms = *job.ms;
      for (int i = tid; i < ms.ntargets; i += kThreads) {
        const int32_t gid = ms.targets[i];
        const int32_t r = gid < 0 || gid >= g.num_nodes ? -2 : w.g2r[gid];
        if (r < 0) {
          if (r == -2) sm.res[1] = 1;
          continue;
        }
        const double c = ms.target_cost[i];
        const unsigned long long was = atomicExch(reinterpret_cast<unsigned long long*>(&ms.tcost[r]),
                                                  (unsigned long long)__double_as_longlong(c));
        if (was != kNoTerm) sm.res[1] = 1;
        // (a target cost that is not a number marks no target)
        if (c == c) w.rec[r].sp = kTgt;
      }
      __syncthreads();
      for (int i = tid; i < ms.nseeds; i += kThreads) {
        const int32_t gid = ms.seeds[i];
        const int32_t r = gid < 0 || gid >= g.num_nodes ? -2 : w.g2r[gid];
        if (r < 0) {
          if (r == -2) sm.res[1] = 1;
          continue;
        }
        const double c = ms.seed_cost[i];
        const unsigned long long was = atomicExch(reinterpret_cast<unsigned long long*>(&ms.init[r]),
                                                  (unsigned long long)__double_as_longlong(c));
        if (was != kNoTerm) {
          sm.res[1] = 1;
          continue;
        }
        if (!(c < __longlong_as_double(0x7ff0000000000000ll))) continue;      // not a start
        const float pen = __ldcg(&w.rec[r].pen);
        unsigned long long lb = ogr_dbits(c + (double)pen);
        if (fix) {
          lb = 0ull;
          if (seed_ticks(c, &lb) && tick_finite(pen)) lb += ticks(pen);
        }
        const int32_t flags = kSeed | (__ldcg(&w.rec[r].sp) & kTgt);
        enter(r, atomicAdd(&sm.res[0], 1), flags);
        w.rec[r].sp = 1 | flags;
        atomicMin(&sm.wmin[0], lb);
      }
    } else if (tid == 0 && !none) {
      enter(rs, 0, 0);
      w.ov[0][0].w = 0;          // src's penalty does not count
      sm.res[0] = 1;
      sm.wmin[0] = 0ull;
    }
  }
  __syncthreads();
  if (tid == 0 && ready) {
    unsigned long long nf0 = 0, tl = kNone;
    if (job.rank == 0) {
      nf0 = sm.res[1] ? 0 : (unsigned)sm.res[0];
      tl = sm.wmin[0];
      w.ctl->merr = sm.res[1];
      w.ctl->team.nov[0] = (int)nf0;
      w.ctl->team.nov[1] = 0;
      w.ctl->team.nov[2] = 0;
    }
    arrive(pr, sm, 1, kArrive + kOut * (nf0 < kMostOut ? nf0 : kMostOut) + kCount * nf0, tl);
    await(pr, sm, 1);
    if (kMulti && sm.ok && __ldcg(&w.ctl->merr)) sm.ok = 2;
  }
  __syncthreads();
  const int ok = sm.ok;
  __syncthreads();
  mark(2);
  int k0 = 2;                  // barriers used so far
  if (ok != 1 || none) {
    o.status = ok == 0 ? OGR_ERR_TIMEOUT : ok == 2 ? OGR_ERR_ARG : OGR_NO_PATH;
  } else {
    o = run_search<L, K, kMulti, true>(pr, smem, 1, max_deg, fix);
    k0 = 1 + o.phases;
    if (o.status == kStInexact) {
      if (leader && max_deg <= L * K) atomicAdd(&g_stage[15], 1ull);
      const Problem p = pr;
      Outcome io = o;
      int k = k0;
      go_over<kMulti, true>(&p, smem, &k, first, step, &io);
      o = io;
      k0 = k;
      fix = false;
    }
  }
  mark(3);
  if (leader) {
    atomicAdd(&g_stage[4], (unsigned long long)o.wait);
    atomicAdd(&g_stage[9], 1ull);
    atomicAdd(&g_stage[10], (unsigned long long)o.phases);
  }
  if (tid == 0) atomicAdd(&g_stage[13], o.examined);
  int status = o.status;
  int32_t tgt = pr.dst;
  if (kMulti && status == OGR_OK) {
    // The reference keeps the first popped target whose label + target cost is
    // strictly below the best so far: the least (total, label, ROI index).
    // Every CTA of the team makes the choice (the statistics depend on it).
    const MultiSeeds& ms = *job.ms;
    const double dinf = __longlong_as_double(0x7ff0000000000000ll);
    unsigned long long best[3] = {kNone, kNone, kNone};
    for (int pass = 0; pass < 3; ++pass) {
      unsigned long long k = kNone;
      for (int i = tid & 31; i < ms.ntargets; i += 32) {
        const int32_t r = w.g2r[ms.targets[i]];
        if (r < 0) continue;
        const Rec x = ld_rec(&w.rec[r]);
        if ((x.sp & kSpMask) < 2) continue;
        const double lr = fix ? label_value<true>(x.lab) : label_value<false>(x.lab);
        const double tot = lr + ms.target_cost[i];
        if (!(tot < dinf)) continue;
        const unsigned long long kt = ogr_order_bits(tot), kl = ogr_order_bits(lr);
        const unsigned long long y = pass == 0   ? kt
                                     : pass == 1 ? (kt == best[0] ? kl : kNone)
                                                 : (kt == best[0] && kl == best[1] ? (unsigned long long)r : kNone);
        k = y < k ? y : k;
      }
      best[pass] = warp_min_u64(k);
    }
    tgt = best[0] == kNone ? -1 : (int32_t)best[2];
    if (tgt < 0) status = OGR_NO_PATH;
  }
  // Statistics of the sequential heap search: the rows of the nodes popped
  // before dst; of a search that cannot reach dst, every node it reaches; of a
  // multi-source search, every settled node, the expanded ones' rows.
  const bool found = status == OGR_OK;
  if (job.stats != nullptr && (found || (!kMulti && o.exhausted))) {
    count_work<kMulti, true>(pr, o, first, step, job.stats);
    if (leader) {
      if (found && !kMulti) atomicAdd(&job.stats[1], 1ull);   // dst's own pop
      atomicAdd(&job.stats[2], (unsigned long long)R);
      atomicAdd(&job.stats[3], (unsigned long long)o.phases);
    }
  }
  // Backtrace dst -> src (reversed into path_out), by the first CTA.
  int len = 0;
  if (job.rank == 0 && found) {
    if (tid < 32) {
      const int limit = min(job.path_cap, R);
      int32_t c = -1;
      len = walk_parents(w.par, tgt, R, limit, job.path_out, &c);
      // (a parent chain longer than the ROI is a cycle)
      if (c != -1) status = len >= R ? OGR_ERR_ITER_CAP : OGR_ERR_CAPACITY;
      else if (len < 2) status = OGR_NO_PATH;
      if (tid == 0) {
        sm.res[0] = status;
        sm.res[1] = len;
      }
    }
    __syncthreads();
    status = sm.res[0];
    len = status == OGR_OK ? sm.res[1] : 0;
    for (int i = tid; i < len / 2; i += kThreads) {
      const int32_t x = job.path_out[i], y = job.path_out[len - 1 - i];
      job.path_out[i] = roi[y];
      job.path_out[len - 1 - i] = roi[x];
    }
    if ((len & 1) && tid == 0) job.path_out[len / 2] = roi[job.path_out[len / 2]];
  }
  mark(7);
  if (kMulti && job.nranks > 1) {
    // the choice of the target reads the map in every CTA
    if (tid == 0) {
      arrive(pr, sm, k0, kArrive, kNone);
      await(pr, sm, k0);
    }
    __syncthreads();
  }
  for (int r = first; r < R; r += step) w.g2r[roi[r]] = -1;
  if (leader) {
    w.ctl->sid = fix || max_deg > kMaxRow ? sid : sid + 1;      // (one that went over to doubles took two)
    // (a CTA that gave up on the last wait left its part of the statistics out)
    if (*(const volatile int32_t*)&w.ctl->team.err) status = OGR_ERR_TIMEOUT;
  }
  __syncthreads();
  mark(8);
  *status_out = status;
  *len_out = len;
}

// The search in the form for rows of ROW arcs.
template <int ROW, bool kMulti>
__device__ __forceinline__ void roi_search_row(const RoiJob& job, char* smem, int* status, int* len) {
  if constexpr (ROW == 4) roi_search<2, 2, kMulti>(&job, smem, status, len);
  else if constexpr (ROW == 8) roi_search<8, 1, kMulti>(&job, smem, status, len);
  else if constexpr (ROW == 16) roi_search<8, 2, kMulti>(&job, smem, status, len);
  else roi_search<16, 2, kMulti>(&job, smem, status, len);
}

// The ROI of one net into w.roi (nothing for a full-graph net), by one CTA:
// sh.status and sh.R tell.
__device__ void build_roi(Shared& sh, const ogr_graph& g, const ogr_net_args& a, const Ws& w, char* smem) {
  StageClock clk;
  clk.start();
  if (threadIdx.x == 0) sh.status = OGR_OK;
  __syncthreads();
  if (a.full_graph) {
    if (threadIdx.x == 0) sh.R = g.num_nodes;
    __syncthreads();
    return;
  }
  roi_build(sh, g, a, w.seen, w.q, w.qcap, w.roi, a.max_roi_nodes, smem, clk);
}

// ---- commit / rip-up ---------------------------------------------------------
constexpr int kViaHops = kMaxViaNodes / 3;     // via hops listed in s_via[kMaxViaNodes]

// Calls f(node) once for every node that the via hops of a path span, from any
// thread of the block; true if there are more than kMaxViaNodes of them.
// s_via: kMaxViaNodes words, s_cnt: two words.
//
// The hops are sorted out by all threads, and a node that several hops span
// belongs to the one listed first.  (One thread walking the path with four
// divisions per hop took 150 us for 450 hops, most of a commit.)
template <typename F>
__device__ bool each_via_node(const int32_t* path, int hops, int32_t plane, int32_t* s_via, int* s_cnt, F&& f) {
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) { s_cnt[0] = 0; s_cnt[1] = 0; }
  __syncthreads();
  for (int i = tid; i < hops; i += nt) {
    const int32_t u = path[i], v = path[i + 1];
    const int zu = u / plane, zv = v / plane;
    if (u - zu * plane != v - zv * plane || zu == zv) continue;
    const int k = atomicAdd(&s_cnt[0], 1);
    if (k < kViaHops) {
      s_via[k] = u - zu * plane;
      s_via[kViaHops + k] = min(zu, zv);
      s_via[2 * kViaHops + k] = max(zu, zv);
    }
  }
  __syncthreads();
  const int n = s_cnt[0];
  if (n <= kViaHops) {
    for (int k = tid; k < n; k += nt) {
      const int32_t r = s_via[k];
      const int lo = s_via[kViaHops + k], hi = s_via[2 * kViaHops + k];
      for (int z = lo; z <= hi; ++z) {
        bool dup = false;
        for (int j = 0; j < k && !dup; ++j)
          dup = s_via[j] == r && z >= s_via[kViaHops + j] && z <= s_via[2 * kViaHops + j];
        if (!dup && atomicAdd(&s_cnt[1], 1) < kMaxViaNodes) f(z * plane + r);
      }
    }
    __syncthreads();
    return s_cnt[1] > kMaxViaNodes;
  }
  // more hops than the list holds: one thread collects the nodes
  __syncthreads();
  if (tid == 0) {
    int nv = 0;
    bool full = false;
    for (int i = 0; i < hops && !full; ++i) {
      const int32_t u = path[i], v = path[i + 1];
      const int zu = u / plane, zv = v / plane;
      const int32_t r = u - zu * plane;
      if (r != v - zv * plane || zu == zv) continue;
      for (int z = min(zu, zv); z <= max(zu, zv); ++z) {
        const int32_t nd = z * plane + r;
        bool dup = false;
        for (int k = 0; k < nv && !dup; ++k) dup = s_via[k] == nd;
        if (dup) continue;
        if (nv >= kMaxViaNodes) { full = true; break; }
        s_via[nv++] = nd;
      }
    }
    s_cnt[0] = nv;
    s_cnt[1] = full ? 1 : 0;
  }
  __syncthreads();
  const int nv = s_cnt[0];
  for (int k = tid; k < nv; k += nt) f(s_via[k]);
  const bool full = s_cnt[1] != 0;
  __syncthreads();
  return full;
}

// The arc u -> v (-1: none).  A row's arcs come four at a time, so a hop waits
// once or twice for its row, not once per arc.
__device__ __forceinline__ int32_t arc_to(const ogr_graph& g, int32_t u, int32_t v) {
  const int32_t e1 = g.indptr[u + 1];
  for (int32_t e = g.indptr[u]; e < e1; e += 4) {
    int32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = e + j < e1 ? g.indices[e + j] : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (w[j] == v) return e + j;
  }
  return -1;
}

// commit_path / clear_path (:1096-1135) + refresh_live_present_costs (:1403),
// _mark/_clear_path_node_use (:4635-4659), barrel ownership of every node a
// via hop spans (:4934-5034), arcs in _path_to_edges order (:9981-10046).
// Returns OGR_OK, OGR_ERR_ARG (a hop is not an arc) or OGR_ERR_CAPACITY.
// s_flags: three words.
__device__ int apply_path_dev(const ogr_graph& g, const ogr_state& st, const int32_t* path, int32_t len,
                              int32_t net_id, int32_t sign, float pres_fac, int32_t live, int32_t* arcs_out,
                              int32_t* s_via, int* s_flags) {
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid == 0) s_flags[2] = 0;
  __syncthreads();
  const int hops = len - 1;
  const int32_t plane = g.nx * g.ny;
  for (int i = tid; i < hops; i += nt) {
    const int32_t f = arc_to(g, path[i], path[i + 1]);
    if (f < 0) { s_flags[2] = 1; continue; }
    const int32_t r = g.rev[f];
    const int j = hops - 1 - i;
    if (arcs_out) { arcs_out[i] = f; arcs_out[hops + j] = r; }
    for (int k = 0; k < 2; ++k) {
      const int32_t e = k == 0 ? f : r;
      float p = st.present[e];
      p = sign > 0 ? __fadd_rn(p, 1.0f) : fmaxf(__fsub_rn(p, 1.0f), 0.0f);
      st.present[e] = p;
      if (live) {
        const float bias = (st.layer_bias != nullptr && st.edge_kind[e] == 0) ? st.layer_bias[st.edge_layer[e]] : 1.0f;
        const float scale = st.layer_bias != nullptr ? __fmul_rn(pres_fac, bias) : pres_fac;
        const float prosp = fmaxf(0.0f, __fsub_rn(__fadd_rn(p, 1.0f), st.capacity[e]));
        const float tc = __fadd_rn(st.live_static[e], __fmul_rn(scale, prosp));
        st.total_cost[e] = tc;
        if (st.rcost) st.rcost[k == 0 ? r : f] = tc;   // the opposite arc's row entry
      }
    }
  }
  for (int i = tid; i < len; i += nt) {
    const int32_t n = path[i];
    const int32_t u = st.path_node_use[n];
    st.path_node_use[n] = sign > 0 ? u + 1 : max(u - 1, 0);
  }
  __syncthreads();
  if (s_flags[2]) {
    __syncthreads();
    return OGR_ERR_ARG;
  }
  const bool full = each_via_node(path, hops, plane, s_via, s_flags, [&](int32_t nd) {
    st.owner_count[nd] += sign > 0 ? 1 : -1;
    st.owner_xor[nd] ^= net_id;
  });
  __syncthreads();
  return full ? OGR_ERR_CAPACITY : OGR_OK;
}

// ---- kernels -------------------------------------------------------------------
// The ROI of a net (not a full-graph one) into w.roi, by one cluster:
// result[0] = status, result[3] = its size.
__global__ void __cluster_dims__(kBfsCtas) __launch_bounds__(kClusterThreads, 1)
build_roi_kernel(ogr_graph g, ogr_net_args a, Ws w) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Shared sh;
  roi_build_cluster(sh, g, a, w, w.roi, a.max_roi_nodes, smem, blockIdx.x);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.result[0] = sh.status;
    w.result[1] = 0;
    w.result[3] = sh.R;
  }
}

// One team's search of a net (or, kMulti, of seeds and targets): a caller's
// ROI, or (roi NULL) the one build_roi_kernel left, or the whole lattice.
template <int ROW, bool kMulti>
__global__ void __launch_bounds__(kThreads, 1)
find_team_kernel(ogr_graph g, ogr_state st, ogr_net_args a, Ws w, const int32_t* roi, int32_t R, const float* roi_pen,
                 MultiSeeds ms, int32_t* path_out, int32_t path_cap, int64_t* stats) {
  extern __shared__ __align__(16) char smem[];
  if (roi == nullptr && !a.full_graph) {
    if (w.result[0] != OGR_OK) return;             // uniform: written by an earlier launch
    roi = w.roi;
    R = (int32_t)w.result[3];
  }
  // A ROI of a few hundred nodes is searched by the first CTA alone, which has
  // no barrier to wait at: given ROIs of 98, 210 and 362 nodes of 100x100x6 take
  // 46, 58 and 63 us instead of 52, 60 and 72; of 567 and 1,071 a team takes 77
  // and 96, one CTA 83 and 109.
  const int team = R < kLoneNodes ? 1 : (int)gridDim.x;
  if ((int)blockIdx.x >= team) return;
  const RoiJob job{&g,       &st,      &a,    &w, roi, R, roi_pen, &ms, path_out, path_cap,
                   reinterpret_cast<unsigned long long*>(stats), (int)blockIdx.x, team};
  int status, len;
  roi_search_row<ROW, kMulti>(job, smem, &status, &len);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.result[0] = status;
    w.result[1] = len;
  }
}

__global__ void __cluster_dims__(kBfsCtas) __launch_bounds__(kClusterThreads, 1)
roi_kernel(ogr_graph g, ogr_net_args a, Ws w, int32_t* roi_out, int32_t roi_cap) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Shared sh;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  if (a.full_graph) {
    const int32_t R = g.num_nodes;
    if (R <= roi_cap)
      for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) roi_out[r] = r;
    if (leader) {
      w.result[0] = R > roi_cap ? OGR_ERR_CAPACITY : OGR_OK;
      w.result[1] = R;
    }
    return;
  }
  roi_build_cluster(sh, g, a, w, roi_out, roi_cap, smem, blockIdx.x);
  if (leader) {
    w.result[0] = sh.status;
    w.result[1] = sh.R;
  }
}

__global__ void ws_init_kernel(Ws w, int64_t N) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    w.seen[i] = 0;
    w.g2r[i] = -1;
    w.claim[i] = 0;
  }
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < (int)(sizeof(SlotCtl) / 4); i += blockDim.x) reinterpret_cast<int32_t*>(w.ctl)[i] = 0;
}

__global__ void bfs_init_kernel(char* base, int32_t slots, size_t slot_bytes, int32_t N, int64_t qcap) {
  for (int s = 0; s < slots; ++s) {
    BfsSlot b = bfs_slot_at(base + (size_t)s * slot_bytes, N, qcap);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
      b.seen[i] = 0;
  }
}

constexpr int kApplyThreads = 256;

__global__ void __launch_bounds__(kApplyThreads)
path_apply_kernel(ogr_graph g, ogr_state st, const int32_t* path, int32_t len, int32_t net_id, int32_t sign,
                  float pres_fac, int32_t live, int32_t* arcs_out, int32_t* status) {
  __shared__ int32_t s_via[kMaxViaNodes];
  __shared__ int s_flags[3];
  const int rc = apply_path_dev(g, st, path, len, net_id, sign, pres_fac, live, arcs_out, s_via, s_flags);
  if (threadIdx.x == 0) *status = rc;
}

// Commit many paths at once (a best-state restore, _restore_routing_state
// :7806-7838): present +1 on both arcs of every hop, path-node use +1, barrel
// ownership of every via-spanned node; no live refresh.  Commits only add
// exact small integers (and XOR ids), so paths may be applied by different
// CTAs in any order and the state equals the sequential one.  Path k is
// nodes[off[k] .. off[k+1]); its arcs go to arcs[2 * (off[k] - k) ..]; with a
// store given, the path, its length and its arcs are also written to slot
// store_slot[k] (the per-net overuse sums read the slot's arcs).
__global__ void __launch_bounds__(kApplyThreads)
paths_commit_kernel(ogr_graph g, ogr_state st, const int32_t* nodes, const int32_t* off, const int32_t* net_ids,
                    int32_t n_paths, int32_t* arcs, int32_t* store_path, int32_t* store_len,
                    int32_t* store_arcs, const int32_t* store_slot, int32_t slot_cap, int32_t* status) {
  __shared__ int32_t s_via[kMaxViaNodes];
  __shared__ int s_cnt[2], s_bad;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int32_t plane = g.nx * g.ny;
  for (int32_t k = blockIdx.x; k < n_paths; k += gridDim.x) {
    const int32_t o = off[k], len = off[k + 1] - off[k];
    const int32_t* path = nodes + o;
    const int hops = len - 1;
    int32_t* a_out = arcs + 2 * (int64_t)(o - k);
    int32_t* a_store = (store_arcs != nullptr && len <= slot_cap)
                           ? store_arcs + (int64_t)store_slot[k] * 2 * slot_cap : nullptr;
    if (tid == 0) s_bad = 0;
    __syncthreads();
    for (int i = tid; i < hops; i += nt) {
      const int32_t f = arc_to(g, path[i], path[i + 1]);
      if (f < 0) { s_bad = 1; continue; }
      const int32_t r = g.rev[f];
      a_out[i] = f;
      a_out[hops + (hops - 1 - i)] = r;
      if (a_store) {
        a_store[i] = f;
        a_store[hops + (hops - 1 - i)] = r;
      }
      atomicAdd(&st.present[f], 1.0f);
      atomicAdd(&st.present[r], 1.0f);
    }
    for (int i = tid; i < len; i += nt) atomicAdd(&st.path_node_use[path[i]], 1);
    if (store_path != nullptr && len <= slot_cap)
      for (int i = tid; i < len; i += nt) store_path[(int64_t)store_slot[k] * slot_cap + i] = path[i];
    __syncthreads();
    if (tid == 0 && store_len != nullptr) store_len[store_slot[k]] = len <= slot_cap ? len : 0;
    const int32_t id = net_ids[k];
    const bool full = !s_bad && each_via_node(path, hops, plane, s_via, s_cnt, [&](int32_t nd) {
      atomicAdd(&st.owner_count[nd], 1);
      atomicXor(&st.owner_xor[nd], id);
    });
    if (tid == 0 && (full || (len > slot_cap && store_path != nullptr))) s_bad = 2;
    if (tid == 0 && s_bad) atomicMax(status, s_bad);
    __syncthreads();
  }
}

// Extract the (cost-independent) ROIs of every ROI net of the pass, one net
// per CTA at a time, each CTA with its own BFS slot.  roi_len[n] = -1 when a
// queue overflowed (the pass then extracts that ROI inline).
__global__ void __launch_bounds__(kBfsThreads, 1)
roi_batch_kernel(ogr_graph g, ogr_net_table t, ogr_pass_args pa, ogr_roi_batch rb) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Shared sh;
  __shared__ int s_k;
  BfsSlot slot = bfs_slot_at((char*)rb.bfs_ws + (size_t)blockIdx.x * rb.slot_bytes, g.num_nodes, rb.qcap);
  while (true) {
    if (threadIdx.x == 0) s_k = atomicAdd(rb.next, 1);
    __syncthreads();
    const int k = s_k;
    __syncthreads();
    if (k >= pa.count) break;
    const int32_t n = pa.order[k];
    if (t.net_full[n]) {
      if (threadIdx.x == 0) rb.roi_len[n] = 0;
      continue;
    }
    ogr_net_args a = ogr_pass_net_args(t, pa, n, 0);
    StageClock clk;
    clk.start();
    if (threadIdx.x == 0) sh.status = OGR_OK;
    __syncthreads();
    roi_build(sh, g, a, slot.seen, slot.q, slot.qcap, rb.roi_pool + (int64_t)n * rb.roi_cap, rb.roi_cap, smem, clk);
    if (threadIdx.x == 0) {
      rb.roi_len[n] = (sh.status == OGR_OK) ? sh.R : -1;
      if (rb.roi_box) {
        rb.roi_box[4 * n + 0] = sh.bx0;
        rb.roi_box[4 * n + 1] = sh.bx1;
        rb.roi_box[4 * n + 2] = sh.by0;
        rb.roi_box[4 * n + 3] = sh.by1;
      }
    }
    __syncthreads();
  }
}

// ---- batched disjoint-ROI windows ---------------------------------------------
// Control block of the window pass (device scratch, cleared per launch).
struct WinCtl {
  unsigned long long bar_count;
  int32_t bar_err;
  int32_t cursor;
  int32_t wsize;
  int32_t error;
  int32_t solo_R;            // size of the ROI built inline (solo member or fallback)
  int32_t fb;                // 1 + position of the net whose fallback is to be searched
  int32_t fb_st, fb_len;
};

struct WinSlots {
  int32_t* k;                      // position in the order of the window's b-th net
  int32_t* solo;                   // 1: ROI extracted inline (the batched one overflowed)
  int32_t* st;                     // status of the b-th search
  int32_t* len;                    // path length of the b-th search
  unsigned long long* stats;       // [4] the b-th search's statistics, added on acceptance
  int32_t* inorder;                // 1: no pending net precedes the b-th net
};

__host__ __device__ inline size_t win_ctl_layout(int32_t slots, char* base, WinCtl** c, WinSlots* s) {
  size_t off = round256(sizeof(WinCtl));
  const size_t k = (size_t)slots;
  char* p[6];
  const size_t sz[6] = {4 * k, 4 * k, 4 * k, 4 * k, 32 * k, 4 * k};
  for (int i = 0; i < 6; ++i) {
    p[i] = base ? base + off : nullptr;
    off += round256(sz[i]);
  }
  if (c) *c = (WinCtl*)base;
  if (s) {
    s->k = (int32_t*)p[0];
    s->solo = (int32_t*)p[1];
    s->st = (int32_t*)p[2];
    s->len = (int32_t*)p[3];
    s->stats = (unsigned long long*)p[4];
    s->inorder = (int32_t*)p[5];
  }
  return off;
}

constexpr unsigned kWinBarSpin = 1u << 24;

// Bounded grid barrier (monotone arrival counter); false once any CTA gave up.
__device__ bool win_barrier(WinCtl* c, unsigned long long& target, int* s_flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    int ok = 1;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&c->bar_count) : "memory");
    unsigned it = 0;
    while (true) {
      unsigned long long v;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&c->bar_count) : "memory");
      if (v >= target) break;
      if (++it > kWinBarSpin || *(volatile int32_t*)&c->bar_err) {
        atomicExch(&c->bar_err, 1);
        ok = 0;
        break;
      }
      if (it > 64) __nanosleep(64);
    }
    *s_flag = ok;
  }
  __syncthreads();
  return *s_flag != 0;
}

// Of boxes {x0, x1, y0, y1}.
__device__ __forceinline__ bool boxes_meet(int4 a, int4 b) {
  return !(a.y < b.x || b.y < a.x || a.w < b.z || b.w < a.z);
}

// Copies a path found into scratch to the net's store slot and commits it.
__device__ int commit_from(const ogr_graph& g, const ogr_state& st, const ogr_net_table& t, const ogr_pass_args& pa,
                           int32_t n, const int32_t* path, int32_t len, int32_t* s_via, int* s_flags) {
  int32_t* slot = t.store_path + (int64_t)n * t.slot_cap;
  for (int i = threadIdx.x; i < len; i += blockDim.x) slot[i] = path[i];
  __syncthreads();
  const int rc = apply_path_dev(g, st, slot, len, t.net_id[n], +1, pa.pres_fac, pa.live,
                                t.store_arcs + (int64_t)n * 2 * t.slot_cap, s_via, s_flags);
  if (threadIdx.x == 0 && rc == OGR_OK) t.store_len[n] = len;
  return rc;
}

// Clears a search slot's team words (between searches).
__device__ __forceinline__ void clear_team(SlotCtl* c) {
  for (int i = threadIdx.x; i < (int)(sizeof(ogr_phase::Ctl) / 4); i += blockDim.x)
    reinterpret_cast<int32_t*>(&c->team)[i] = 0;
}

// The ROI nets of a pass (pa.order[0..count)) in windows of mutually disjoint
// footprints.  CTA 0 forms each window; the CTAs split into one team per
// member, which rips up and searches its net into scratch; then either every
// net commits (no failure) or CTA 0 commits in order up to the first failed
// net and undoes the later nets' rip-ups, and a team runs the failed net's
// fallback.  Without windows (nslots = 0) every window is one net, searched in
// the route workspace w.
template <int ROW>
__global__ void __launch_bounds__(kThreads, 1)
window_pass_kernel(ogr_graph g, ogr_state st, ogr_net_table t, ogr_pass_args pa, ogr_roi_batch rb, int use_batch,
                   char* slot_base, size_t slot_bytes, int32_t rmax, int32_t nslots, int32_t* scratch,
                   char* ctl_base, Ws w, int32_t look, unsigned long long* discarded) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Shared sh;
  __shared__ int s_flags[3];
  __shared__ int s_bar;
  __shared__ int4 s_box[kWarps], s_grown[kWarps], s_skip[kMaxSkip];
  __shared__ int2 s_cand[kWarps];
  __shared__ int s_win[4];
  int32_t* s_via = reinterpret_cast<int32_t*>(smem);     // (no search is on while paths are applied)
  const int b = blockIdx.x, tid = threadIdx.x, G = gridDim.x;
  if (w.result[0] < 0) return;  // uniform: an earlier step of this pass failed
  const int wmax = nslots > 0 ? nslots : 1;
  WinCtl* c;
  WinSlots ws;
  win_ctl_layout(wmax, ctl_base, &c, &ws);
  unsigned long long* stats = reinterpret_cast<unsigned long long*>(pa.stats);
  const int32_t plane = g.nx * g.ny;
  unsigned long long target = 0;
  // member m's search slot and path buffer
  auto slot_of = [&](int m, bool solo) {
    Ws x = w;
    if (nslots > 0 && !solo) ws_slot_layout(g.num_nodes, rmax, slot_base + (size_t)m * slot_bytes, &x);
    x.spin = w.spin;
    x.max_phases = w.max_phases;
    return x;
  };
  auto path_of = [&](int m, int32_t n) {
    return nslots > 0 ? scratch + (int64_t)m * t.slot_cap : t.store_path + (int64_t)n * t.slot_cap;
  };
  // On an error before the commits every member of the window is without its
  // old path: so says the store.
  auto ripped_up = [&](int members) {
    if (b < members && tid == 0) t.store_len[pa.order[ws.k[b]]] = 0;
  };
  if (b < wmax) clear_team(slot_of(b, false).ctl);
  if (b == 0) clear_team(w.ctl);
  while (true) {
    // 1. window formation (CTA 0).  Nets are taken in order from the first
    // pending one while their footprints (ROI box and old-path box) are
    // pairwise disjoint.  With look > 0 a clashing net is skipped (it stays
    // pending) and the scan goes on: a later net joins only if it is also
    // disjoint from every skipped net's footprint grown to the bound of its
    // fallback ROI (terminals +- fallback BFS depth + halo), so it commutes
    // with the skipped nets whatever they do when their turn comes.
    // Pending = net_status still -1 (set before the launch).
    StageClock clk;
    clk.start();
    if (b == 0) {
      // A warp looks up each candidate's footprint, kWarps candidates at a
      // time, and the first warp decides on them in order.  (One candidate
      // after the other, by all threads, took 13 us a window at 100x100x6.)
      const int lane = tid & 31, warp = tid >> 5;
      int4* members = reinterpret_cast<int4*>(smem);
      if (warp == 0) {
        int cur = c->cursor;
        while (true) {
          const bool open = cur + lane >= pa.count || __ldcg(&pa.net_status[cur + lane]) == -1;
          const unsigned m = __ballot_sync(0xffffffffu, open);
          cur += m ? __ffs(m) - 1 : 32;
          if (m) break;
        }
        cur = min(cur, pa.count);
        if (lane == 0) {
          c->cursor = cur;
          c->fb = 0;
          s_win[0] = cur;
          s_win[1] = 0;
        }
      }
      __syncthreads();
      const int k0 = s_win[0], kend = min(pa.count, k0 + 4 * wmax);
      int W = 0, nskip = 0;
      for (int kb = k0; kb < kend && W < wmax && s_win[1] == 0; kb += kWarps) {
        const int k = kb + warp;
        int32_t n = -1, R = 0;
        int4 box = make_int4(0, 0, 0, 0), grown = box;
        if (k < kend && __ldcg(&pa.net_status[k]) == -1) {      // (else done out of order earlier)
          n = pa.order[k];
          R = use_batch ? rb.roi_len[n] : -1;
          if (R > 0 && nslots > 0) {
            int x0 = rb.roi_box[4 * n], x1 = rb.roi_box[4 * n + 1], y0 = rb.roi_box[4 * n + 2], y1 = rb.roi_box[4 * n + 3];
            const int32_t ol = t.store_len[n];
            const int32_t* op = t.store_path + (int64_t)n * t.slot_cap;
            for (int i = lane; i < ol; i += 32) {
              const int32_t r = op[i] % plane;
              const int x = r % g.nx, y = r / g.nx;
              x0 = min(x0, x); x1 = max(x1, x);
              y0 = min(y0, y); y1 = max(y1, y);
            }
            box.x = __reduce_min_sync(0xffffffffu, x0); box.y = __reduce_max_sync(0xffffffffu, x1);
            box.z = __reduce_min_sync(0xffffffffu, y0); box.w = __reduce_max_sync(0xffffffffu, y1);
            const int32_t sr = t.net_src[n] % plane, dr = t.net_dst[n] % plane;
            const int sx = sr % g.nx, sy = sr / g.nx, dx = dr % g.nx, dy = dr / g.nx;
            const int m = t.net_depth[2 * n + 1] + t.net_halo[2 * n + 1];
            grown = make_int4(min(box.x, min(sx, dx) - m), max(box.y, max(sx, dx) + m),
                              min(box.z, min(sy, dy) - m), max(box.w, max(sy, dy) + m));
          }
        }
        if (lane == 0) {
          s_cand[warp] = make_int2(n, R);
          s_box[warp] = box;
          s_grown[warp] = grown;
        }
        __syncthreads();
        if (warp == 0) {
          bool end = false;
          for (int j = 0; j < kWarps && kb + j < kend && W < wmax && !end; ++j) {
            const int2 cand = s_cand[j];
            if (cand.x < 0) continue;
            if (cand.y <= 0 || nslots == 0) {
              // without a ROI from the batch, or one net at a time: alone
              if (W == 0 && nskip == 0) {
                if (lane == 0) { ws.k[0] = kb + j; ws.solo[0] = cand.y <= 0 ? 1 : 0; ws.inorder[0] = 1; }
                W = 1;
              }
              end = true;
              break;
            }
            const int4 bx = s_box[j];
            bool meet = lane < nskip && boxes_meet(bx, s_skip[lane]);
            for (int m = lane; m < W; m += 32) meet = meet || boxes_meet(bx, members[m]);
            if (__any_sync(0xffffffffu, meet)) {
              if (nskip >= look) { end = true; break; }   // no look-ahead left: the window ends here
              if (lane == 0) s_skip[nskip] = s_grown[j];
              ++nskip;
            } else {
              if (lane == 0) {
                ws.k[W] = kb + j;
                ws.solo[W] = 0;
                ws.inorder[W] = nskip == 0 ? 1 : 0;
                members[W] = bx;
              }
              ++W;
            }
            __syncwarp();
          }
          if (lane == 0) {
            s_win[1] = end ? 1 : 0;
            s_win[2] = W;
            s_win[3] = nskip;
          }
        }
        __syncthreads();
        W = s_win[2];
        nskip = s_win[3];
      }
      if (tid == 0) c->wsize = W;
      clk.mark(6);
    }
    if (!win_barrier(c, target, &s_bar)) break;
    const int W = *(volatile int32_t*)&c->wsize;
    if (W == 0 || *(volatile int32_t*)&c->error) break;
    // 2. rip-up, one member per CTA (and the ROI of a member without one)
    const bool solo = *(volatile int32_t*)&ws.solo[0] != 0;
    if (b < W) {
      const int32_t n = pa.order[ws.k[b]];
      const int32_t ol = t.store_len[n];
      int rc = OGR_OK;
      if (ol >= 2)
        rc = apply_path_dev(g, st, t.store_path + (int64_t)n * t.slot_cap, ol, t.net_id[n], -1, pa.pres_fac,
                            pa.live, nullptr, s_via, s_flags);
      if (tid < 4) ws.stats[4 * b + tid] = 0ull;
      if (nslots == 0 && tid == 0) t.store_len[n] = 0;   // (a window's rip-ups may yet be undone)
      if (solo && rc == OGR_OK) {
        const ogr_net_args a = ogr_pass_net_args(t, pa, n, 0);
        build_roi(sh, g, a, w, smem);
        rc = sh.status;
        if (tid == 0) c->solo_R = sh.R;
      } else if (use_batch && tid == 0) {
        atomicAdd(&g_stage[14], 1ull);
      }
      if (tid == 0 && rc != OGR_OK) atomicExch(&c->error, rc);
      if (b == 0) clk.mark(5);
    }
    if (!win_barrier(c, target, &s_bar)) break;
    if (*(volatile int32_t*)&c->error) {
      ripped_up(W);
      break;
    }
    // 3. search, one team of CTAs per member, paths into scratch
    const int T = min(kTeam, G / W), mem = b / T, rank = b - mem * T;
    if (mem < W) {
      const int32_t n = pa.order[ws.k[mem]];
      const ogr_net_args a = ogr_pass_net_args(t, pa, n, 0);
      const Ws mine = slot_of(mem, solo);
      const RoiJob job{&g, &st, &a, &mine,
                       solo ? w.roi : rb.roi_pool + (int64_t)n * rb.roi_cap,
                       solo ? *(volatile int32_t*)&c->solo_R : rb.roi_len[n],
                       nullptr, nullptr, path_of(mem, n), t.slot_cap, ws.stats + 4 * mem, rank, T};
      int status, len;
      roi_search_row<ROW, false>(job, smem, &status, &len);
      if (tid == 0 && rank == 0) {
        ws.st[mem] = status;
        ws.len[mem] = len;
        if (status < 0) atomicExch(&c->error, status);
      }
    }
    if (!win_barrier(c, target, &s_bar)) break;
    if (*(volatile int32_t*)&c->error) {
      ripped_up(W);
      break;
    }
    // 4. commit
    clk.start();
    if (b < W) clear_team(slot_of(b, solo).ctl);
    int ff = W;
    for (int m = 0; m < W; ++m)
      if (ws.st[m] != OGR_OK) { ff = m; break; }
    // With the pass's fallbacks used up (the count only grows, and only CTA 0
    // writes it, before a barrier) a failed member takes no fallback: it stays
    // unrouted with its old path ripped up, the state every member's search
    // already saw, so every member's result is the sequential pass's and all
    // of them are final -- in or out of order.
    const bool no_fallback = (int)__ldcg(reinterpret_cast<const long long*>(&w.result[2])) >= pa.fallback_quota;
    if (ff == W || no_fallback) {
      if (b < W) {
        const int32_t k = ws.k[b], n = pa.order[k];
        if (tid < 4) atomicAdd(&stats[tid], ws.stats[4 * b + tid]);
        if (ws.st[b] == OGR_OK) {
          const int rc = commit_from(g, st, t, pa, n, path_of(b, n), ws.len[b], s_via, s_flags);
          if (tid == 0) {
            pa.net_status[k] = 0;
            if (rc != OGR_OK) atomicExch(&c->error, rc);
          }
        } else if (tid == 0) {
          t.store_len[n] = 0;
          pa.net_status[k] = 1;
        }
      }
    } else if (b == 0) {
      int rc = OGR_OK;
      for (int m = 0; m < ff && rc == OGR_OK; ++m) {
        const int32_t k = ws.k[m], n = pa.order[k];
        rc = commit_from(g, st, t, pa, n, path_of(m, n), ws.len[m], s_via, s_flags);
        if (tid < 4) atomicAdd(&stats[tid], ws.stats[4 * m + tid]);
        if (tid == 0) pa.net_status[k] = 0;
        __syncthreads();
      }
      // A failed net with pending nets before it (taken out of order) must
      // not take its fallback yet: it is undone like the later members and
      // stays pending, to be searched again when its turn comes.
      const bool defer = !ws.inorder[ff];
      for (int m = defer ? ff : ff + 1; m < W && rc == OGR_OK; ++m) {   // undo the later rip-ups
        if (discarded != nullptr && tid == 0) {
          atomicAdd(&discarded[0], 1ull);
          atomicAdd(&discarded[1], ws.stats[4 * m + 0]);
          atomicAdd(&discarded[2], ws.stats[4 * m + 1]);
        }
        const int32_t n = pa.order[ws.k[m]];
        const int32_t ol = t.store_len[n];
        if (ol >= 2)
          rc = apply_path_dev(g, st, t.store_path + (int64_t)n * t.slot_cap, ol, t.net_id[n], +1, pa.pres_fac,
                              pa.live, nullptr, s_via, s_flags);
      }
      if (!defer) {
        // its fallback's ROI; a team searches it below
        const int32_t kf = ws.k[ff], nf = pa.order[kf];
        if (tid < 4) atomicAdd(&stats[tid], ws.stats[4 * ff + tid]);
        if (tid == 0) t.store_len[nf] = 0;
        __syncthreads();
        if (rc == OGR_OK) {
          const ogr_net_args a = ogr_pass_net_args(t, pa, nf, 1);
          build_roi(sh, g, a, w, smem);
          rc = sh.status;
          if (tid == 0) {
            c->solo_R = sh.R;
            c->fb = 1 + kf;
          }
        }
      }
      if (tid == 0 && rc != OGR_OK) atomicExch(&c->error, rc);
    }
    if (b == 0) clk.mark(5);
    if (!win_barrier(c, target, &s_bar)) break;
    if (*(volatile int32_t*)&c->error) break;
    const int fb = *(volatile int32_t*)&c->fb;
    if (fb == 0) continue;
    // 5. the fallback of the failed net
    const int32_t kf = fb - 1, nf = pa.order[kf];
    const int Tf = min(kTeam, G);
    if (b < Tf) {
      const ogr_net_args a = ogr_pass_net_args(t, pa, nf, 1);
      const RoiJob job{&g, &st, &a, &w, w.roi, *(volatile int32_t*)&c->solo_R, nullptr, nullptr,
                       t.store_path + (int64_t)nf * t.slot_cap, t.slot_cap, stats, b, Tf};
      int status, len;
      roi_search_row<ROW, false>(job, smem, &status, &len);
      if (tid == 0 && b == 0) {
        c->fb_st = status;
        c->fb_len = len;
        w.result[2] = w.result[2] + 1;
        if (status < 0) atomicExch(&c->error, status);
      }
    }
    if (!win_barrier(c, target, &s_bar)) break;
    if (*(volatile int32_t*)&c->error) break;
    if (b == 0) {
      const int fin = *(volatile int32_t*)&c->fb_st, len = *(volatile int32_t*)&c->fb_len;
      int flags = 2;
      if (fin == OGR_OK) {
        const int rc = apply_path_dev(g, st, t.store_path + (int64_t)nf * t.slot_cap, len, t.net_id[nf], +1,
                                      pa.pres_fac, pa.live, t.store_arcs + (int64_t)nf * 2 * t.slot_cap, s_via,
                                      s_flags);
        if (tid == 0) {
          if (rc == OGR_OK) t.store_len[nf] = len;
          else atomicExch(&c->error, rc);
        }
      } else {
        flags |= 1;
      }
      if (tid == 0) pa.net_status[kf] = flags;
      clear_team(w.ctl);
    }
    // (the next window's first barrier orders this before anyone reads it;
    // c->fb is cleared by CTA 0 only then, after every CTA has read it)
    if (!win_barrier(c, target, &s_bar)) break;
  }
  if (b == 0 && tid == 0) {
    if (*(volatile int32_t*)&c->bar_err) w.result[0] = OGR_ERR_TIMEOUT;
    else if (*(volatile int32_t*)&c->error) w.result[0] = *(volatile int32_t*)&c->error;
  }
}

__global__ void window_ws_init_kernel(char* base, int32_t slots, size_t slot_bytes, int32_t N, int32_t rmax) {
  for (int32_t sidx = 0; sidx < slots; ++sidx) {
    Ws t;
    ws_slot_layout(N, rmax, base + (size_t)sidx * slot_bytes, &t);
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = i0; i < N; i += step) t.g2r[i] = -1;
  }
}

// Claims and stamps of the window slots, cleared for every pass: they lie
// where the pass's own ROI limit puts them, over whatever a pass of another
// limit left there.  Only the node map, first in a slot, outlives a pass.
__global__ void window_claims_kernel(char* base, int32_t slots, size_t slot_bytes, int32_t N, int32_t rmax) {
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int32_t sidx = blockIdx.y; sidx < slots; sidx += gridDim.y) {
    Ws t;
    ws_slot_layout(N, rmax, base + (size_t)sidx * slot_bytes, &t);
    for (int64_t i = i0; i < rmax; i += step) t.claim[i] = 0;
    for (int64_t i = i0; i < (int64_t)(sizeof(SlotCtl) / 4); i += step) reinterpret_cast<int32_t*>(t.ctl)[i] = 0;
  }
}

// Long nets of a pass run as three launches each: this rip-up, the
// whole-lattice search on every SM (fullgraph.cu), then pass_full_tail_kernel.
__global__ void __launch_bounds__(kThreads, 1)
pass_ripup_kernel(ogr_graph g, ogr_state st, ogr_net_table t, ogr_pass_args pa, int32_t k, Ws w) {
  __shared__ int32_t s_via[kMaxViaNodes];
  __shared__ int s_flags[3];
  if (w.result[0] < 0) return;
  const int32_t n = pa.order[k];
  const int32_t old_len = t.store_len[n];
  if (old_len >= 2) {
    const int rc = apply_path_dev(g, st, t.store_path + (int64_t)n * t.slot_cap, old_len, t.net_id[n], -1,
                                  pa.pres_fac, pa.live, nullptr, s_via, s_flags);
    if (rc != OGR_OK) {
      if (threadIdx.x == 0) w.result[0] = rc;
      return;
    }
  }
  if (threadIdx.x == 0) t.store_len[n] = 0;
}

// After the whole-lattice search of net order[k]: the fallback ROI search if
// it failed and the pass has fallbacks left (at most five of a pass, by this
// one CTA), then the commit.
template <int ROW>
__global__ void __launch_bounds__(kThreads, 1)
pass_full_tail_kernel(ogr_graph g, ogr_state st, ogr_net_table t, ogr_pass_args pa, int32_t k, Ws w,
                      const int32_t* full_res) {
  extern __shared__ __align__(16) char smem[];
  __shared__ Shared sh;
  __shared__ int s_flags[3];
  int32_t* s_via = reinterpret_cast<int32_t*>(smem);
  if (w.result[0] < 0) return;
  const int32_t n = pa.order[k];
  int32_t* slot = t.store_path + (int64_t)n * t.slot_cap;
  int32_t* arcs = t.store_arcs + (int64_t)n * 2 * t.slot_cap;
  int fin = full_res[0];
  int len = full_res[1];
  if (fin < 0) {
    if (threadIdx.x == 0) w.result[0] = fin;
    return;
  }
  int flags = 0;
  const int used = (int)w.result[2];
  if (fin != OGR_OK && used < pa.fallback_quota) {
    const ogr_net_args a = ogr_pass_net_args(t, pa, n, 1);
    build_roi(sh, g, a, w, smem);
    fin = sh.status;
    if (fin == OGR_OK) {
      clear_team(w.ctl);
      __syncthreads();
      const RoiJob job{&g, &st, &a, &w, w.roi, sh.R, nullptr, nullptr, slot, t.slot_cap,
                       reinterpret_cast<unsigned long long*>(pa.stats), 0, 1};
      roi_search_row<ROW, false>(job, smem, &fin, &len);
    }
    if (fin < 0) {
      if (threadIdx.x == 0) w.result[0] = fin;
      return;
    }
    flags |= 2;
    __syncthreads();
    if (threadIdx.x == 0) w.result[2] = used + 1;
  }
  __syncthreads();
  if (fin == OGR_OK) {
    const int rc = apply_path_dev(g, st, slot, len, t.net_id[n], +1, pa.pres_fac, pa.live, arcs, s_via, s_flags);
    if (rc != OGR_OK) {
      if (threadIdx.x == 0) w.result[0] = rc;
      return;
    }
    if (threadIdx.x == 0) t.store_len[n] = len;
  } else {
    flags |= 1;
  }
  if (threadIdx.x == 0) pa.net_status[k] = flags;
}

// Variants by the arcs of a row (phases.cuh).
#define OGR_WITH_ROW(ROWV, g, ...)                             \
  do {                                                         \
    switch (ogr_full::row_for(g)) {                            \
      case 4: { constexpr int ROWV = 4; __VA_ARGS__; } break;  \
      case 8: { constexpr int ROWV = 8; __VA_ARGS__; } break;  \
      case 16: { constexpr int ROWV = 16; __VA_ARGS__; } break;\
      default: { constexpr int ROWV = 32; __VA_ARGS__; } break;\
    }                                                          \
  } while (0)

cudaError_t wide_smem(const void* f) {
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ogr_phase::kSmemBytes);
}

// A cooperative launch of `grid` CTAs, all of them resident.
int launch_team(const void* f, int grid, void** args, cudaStream_t s) {
  OGR_CUDA_TRY(wide_smem(f));
  OGR_CUDA_TRY(cudaLaunchCooperativeKernel(f, dim3(grid), dim3(kThreads), args, ogr_phase::kSmemBytes, s));
  return OGR_OK;
}

// The search of a net in workspace w (ROI built here if roi is NULL) on s.
int launch_find(const ogr_graph& g, const ogr_state& st, const ogr_net_args& a, const Ws& w, const int32_t* roi,
                int32_t R, const float* roi_pen, const MultiSeeds* ms, int32_t* path_out, int32_t path_cap,
                int64_t* stats, cudaStream_t s) {
  OGR_CUDA_TRY(cudaMemsetAsync(&w.ctl->team, 0, sizeof(ogr_phase::Ctl), s));
  if (roi == nullptr && !a.full_graph) {
    OGR_CUDA_TRY(wide_smem((const void*)build_roi_kernel));
    build_roi_kernel<<<kBfsCtas, kClusterThreads, ogr_phase::kSmemBytes, s>>>(g, a, w);
    OGR_LAUNCH_CHECK();
  }
  if (a.full_graph) R = g.num_nodes;
  ogr_graph gv = g;
  ogr_state sv = st;
  ogr_net_args av = a;
  Ws wv = w;
  MultiSeeds mv = ms ? *ms : MultiSeeds{};
  void* args[] = {&gv, &sv, &av, &wv, &roi, &R, &roi_pen, &mv, &path_out, &path_cap, &stats};
  // a team within this host thread's share of the SMs (ogr_full_grid): a
  // cooperative launch wider than that waits for other jobs' searches to end
  const int share = ogr_full::grid_blocks();
  if (share < 1) return OGR_ERR_CUDA;
  const void* f = nullptr;
  OGR_WITH_ROW(ROW, g, f = ms ? (const void*)find_team_kernel<ROW, true> : (const void*)find_team_kernel<ROW, false>);
  return launch_team(f, share < kTeam ? share : kTeam, args, s);
}

}  // namespace

extern "C" size_t ogr_route_workspace_bytes(int32_t num_nodes) { return ws_layout(num_nodes, nullptr, nullptr); }

extern "C" size_t ogr_bfs_workspace_bytes(int32_t num_nodes, int64_t qcap, int32_t slots) {
  return bfs_slot_bytes(num_nodes, qcap) * (size_t)slots;
}

extern "C" int ogr_bfs_workspace_init(void* ws, int32_t num_nodes, int64_t qcap, int32_t slots, void* stream) {
  if (!ws || slots < 1 || qcap < 1) return OGR_ERR_ARG;
  bfs_init_kernel<<<ogr_blocks(num_nodes, 256), 256, 0, ogr_stream(stream)>>>(
      (char*)ws, slots, bfs_slot_bytes(num_nodes, qcap), num_nodes, qcap);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

extern "C" size_t ogr_window_workspace_bytes(int32_t num_nodes, int32_t max_roi_nodes, int32_t slots) {
  const int32_t r = max_roi_nodes < num_nodes ? max_roi_nodes : num_nodes;
  return ws_slot_layout(num_nodes, r, nullptr, nullptr) * (size_t)(slots > 0 ? slots : 0);
}

extern "C" int ogr_window_workspace_init(void* ws, int32_t num_nodes, int32_t max_roi_nodes, int32_t slots,
                                         void* stream) {
  if (!ws || slots < 1 || num_nodes < 1 || max_roi_nodes < 1) return OGR_ERR_ARG;
  const int32_t r = max_roi_nodes < num_nodes ? max_roi_nodes : num_nodes;
  window_ws_init_kernel<<<ogr_blocks(num_nodes, 256), 256, 0, ogr_stream(stream)>>>(
      (char*)ws, slots, ws_slot_layout(num_nodes, r, nullptr, nullptr), num_nodes, r);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

static_assert(sizeof(SlotCtl) % 4 == 0, "cleared as words");

extern "C" size_t ogr_window_ctl_bytes(int32_t slots) { return win_ctl_layout(slots, nullptr, nullptr, nullptr); }

extern "C" int ogr_window_lookahead(int32_t nets, int32_t* current) {
  if (nets < -1 || nets > kMaxSkip) return OGR_ERR_ARG;
  if (nets >= 0) g_window_look = nets;
  if (current) *current = g_window_look;
  return OGR_OK;
}

extern "C" int ogr_search_lanes(int32_t lanes, int32_t* current) {
  if (lanes != 0 && lanes != 2 && lanes != 4 && lanes != 8 && lanes != 16) return OGR_ERR_ARG;
  if (lanes != 0) g_search_lanes = lanes;
  if (current) *current = g_search_lanes;
  return OGR_OK;
}

extern "C" int ogr_search_profile(int64_t* out16, int32_t reset) {
  if (!out16) return OGR_ERR_ARG;
  OGR_CUDA_TRY(cudaMemcpyFromSymbol(out16, g_stage, sizeof(unsigned long long) * 16));
  if (reset) {
    unsigned long long z[16] = {};
    OGR_CUDA_TRY(cudaMemcpyToSymbol(g_stage, z, sizeof(z)));
  }
  return OGR_OK;
}

extern "C" int ogr_route_workspace_init(void* ws, size_t bytes, int32_t N, void* stream) {
  if (!ws || bytes < ogr_route_workspace_bytes(N)) return OGR_ERR_CAPACITY;
  Ws w;
  ws_layout(N, (char*)ws, &w);
  ws_init_kernel<<<ogr_blocks(N, 256), 256, 0, ogr_stream(stream)>>>(w, N);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

extern "C" int ogr_find_path(const ogr_graph* g, const ogr_state* st, const ogr_net_args* net, void* ws,
                             size_t bytes, int32_t* path_out, int32_t path_cap, int32_t* path_len_out,
                             int64_t* stats, void* stream) {
  if (!g || !st || !net || !ws || !path_out || !path_len_out) return OGR_ERR_ARG;
  if (bytes < ogr_route_workspace_bytes(g->num_nodes)) return OGR_ERR_CAPACITY;
  if (net->src < 0 || net->dst < 0 || net->src >= g->num_nodes || net->dst >= g->num_nodes) return OGR_ERR_ARG;
  Ws w;
  ws_layout(g->num_nodes, (char*)ws, &w);
  cudaStream_t s = ogr_stream(stream);
  const int rc = launch_find(*g, *st, *net, w, nullptr, 0, nullptr, nullptr, path_out, path_cap, stats, s);
  if (rc != OGR_OK) return rc;
  int64_t res[2];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = (res[0] == OGR_OK) ? (int32_t)res[1] : 0;
  return (int)res[0];
}

extern "C" int ogr_find_path_roi(const ogr_graph* g, const float* costs, const int32_t* roi_nodes, int32_t n_roi,
                                 const float* roi_penalty, int32_t src, int32_t dst, void* ws, size_t bytes,
                                 int32_t* path_out, int32_t path_cap, int32_t* path_len_out, int64_t* stats,
                                 void* stream) {
  if (!g || !costs || !roi_nodes || !ws || !path_out || !path_len_out || n_roi < 0 || n_roi > g->num_nodes)
    return OGR_ERR_ARG;
  if (bytes < ogr_route_workspace_bytes(g->num_nodes)) return OGR_ERR_CAPACITY;
  if (src < 0 || dst < 0 || src >= g->num_nodes || dst >= g->num_nodes) return OGR_ERR_ARG;
  *path_len_out = 0;
  if (n_roi == 0) return OGR_NO_PATH;
  Ws w;
  ws_layout(g->num_nodes, (char*)ws, &w);
  ogr_state st{};
  st.total_cost = const_cast<float*>(costs);
  ogr_net_args a{};
  a.net_id = -1;
  a.src = src;
  a.dst = dst;
  a.full_graph = 0;
  a.penalty_enabled = 0;
  cudaStream_t s = ogr_stream(stream);
  const int rc = launch_find(*g, st, a, w, roi_nodes, n_roi, roi_penalty, nullptr, path_out, path_cap, stats, s);
  if (rc != OGR_OK) return rc;
  int64_t res[2];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = (res[0] == OGR_OK) ? (int32_t)res[1] : 0;
  return (int)res[0];
}

extern "C" size_t ogr_multi_workspace_bytes(int32_t num_nodes) {
  return ogr_route_workspace_bytes(num_nodes) + 2 * round256(8 * (size_t)(num_nodes > 0 ? num_nodes : 0));
}

extern "C" int ogr_find_path_multi(const ogr_graph* g, const float* costs, const int32_t* roi_nodes, int32_t n_roi,
                                   const float* roi_penalty, const int32_t* seeds, const double* seed_cost,
                                   int32_t n_seeds, const int32_t* targets, const double* target_cost,
                                   int32_t n_targets, void* ws, size_t bytes, int32_t* path_out, int32_t path_cap,
                                   int32_t* path_len_out, int64_t* stats, void* stream) {
  if (!g || !costs || !roi_nodes || !ws || !path_out || !path_len_out || n_roi < 0 || n_roi > g->num_nodes ||
      n_seeds < 0 || n_targets < 0 || (n_seeds > 0 && (!seeds || !seed_cost)) ||
      (n_targets > 0 && (!targets || !target_cost)))
    return OGR_ERR_ARG;
  if (bytes < ogr_multi_workspace_bytes(g->num_nodes)) return OGR_ERR_CAPACITY;
  *path_len_out = 0;
  if (n_roi == 0 || n_seeds == 0 || n_targets == 0) return OGR_NO_PATH;
  Ws w;
  const size_t base = ws_layout(g->num_nodes, (char*)ws, &w);
  MultiSeeds ms{};
  ms.seeds = seeds;
  ms.seed_cost = seed_cost;
  ms.nseeds = n_seeds;
  ms.targets = targets;
  ms.target_cost = target_cost;
  ms.ntargets = n_targets;
  ms.init = (double*)((char*)ws + base);
  ms.tcost = (double*)((char*)ws + base + round256(8 * (size_t)g->num_nodes));
  ogr_state st{};
  st.total_cost = const_cast<float*>(costs);
  ogr_net_args a{};
  a.net_id = -1;
  a.src = -1;
  a.dst = -1;
  a.full_graph = 0;
  a.penalty_enabled = 0;
  cudaStream_t s = ogr_stream(stream);
  const int rc = launch_find(*g, st, a, w, roi_nodes, n_roi, roi_penalty, &ms, path_out, path_cap, stats, s);
  if (rc != OGR_OK) return rc;
  int64_t res[2];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = (res[0] == OGR_OK) ? (int32_t)res[1] : 0;
  return (int)res[0];
}

extern "C" int ogr_extract_roi(const ogr_graph* g, const ogr_net_args* net, void* ws, size_t bytes,
                               int32_t* roi_out, int32_t roi_cap, int32_t* roi_len_out, void* stream) {
  if (!g || !net || !ws || !roi_out || !roi_len_out) return OGR_ERR_ARG;
  if (bytes < ogr_route_workspace_bytes(g->num_nodes)) return OGR_ERR_CAPACITY;
  if (!net->full_graph && roi_cap < (net->max_roi_nodes < g->num_nodes ? net->max_roi_nodes : g->num_nodes))
    return OGR_ERR_ARG;
  Ws w;
  ws_layout(g->num_nodes, (char*)ws, &w);
  cudaStream_t s = ogr_stream(stream);
  OGR_CUDA_TRY(wide_smem((const void*)roi_kernel));
  roi_kernel<<<kBfsCtas, kClusterThreads, ogr_phase::kSmemBytes, s>>>(*g, *net, w, roi_out, roi_cap);
  OGR_LAUNCH_CHECK();
  int64_t res[2];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *roi_len_out = (int32_t)res[1];
  return (int)res[0];
}

extern "C" int ogr_paths_commit(const ogr_graph* g, const ogr_state* st, const int32_t* nodes, const int32_t* offsets,
                                const int32_t* net_ids, int32_t n_paths, int32_t* arcs_out, int32_t* store_path,
                                int32_t* store_len, int32_t* store_arcs, const int32_t* store_slot, int32_t slot_cap,
                                int32_t* status_dev, void* stream) {
  if (!g || !st || n_paths < 0 || !status_dev) return OGR_ERR_ARG;
  if (n_paths == 0) return OGR_OK;
  if (!nodes || !offsets || !net_ids || !arcs_out ||
      ((store_path || store_len || store_arcs) && (!store_slot || slot_cap < 2)))
    return OGR_ERR_ARG;
  cudaStream_t s = ogr_stream(stream);
  OGR_CUDA_TRY(cudaMemsetAsync(status_dev, 0, sizeof(int32_t), s));
  const int grid = n_paths < 152 * 8 ? n_paths : 152 * 8;
  paths_commit_kernel<<<grid, kApplyThreads, 0, s>>>(*g, *st, nodes, offsets, net_ids, n_paths, arcs_out, store_path,
                                                      store_len, store_arcs, store_slot, slot_cap, status_dev);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

extern "C" int ogr_path_apply(const ogr_graph* g, const ogr_state* st, const int32_t* path, int32_t len,
                              int32_t net_id, int32_t sign, float pres_fac_f32, int32_t live, int32_t* arcs_out,
                              int32_t* status_dev, void* stream) {
  if (!g || !st || !path || !status_dev || len < 2 || (sign != 1 && sign != -1)) return OGR_ERR_ARG;
  path_apply_kernel<<<1, kApplyThreads, 0, ogr_stream(stream)>>>(*g, *st, path, len, net_id, sign, pres_fac_f32,
                                                                   live, arcs_out, status_dev);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

extern "C" int ogr_route_pass(const ogr_graph* g, const ogr_state* st, const ogr_net_table* t,
                              const ogr_pass_args* pa, const ogr_roi_batch* rb, void* ws, size_t bytes,
                              const uint8_t* order_full, void* full_ws, size_t full_bytes,
                              const ogr_window_args* win, int32_t* status_out, void* stream) {
  if (!g || !st || !t || !pa || !ws || !status_out) return OGR_ERR_ARG;
  if (bytes < ogr_route_workspace_bytes(g->num_nodes)) return OGR_ERR_CAPACITY;
  if (pa->count < 0 || t->slot_cap < 2) return OGR_ERR_ARG;
  if (pa->count == 0) {
    *status_out = OGR_OK;
    return OGR_OK;
  }
  if (!pa->order || !pa->net_status || !pa->stats) return OGR_ERR_ARG;
  const bool batch = rb != nullptr && rb->slots > 0;
  const int32_t need_cap = pa->max_roi_nodes < g->num_nodes ? pa->max_roi_nodes : g->num_nodes;
  if (batch && (!rb->bfs_ws || !rb->roi_pool || !rb->roi_len || !rb->next || rb->roi_cap < need_cap))
    return OGR_ERR_ARG;
  bool any_full = false;
  if (order_full)
    for (int32_t k = 0; k < pa->count; ++k) any_full = any_full || order_full[k] != 0;
  if (any_full && (!full_ws || full_bytes < ogr_full::workspace_bytes(g->num_nodes, g->num_edges)))
    return OGR_ERR_CAPACITY;
  Ws w;
  ws_layout(g->num_nodes, (char*)ws, &w);
  cudaStream_t s = ogr_stream(stream);
  // result[0] = first error of the pass, result[2] = fallbacks used so far
  OGR_CUDA_TRY(cudaMemsetAsync(w.result, 0, 64, s));
  ogr_roi_batch rbv{};
  if (batch) {
    rbv = *rb;
    OGR_CUDA_TRY(cudaMemsetAsync(rbv.next, 0, sizeof(int32_t), s));
    OGR_CUDA_TRY(wide_smem((const void*)roi_batch_kernel));
    roi_batch_kernel<<<rbv.slots, kBfsThreads, ogr_phase::kSmemBytes, s>>>(*g, *t, *pa, rbv);
    OGR_LAUNCH_CHECK();
  }
  const bool windows = win != nullptr && win->slots > 0 && batch && rbv.roi_box != nullptr;
  // CTAs: one team per window member, within this host thread's share of the
  // SMs (ogr_full_grid)
  const int share = ogr_full::grid_blocks();
  if (share < 1) return OGR_ERR_CUDA;
  int nslots = 0;
  if (windows) {
    if (!win->ws || !win->scratch || !win->ctl ||
        win->slot_bytes < ogr_window_workspace_bytes(g->num_nodes, pa->max_roi_nodes, 1))
      return OGR_ERR_ARG;
    nslots = win->slots < share ? win->slots : share;
    window_claims_kernel<<<dim3(8, nslots), 256, 0, s>>>((char*)win->ws, nslots, win->slot_bytes, g->num_nodes, need_cap);
    OGR_LAUNCH_CHECK();
  }
  const int64_t want = (int64_t)(nslots > 0 ? nslots : 1) * kTeam;
  const int grid = want < share ? (int)want : share;
  // one run of ROI nets: batched windows, or one net at a time
  auto roi_segment = [&](const ogr_pass_args& seg) -> int {
    char* ctl = windows ? (char*)win->ctl : w.win1;
    OGR_CUDA_TRY(cudaMemsetAsync(ctl, 0, ogr_window_ctl_bytes(nslots > 0 ? nslots : 1), s));
    // every net of the segment starts pending (-1); the window pass sets its status when done
    OGR_CUDA_TRY(cudaMemsetAsync(seg.net_status, 0xff, sizeof(int32_t) * (size_t)seg.count, s));
    int32_t lookv = g_window_look < 0 ? 0 : (g_window_look > kMaxSkip ? kMaxSkip : g_window_look);
    ogr_graph gv = *g;
    ogr_state sv = *st;
    ogr_net_table tv = *t;
    ogr_pass_args pv = seg;
    int use_batch = batch ? 1 : 0;
    char* slot_base = windows ? (char*)win->ws : nullptr;
    size_t slot_bytes = windows ? win->slot_bytes : 0;
    int32_t rmax = need_cap;
    int32_t* scratch = windows ? win->scratch : nullptr;
    Ws wv = w;
    unsigned long long* discarded = windows ? reinterpret_cast<unsigned long long*>(win->discarded) : nullptr;
    void* args[] = {&gv, &sv, &tv, &pv, &rbv, &use_batch, &slot_base, &slot_bytes, &rmax, &nslots, &scratch, &ctl,
                    &wv, &lookv, &discarded};
    const void* wk = nullptr;
    OGR_WITH_ROW(ROW, *g, wk = (const void*)window_pass_kernel<ROW>);
    return launch_team(wk, grid, args, s);
  };
  if (!any_full) {
    const int rc = roi_segment(*pa);
    if (rc != OGR_OK) return rc;
  } else {
    // Runs of ROI nets go through one launch each; every long net
    // gets the whole GPU for its search.  Same order, same state updates.
    int32_t* full_res = ogr_full::result_words(full_ws, g->num_nodes, g->num_edges);
    int32_t k = 0;
    while (k < pa->count) {
      if (order_full[k]) {
        pass_ripup_kernel<<<1, kThreads, 0, s>>>(*g, *st, *t, *pa, k, w);
        OGR_LAUNCH_CHECK();
        ogr_full::Job job{};
        job.from_pass = 1;
        job.t = *t;
        job.pa = *pa;
        job.k = k;
        job.pass_result = w.result;
        job.stats = reinterpret_cast<unsigned long long*>(pa->stats);
        const int rc = ogr_full::launch(*g, *st, job, full_ws, s);
        if (rc != OGR_OK) return rc;
        OGR_WITH_ROW(ROW, *g, {
          OGR_CUDA_TRY(wide_smem((const void*)pass_full_tail_kernel<ROW>));
          pass_full_tail_kernel<ROW><<<1, kThreads, ogr_phase::kSmemBytes, s>>>(*g, *st, *t, *pa, k, w, full_res);
        });
        OGR_LAUNCH_CHECK();
        ++k;
      } else {
        int32_t k1 = k;
        while (k1 < pa->count && !order_full[k1]) ++k1;
        ogr_pass_args seg = *pa;
        seg.order = pa->order + k;
        seg.count = k1 - k;
        seg.net_status = pa->net_status + k;
        const int rc = roi_segment(seg);
        if (rc != OGR_OK) return rc;
        k = k1;
      }
    }
  }
  int64_t res;
  OGR_CUDA_TRY(cudaMemcpyAsync(&res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *status_out = (int32_t)res;
  return res < 0 ? (int)res : OGR_OK;
}

// ---- allocation-free search ----------------------------------------------------
// Some hosts cannot hand this library a workspace: a plugin loaded into an
// application that owns the device allocator, or a serving process that
// reserves its whole memory budget at start-up and forbids allocations on the
// request path.  ogr_find_path_noalloc runs the same search as ogr_find_path
// with its scratch in a fixed device array that lives in this library's image
// (resident on every GPU that loads the library until the process exits).
//
// Limits and rules:
//  - at most OGR_NOALLOC_MAX_NODES lattice nodes; larger graphs are rejected
//    with OGR_ERR_CAPACITY before anything is launched;
//  - the first call on a device looks up the array's device address for that
//    device (cudaGetSymbolAddress); make that first call before any stream
//    capture;
//  - all calls share the one array: each call re-initialises the parts the
//    search needs cleared, and calls that overlap on the GPU (another stream,
//    another host thread) race on it — serialise them.
namespace {

constexpr size_t noalloc_ws_bytes() { return ws_bytes_for((size_t)OGR_NOALLOC_MAX_NODES); }

static __device__ __align__(256) unsigned char g_noalloc_ws[noalloc_ws_bytes()];

constexpr int kMaxDevices = 64;
// Device address of the array per device, looked up on the first call there
// (atomic: concurrent first calls from several host threads store the same
// value).  A device reset invalidates it; the process does not reset here.
std::atomic<void*> g_noalloc_ptr[kMaxDevices] = {};

}  // namespace

extern "C" int ogr_find_path_noalloc(const ogr_graph* g, const ogr_state* st, const ogr_net_args* net,
                                     int32_t* path_out, int32_t path_cap, int32_t* path_len_out, int64_t* stats,
                                     void* stream) {
  if (!g || !st || !net || !path_out || !path_len_out) return OGR_ERR_ARG;
  if (g->num_nodes < 1 || g->num_nodes > OGR_NOALLOC_MAX_NODES) return OGR_ERR_CAPACITY;
  if (net->src < 0 || net->dst < 0 || net->src >= g->num_nodes || net->dst >= g->num_nodes) return OGR_ERR_ARG;
  int dev = 0;
  OGR_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return OGR_ERR_ARG;
  void* base = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (base == nullptr) {
    OGR_CUDA_TRY(cudaGetSymbolAddress(&base, g_noalloc_ws));
    g_noalloc_ptr[dev].store(base, std::memory_order_release);
  }
  const size_t need = ws_layout(g->num_nodes, nullptr, nullptr);
  if (need > noalloc_ws_bytes()) return OGR_ERR_CAPACITY;
  Ws w;
  ws_layout(g->num_nodes, (char*)base, &w);
  cudaStream_t s = ogr_stream(stream);
  // The array keeps whatever the previous call left: clear seen[] / g2r[] / claims.
  ws_init_kernel<<<ogr_blocks(g->num_nodes, 256), 256, 0, s>>>(w, g->num_nodes);
  const int rc = launch_find(*g, *st, *net, w, nullptr, 0, nullptr, nullptr, path_out, path_cap, stats, s);
  if (rc != OGR_OK) return rc;
  int64_t res[2];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, w.result, sizeof(res), cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = (res[0] == OGR_OK) ? (int32_t)res[1] : 0;
  return (int)res[0];
}
