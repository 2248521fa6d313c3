// A7 for long nets: the exact search over the whole lattice on every SM.
//
// The reference searches nets whose Manhattan length is 125 steps or more on
// the full graph (_route_all, unified_pathfinder.py:8219-8262: roi_nodes =
// arange(N)), so its heap Dijkstra (find_path_roi, :2451-2548) settles every
// node cheaper than dst — most of a 600x400x12 lattice.  The result here is
// the same as the heap's: every node takes the lexicographic minimum of
// (float32(alt), L(u), u) over its in-neighbours u, alt = (L(u) + c) + pen.
//
// The search itself is phases.cuh with every SM in one team: one CTA per SM,
// launched cooperatively so that all of them are resident; its barrier gives
// up after a bounded wait and reports OGR_ERR_TIMEOUT.  A launch first writes
// every node's record (penalty, row bounds): a stream over the node arrays
// (600x400x12: 37 us of a search of 3.6 ms) that spares each phase the
// four loads of the penalty and the two of the row bounds per neighbour.
#include <atomic>

#include "fullgraph.cuh"
#include "phases.cuh"

namespace {

using namespace ogr_phase;

// The tuning knobs below are per host thread: each job of a server routes in
// its own thread and keeps its own settings.
// Accepted and kept for callers (ogr_full_lanes, ogr_full_reuse): results
// never depended on them, and the search fits its lanes to the lattice's rows
// and keeps an entry's row with its CTA.
thread_local int g_full_lanes = 16;
thread_local int g_full_reuse = 0;
constexpr unsigned kBarSpin = 1u << 22;
// Limits for tests of failure handling (ogr_debug_limits): the spin bound of a
// search team's barrier and a cap on settle phases, of whole-lattice and ROI
// searches alike; the defaults are kBarSpin and 2N + 4 (no search needs more).
thread_local unsigned g_dbg_spin = kBarSpin;
thread_local int g_dbg_phases = 0;

struct FCtl {
  Ctl team;                                    // cleared before every launch
  alignas(128) int32_t res[4];
  int32_t sid;                                 // searches so far: the claim stamp, kept across searches
  int32_t tile_gate;                           // 1: the tile engine handed this net over
  int32_t merr;                                // multi-source: a bad or repeated seed / target
};

// Multi-source searches mark seeds and targets in per-node doubles that hold
// this NaN pattern otherwise (written by the workspace init, restored by
// every search).
constexpr unsigned long long kNoTerm = 0x7ff8deadbeef0001ull;

struct FWs {
  Rec* rec;
  int32_t* par;              // winning in-neighbour of a settled node
  int32_t* claim;
  float* rcost;              // reverse-arc cost gather when the state carries none
  int4* ov[2];               // surplus lists
  unsigned bar_spin;         // barrier spin bound
  int32_t max_phases;        // > 0: cap on settle phases (else 2N + 4)
  FCtl* ctl;
  char* tile;                // scratch of the tile-window engine
  double* mseed;             // multi-source: seed cost per node (kNoTerm bits otherwise)
  double* mtgt;              // multi-source: target cost per node (kNoTerm bits otherwise)
};

constexpr size_t r256(size_t v) { return (v + 255) & ~(size_t)255; }

size_t fws_layout(int32_t N, int64_t E, char* base, FWs* w) {
  size_t off = 0;
  auto take = [&](size_t b) -> char* {
    char* p = base ? base + off : nullptr;
    off += r256(b);
    return p;
  };
  const size_t n = (size_t)N;
  FWs t{};
  t.ctl = (FCtl*)take(sizeof(FCtl));
  t.rec = (Rec*)take(16 * n);
  t.par = (int32_t*)take(4 * n);
  t.claim = (int32_t*)take(4 * n);
  t.rcost = (float*)take(4 * (size_t)E);
  for (int i = 0; i < 2; ++i) t.ov[i] = (int4*)take(16 * n);
  t.tile = take(ogr_tile::workspace_bytes(N));
  t.mseed = (double*)take(8 * n);
  t.mtgt = (double*)take(8 * n);
  if (w) *w = t;
  return off;
}

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Tracing counters of the whole-lattice search (read with ogr_full_profile):
// [0] searches, [1] phases, [2] kernel ns, [3] init ns (CTA 0), [4] phase
// work ns (CTA 0), [5] frontier entries examined, [6] barrier wait ns
// (CTA 0), [7] statistics + backtrace ns (CTA 0).
__device__ unsigned long long g_full_prof[8];

template <int L, int K, bool kMulti>
__global__ void __launch_bounds__(kThreads, 1)
full_sssp_kernel(ogr_graph g, ogr_state st, ogr_full::Job job, FWs w) {
  extern __shared__ __align__(16) char smem_raw[];
  Head& sm = *reinterpret_cast<Head*>(smem_raw);
  const int tid = threadIdx.x;
  const int64_t gthreads = (int64_t)gridDim.x * kThreads;
  const int64_t gtid = (int64_t)blockIdx.x * kThreads + tid;
  const bool leader = gtid == 0;
  FCtl* ctl = w.ctl;

  if (job.from_pass && job.pass_result[0] < 0) return;  // uniform: written by an earlier launch
  if (job.gated && __ldcg(&ctl->tile_gate) == 0) return;  // uniform: the tile engine found the result
  ogr_net_args a = job.a;
  int32_t* path_out = job.path_out;
  int32_t path_cap = job.path_cap;
  if (job.from_pass) {
    const int32_t n = job.pa.order[job.k];
    a = ogr_pass_net_args(job.t, job.pa, n, 0);
    path_out = job.t.store_path + (int64_t)n * job.t.slot_cap;
    path_cap = job.t.slot_cap;
  }
  const int32_t N = g.num_nodes;
  const int32_t src = kMulti ? -1 : a.src, dst = kMulti ? -1 : a.dst;
  if (!kMulti && src == dst) {
    if (leader) {
      ctl->res[0] = OGR_NO_PATH;
      ctl->res[1] = 0;
      ctl->res[2] = 0;
    }
    return;
  }
  unsigned long long t_start = 0, t_init = 0, t_loop = 0;
  if (leader) t_start = gtimer();
  const int32_t* __restrict__ indptr = g.indptr;
  // claim stamps count the searches (two for one that goes over to doubles);
  // when the count runs out they are cleared
  int32_t sid = __ldcg(&ctl->sid) + 1;
  const bool wrap = sid < 1 || sid == 0x7fffffff;
  if (wrap) {
    sid = 1;
    for (int64_t i = gtid; i < N; i += gthreads) w.claim[i] = 0;
  }
  if (st.rcost == nullptr) {
    const int64_t E = g.num_edges;
#pragma unroll 4
    for (int64_t e = gtid; e < E; e += gthreads) w.rcost[e] = st.total_cost[g.rev[e]];
  }
  Problem pr{};
  pr.R = N;
  pr.src = src;
  pr.dst = dst;
  pr.indptr = indptr;
  pr.indices = g.indices;
  pr.rev = g.rev;
  pr.cost = st.total_cost;
  pr.rcost = st.rcost ? st.rcost : w.rcost;
  pr.rec = w.rec;
  pr.par = w.par;
  pr.claim = w.claim;
  pr.ov[0] = w.ov[0];
  pr.ov[1] = w.ov[1];
  pr.mseed = w.mseed;
  pr.ctl = &ctl->team;
  pr.rank = blockIdx.x;
  pr.nranks = gridDim.x;
  if (tid == 0) {
    sm.spin = w.bar_spin;
    sm.max_phase = w.max_phases > 0 ? min(w.max_phases, 2 * N + 4) : 2 * N + 4;
    sm.first = 0;
  }
  // With statistics requested the search goes on after dst is settled until
  // every node with a label <= L(dst) is settled (T > L(dst)): the IN bound
  // can settle dst before cheaper nodes, which the heap pops earlier.
  pr.want_stats = job.stats != nullptr;
  Outcome o{};
  bool fix = true;
  pr.sid = sid;
  // every node's record
  int md = 0;
#pragma unroll 4
  for (int64_t i = gtid; i < N; i += gthreads) {
    const int32_t f0 = indptr[i], f1 = indptr[i + 1];
    md = max(md, f1 - f0);
    const float pen = ogr_node_penalty(st, a, (int32_t)i);
    __stcg(reinterpret_cast<int4*>(&w.rec[i]), make_int4(f0, f1 - f0, 0, __float_as_int(pen)));
  }
  md = __reduce_max_sync(0xffffffffu, md);
  if ((tid & 31) == 0) sm.wmin[tid >> 5] = (unsigned long long)md;
  // Thread 0: the first frontier (the leader's nf0 entries, their least label
  // t0) at the second barrier.
  auto enter = [&](int nf0, unsigned long long t0) {
    if (leader) {
      ctl->team.nov[0] = nf0;
      ctl->team.nov[1] = 0;
      ctl->team.nov[2] = 0;
      t_init = gtimer();
    }
    if (sm.ok) {
      arrive(pr, sm, 1, kArrive + kOut * (unsigned long long)(nf0 < (int)kMostOut ? nf0 : (int)kMostOut) + kCount * (unsigned long long)nf0, t0);
      await(pr, sm, 1);
    }
    if (leader) t_loop = gtimer();
  };
  __syncthreads();
  if (tid == 0) {
    unsigned long long t0 = kNone;
    int nf0 = 0;
    sm.ok = 1;
    // The records are written and the longest row is known (it travels in
    // the word's maximum).  Several seeds may settle in one phase, each the
    // other's neighbour, so only now are their records marked reached.
    for (int i = 1; i < kWarps; ++i) md = max(md, (int)sm.wmin[i]);
    arrive(pr, sm, 0, kArrive, ~(unsigned long long)md);
    await(pr, sm, 0);
    sm.res[2] = (int)sm.t;
    if (leader && !kMulti) {
      w.claim[src] = pr.sid;
      w.ov[0][0] = make_int4(src, indptr[src], indptr[src + 1] - indptr[src], __float_as_int(0.0f));
      nf0 = 1;
      t0 = 0ull;
    }
    if (kMulti) {
      sm.res[0] = 0;             // first entries
      sm.res[1] = 0;             // a bad or repeated seed or target
      sm.wmin[0] = kNone;        // their least label
    } else {
      enter(nf0, t0);
    }
  }
  if constexpr (kMulti) {
    // CTA 0 marks the targets, then puts every seed in the first frontier
    // with its label seed cost + penalty
    __syncthreads();
    const bool mine = blockIdx.x == 0 && sm.ok;
    const bool in_ticks = sm.res[2] <= kMaxRow;
    if (mine) {
      for (int i = tid; i < job.n_targets; i += kThreads) {
        const int32_t t = job.targets[i];
        const double tc = job.target_cost[i];
        if (t < 0 || t >= N || tc != tc) {
          sm.res[1] = 1;
          continue;
        }
        const unsigned long long was = atomicExch(reinterpret_cast<unsigned long long*>(&w.mtgt[t]),
                                                  (unsigned long long)__double_as_longlong(tc));
        if (was != kNoTerm) sm.res[1] = 1;
        w.rec[t].sp = kTgt;
      }
    }
    __syncthreads();
    if (mine) {
      for (int i = tid; i < job.n_seeds; i += kThreads) {
        const int32_t s0 = job.seeds[i];
        const double sc = job.seed_cost[i];
        if (s0 < 0 || s0 >= N || !(sc >= 0.0)) {
          sm.res[1] = 1;
          continue;
        }
        const unsigned long long was = atomicExch(reinterpret_cast<unsigned long long*>(&w.mseed[s0]),
                                                  (unsigned long long)__double_as_longlong(sc));
        if (was != kNoTerm) {
          sm.res[1] = 1;
          continue;
        }
        const float pen = __ldcg(&w.rec[s0].pen);
        w.claim[s0] = pr.sid;
        const int32_t f0 = indptr[s0], flags = kSeed | (__ldcg(&w.rec[s0].sp) & kTgt);
        w.rec[s0].sp = 1 | flags;
        w.ov[0][atomicAdd(&sm.res[0], 1)] = make_int4(s0, f0, (indptr[s0 + 1] - f0) | flags, __float_as_int(pen));
        unsigned long long lb = ogr_dbits(sc + (double)pen);
        if (in_ticks) {
          lb = 0ull;
          if (seed_ticks(sc, &lb) && tick_finite(pen)) lb += ticks(pen);
        }
        atomicMin(&sm.wmin[0], lb);
      }
    }
    __syncthreads();
    if (tid == 0) {
      if (leader) ctl->merr = sm.res[1];
      enter(leader && !sm.res[1] ? sm.res[0] : 0, leader ? sm.wmin[0] : kNone);
      if (sm.ok && __ldcg(&ctl->merr)) sm.ok = 2;
    }
  }
  __syncthreads();
  const int ok = sm.ok, max_deg = sm.res[2];
  __syncthreads();
  int k0 = 2;                  // barriers used so far
  if (max_deg > kMaxRow) fix = false;
  if (ok != 1) {
    o.status = ok == 0 ? OGR_ERR_TIMEOUT : OGR_ERR_ARG;
  } else {
    // (as a loop of two turns: with the second one plainly behind the first the
    // search in ticks is 1 to 2 % slower, by how the compiler places it)
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (attempt == 0) {
        o = run_search<L, K, kMulti, false>(pr, smem_raw, 1, max_deg, fix);
        k0 = 1 + o.phases;
        if (o.status != kStInexact) break;
      } else {
        const Problem p = pr;
        Outcome io = o;
        int k = k0;
        go_over<kMulti, false>(&p, smem_raw, &k, gtid, gthreads, &io);
        o = io;
        k0 = k;
        fix = false;
      }
    }
  }
  unsigned long long t_done = 0;
  if (leader) t_done = gtimer();
  int status = o.status;
  bool found = o.found && status == OGR_OK;
  // Multi-source: the settled target with the least (label + target cost,
  // label, id) -- the first strict improvement in the heap's pop order.
  int32_t tgt = dst;
  if (kMulti && found && blockIdx.x == 0 && tid < 32) {
    const double dinf = __longlong_as_double(0x7ff0000000000000ll);
    unsigned long long k1 = kNone, k2 = kNone, k3 = kNone;
    for (int pass = 0; pass < 3; ++pass) {
      unsigned long long k = kNone;
      for (int i = tid; i < job.n_targets; i += 32) {
        const int32_t r = job.targets[i];
        const Rec x = ld_rec(&w.rec[r]);
        if ((x.sp & kSpMask) < 2) continue;
        const double lr = fix ? label_value<true>(x.lab) : label_value<false>(x.lab);
        const double tot = lr + job.target_cost[i];
        if (!(tot < dinf)) continue;
        const unsigned long long kt = ogr_order_bits(tot), kl = ogr_order_bits(lr);
        const unsigned long long y = pass == 0 ? kt : pass == 1 ? (kt == k1 ? kl : kNone)
                                                               : (kt == k1 && kl == k2 ? (unsigned long long)r : kNone);
        k = y < k ? y : k;
      }
      k = warp_min_u64(k);
      if (pass == 0) k1 = k;
      if (pass == 1) k2 = k;
      if (pass == 2) k3 = k;
    }
    tgt = k1 == kNone ? -1 : (int32_t)k3;
  }
  // A search that cannot reach dst pops every node it reaches and scans each
  // one's row.  (A multi-source search that reaches no target counts nothing,
  // so its statistics wait for the choice of CTA 0.)
  if ((found || o.exhausted) && pr.want_stats && status >= 0) {
    bool count = true;
    if (kMulti) {
      // whether any target settled, as CTA 0 decides it
      int any = 0;
      for (int i = tid; i < job.n_targets; i += kThreads) {
        const Rec x = ld_rec(&w.rec[job.targets[i]]);
        const double lr = fix ? label_value<true>(x.lab) : label_value<false>(x.lab);
        any |= (x.sp & kSpMask) >= 2 && lr + job.target_cost[i] < __longlong_as_double(0x7ff0000000000000ll);
      }
      count = __syncthreads_or(any) != 0;
    }
    if (count) {
      count_work<kMulti, false>(pr, o, gtid, gthreads, job.stats);
      if (leader) {
        if (found && !kMulti) atomicAdd(&job.stats[1], 1ull);   // dst's own pop
        atomicAdd(&job.stats[2], (unsigned long long)N);
        atomicAdd(&job.stats[3], (unsigned long long)o.phases);
      }
    }
  }
  if (tid == 0) atomicAdd(&g_full_prof[5], o.examined);
  if (kMulti) {
    // once every CTA is past its reads of the marks, CTA 0 restores them for
    // the next search
    if (tid == 0) {
      sm.ok = 1;
      arrive(pr, sm, k0, kArrive, kNone);
    }
  }
  if (blockIdx.x != 0) return;
  // backtrace dst -> src in one walk (reversed into path_out), then CTA 0
  // turns it around
  if (tid < 32) {
    int len = 0;
    if (kMulti && found && tgt < 0) {
      status = OGR_NO_PATH;
      found = false;
    }
    if (found) {
      const int limit = min(path_cap, N);
      int32_t c = -1;
      len = walk_parents(w.par, tgt, N, limit, path_out, &c);
      if (c != -1) status = len >= N ? OGR_ERR_ITER_CAP : OGR_ERR_CAPACITY;
      else if (len < 2) status = OGR_NO_PATH;
    }
    if (*(const volatile int32_t*)&ctl->team.err) status = OGR_ERR_TIMEOUT;
    if (tid == 0) {
      sm.res[0] = status;
      sm.res[1] = (found && status == OGR_OK) ? len : 0;
    }
  }
  __syncthreads();
  status = sm.res[0];
  const int len = sm.res[1];
  for (int i = tid; i < len / 2; i += kThreads) {
    const int32_t t = path_out[i];
    path_out[i] = path_out[len - 1 - i];
    path_out[len - 1 - i] = t;
  }
  if (kMulti) {
    if (tid == 0) await(pr, sm, k0);
    __syncthreads();
    const double none = __longlong_as_double((long long)kNoTerm);
    for (int64_t i = tid; i < job.n_seeds; i += kThreads) {
      const int32_t x = job.seeds[i];
      if (x >= 0 && x < N) w.mseed[x] = none;
    }
    for (int64_t i = tid; i < job.n_targets; i += kThreads) {
      const int32_t x = job.targets[i];
      if (x >= 0 && x < N) w.mtgt[x] = none;
    }
  }
  if (tid != 0) return;
  ctl->res[0] = status;
  ctl->res[1] = len;
  ctl->res[2] = o.phases;
  ctl->sid = fix || max_deg > kMaxRow ? sid : sid + 1;      // (one that went over to doubles took two)
  const unsigned long long t_end = gtimer();
  const unsigned long long clocks = (unsigned long long)(o.clocks > 0 ? o.clocks : 1);
  const unsigned long long wait = (unsigned long long)((double)(t_done - t_loop) * ((double)o.wait / (double)clocks));
  atomicAdd(&g_full_prof[0], 1ull);
  atomicAdd(&g_full_prof[1], (unsigned long long)o.phases);
  atomicAdd(&g_full_prof[2], t_end - t_start);
  atomicAdd(&g_full_prof[3], t_init - t_start);
  atomicAdd(&g_full_prof[4], t_done - t_loop - wait);
  atomicAdd(&g_full_prof[6], wait);
  atomicAdd(&g_full_prof[7], t_end - t_done);
}

__global__ void fill_u64_kernel(unsigned long long* p, int64_t n, unsigned long long v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

constexpr int kMaxDevices = 64;
thread_local int g_grid_blocks[kMaxDevices] = {};   // grid of the cooperative launch (0: not sized yet)
std::atomic<int> g_grid_limit[kMaxDevices] = {};    // SMs x resident CTAs per SM (a device property)

// Variants by the arcs of a row that an entry's lanes hold.
const void* kernel_for(int row, bool multi) {
  if (multi)
    return row == 4    ? (const void*)full_sssp_kernel<2, 2, true>
           : row == 8  ? (const void*)full_sssp_kernel<8, 1, true>
           : row == 16 ? (const void*)full_sssp_kernel<8, 2, true>
                       : (const void*)full_sssp_kernel<16, 2, true>;
  return row == 4    ? (const void*)full_sssp_kernel<2, 2, false>
         : row == 8  ? (const void*)full_sssp_kernel<8, 1, false>
         : row == 16 ? (const void*)full_sssp_kernel<8, 2, false>
                     : (const void*)full_sssp_kernel<16, 2, false>;
}

int size_grid(int dev) {
  if (g_grid_limit[dev] == 0) {
    int sms = 0, coop = 0;
    OGR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    OGR_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return OGR_ERR_CUDA;
    for (int k = 0; k < 8; ++k) {
      const void* f = kernel_for(4 << (k >> 1), (k & 1) != 0);
      int per_sm = 0;
      OGR_CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
      OGR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kThreads, kSmemBytes));
      if (per_sm < 1) return OGR_ERR_CUDA;
    }
    g_grid_limit[dev] = sms;   // one CTA per SM: its shared memory holds the frontier's rows
  }
  if (g_grid_blocks[dev] == 0) g_grid_blocks[dev] = g_grid_limit[dev];
  return OGR_OK;
}

}  // namespace

namespace ogr_full {

// The least form that holds the lattice's longest row, where the caller tells
// it.  Else by the average over the inner layers, which is below the longest
// row: a search that meets a longer one takes the 32-arc form out of line, 16
// entries at a time instead of 64 (two whole-lattice searches each, told
// against not told: 600x400x10 with spans up to 4, average 7.5 and longest 10,
// 7.50 ms against 9.65; 600x400x8 with spans up to 3 and wrong-way arcs, 7.7
// and 10, 6.74 against 8.62; 600x400x12 with sites on a checkerboard, 6.8 and
// 12, 6.88 against 8.06).
int row_for(const ogr_graph& g) {
  if (g.max_row > 0) return g.max_row <= 4 ? 4 : g.max_row <= 8 ? 8 : g.max_row <= 16 ? 16 : 32;
  const double n = (double)(g.num_nodes > 0 ? g.num_nodes : 1), z = (double)(g.nz > 1 ? g.nz : 2);
  const double inner = (double)g.num_edges / n * z / (z - 1.0);
  return inner <= 3.95 ? 4 : inner <= 7.75 ? 8 : inner <= 16.0 ? 16 : 32;
}

int grid_blocks() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  return size_grid(dev) == OGR_OK ? g_grid_blocks[dev] : 0;
}

unsigned wait_limit() { return g_dbg_spin; }
int phase_limit() { return g_dbg_phases; }

size_t workspace_bytes(int32_t num_nodes, int64_t num_edges) {
  return fws_layout(num_nodes, num_edges, nullptr, nullptr);
}

int32_t* result_words(void* ws, int32_t num_nodes, int64_t num_edges) {
  FWs w;
  fws_layout(num_nodes, num_edges, (char*)ws, &w);
  return w.ctl->res;
}

int launch(const ogr_graph& g, const ogr_state& st, const Job& job, void* ws, cudaStream_t s) {
  int dev = 0;
  OGR_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return OGR_ERR_ARG;
  const int rc = size_grid(dev);
  if (rc != OGR_OK) return rc;
  FWs w;
  fws_layout(g.num_nodes, g.num_edges, (char*)ws, &w);
  w.bar_spin = g_dbg_spin;
  w.max_phases = g_dbg_phases;
  ogr_full::Job jv = job;
  jv.gated = 0;
  if (ogr_tile::enabled() && !job.multi) {
    const int trc = ogr_tile::launch(g, st, job, w.tile, w.ctl->res, &w.ctl->tile_gate, s);
    if (trc == OGR_OK)
      jv.gated = 1;              // the phase engine runs only if the net was handed over
    else if (trc != OGR_ERR_CAPACITY)
      return trc;                // (capacity: this lattice does not tile; phase engine alone)
  }
  // the team's barrier words and surplus counts start at zero on every launch
  OGR_CUDA_TRY(cudaMemsetAsync(&w.ctl->team, 0, sizeof(Ctl), s));
  ogr_graph gv = g;
  ogr_state sv = st;
  void* args[] = {&gv, &sv, &jv, &w};
  const void* fn = kernel_for(ogr_full::row_for(g), job.multi != 0);
  OGR_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(g_grid_blocks[dev]), dim3(kThreads), args, kSmemBytes, s));
  return OGR_OK;
}

}  // namespace ogr_full

extern "C" int ogr_debug_limits(int32_t barrier_spin, int32_t max_phases, int32_t* cur_spin,
                                int32_t* cur_phases) {
  if (barrier_spin < -1 || max_phases < -1) return OGR_ERR_ARG;
  if (barrier_spin >= 0) g_dbg_spin = barrier_spin == 0 ? kBarSpin : (unsigned)barrier_spin - 1u;
  if (max_phases >= 0) g_dbg_phases = max_phases;
  if (cur_spin) *cur_spin = (int32_t)(g_dbg_spin == kBarSpin ? 0 : g_dbg_spin + 1u);
  if (cur_phases) *cur_phases = g_dbg_phases;
  return OGR_OK;
}

extern "C" int ogr_full_lanes(int32_t lanes, int32_t* current) {
  if (lanes != 0 && lanes != 4 && lanes != 8 && lanes != 16) return OGR_ERR_ARG;
  if (lanes != 0) g_full_lanes = lanes;
  if (current) *current = g_full_lanes;
  return OGR_OK;
}

extern "C" int ogr_full_reuse(int32_t mode, int32_t* current) {
  if (mode < -1 || mode > 1) return OGR_ERR_ARG;
  if (mode >= 0) g_full_reuse = mode;
  if (current) *current = g_full_reuse;
  return OGR_OK;
}

extern "C" int ogr_full_grid(int32_t ctas, int32_t* current, int32_t* limit) {
  int dev = 0;
  OGR_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return OGR_ERR_ARG;
  const int rc = size_grid(dev);
  if (rc != OGR_OK) return rc;
  // up to two CTAs per SM may be asked for (a stored setting of an engine that
  // ran two); one per SM is what runs
  const int lim = g_grid_limit[dev];
  if (ctas < 0 || ctas > 2 * lim) return OGR_ERR_ARG;
  if (ctas > 0) g_grid_blocks[dev] = ctas < lim ? ctas : lim;
  if (current) *current = g_grid_blocks[dev];
  if (limit) *limit = g_grid_limit[dev];
  return OGR_OK;
}

extern "C" size_t ogr_full_workspace_bytes(int32_t num_nodes, int64_t num_edges) {
  return ogr_full::workspace_bytes(num_nodes, num_edges);
}

extern "C" int ogr_full_workspace_init(void* ws, size_t bytes, int32_t num_nodes, int64_t num_edges,
                                       void* stream) {
  if (!ws || num_nodes < 1 || num_edges < 0) return OGR_ERR_ARG;
  if (bytes < ogr_full::workspace_bytes(num_nodes, num_edges)) return OGR_ERR_CAPACITY;
  FWs w;
  fws_layout(num_nodes, num_edges, (char*)ws, &w);
  // no node is claimed by search 1, 2, ...; tile stamp 0: the first tile
  // search clears its node words
  cudaStream_t s = ogr_stream(stream);
  OGR_CUDA_TRY(cudaMemsetAsync(w.ctl, 0, sizeof(FCtl), s));
  OGR_CUDA_TRY(cudaMemsetAsync(w.claim, 0, sizeof(int32_t) * (size_t)num_nodes, s));
  OGR_CUDA_TRY(cudaMemsetAsync(w.tile, 0, ogr_tile::ctl_bytes(), s));
  // no node is a multi-source seed or target until a search marks it
  const int blocks = (int)std::min<int64_t>((num_nodes + 255) / 256, 152 * 8);
  fill_u64_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<unsigned long long*>(w.mseed), num_nodes, kNoTerm);
  OGR_LAUNCH_CHECK();
  fill_u64_kernel<<<blocks, 256, 0, s>>>(reinterpret_cast<unsigned long long*>(w.mtgt), num_nodes, kNoTerm);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}

extern "C" int ogr_full_profile(int64_t* out8, int32_t reset) {
  if (!out8) return OGR_ERR_ARG;
  OGR_CUDA_TRY(cudaMemcpyFromSymbol(out8, g_full_prof, sizeof(unsigned long long) * 8));
  if (reset) {
    unsigned long long z[8] = {};
    OGR_CUDA_TRY(cudaMemcpyToSymbol(g_full_prof, z, sizeof(z)));
  }
  return OGR_OK;
}

extern "C" int ogr_find_path_full(const ogr_graph* g, const ogr_state* st, const ogr_net_args* net, void* ws,
                                  size_t bytes, int32_t* path_out, int32_t path_cap, int32_t* path_len_out,
                                  int64_t* stats, void* stream) {
  if (!g || !st || !net || !ws || !path_out || !path_len_out || path_cap < 2) return OGR_ERR_ARG;
  if (bytes < ogr_full::workspace_bytes(g->num_nodes, g->num_edges)) return OGR_ERR_CAPACITY;
  if (net->src < 0 || net->dst < 0 || net->src >= g->num_nodes || net->dst >= g->num_nodes) return OGR_ERR_ARG;
  ogr_full::Job job{};
  job.a = *net;
  job.path_out = path_out;
  job.path_cap = path_cap;
  job.from_pass = 0;
  job.stats = reinterpret_cast<unsigned long long*>(stats);
  cudaStream_t s = ogr_stream(stream);
  const int rc = ogr_full::launch(*g, *st, job, ws, s);
  if (rc != OGR_OK) return rc;
  int32_t res[4];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, ogr_full::result_words(ws, g->num_nodes, g->num_edges), sizeof(res),
                               cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = res[0] == OGR_OK ? res[1] : 0;
  return res[0];
}

extern "C" int ogr_find_path_full_multi(const ogr_graph* g, const ogr_state* st, const ogr_net_args* net,
                                        const int32_t* seeds, const double* seed_cost, int32_t n_seeds,
                                        const int32_t* targets, const double* target_cost, int32_t n_targets,
                                        void* ws, size_t bytes, int32_t* path_out, int32_t path_cap,
                                        int32_t* path_len_out, int64_t* stats, void* stream) {
  if (!g || !st || !net || !ws || !path_out || !path_len_out || path_cap < 2) return OGR_ERR_ARG;
  if (n_seeds < 0 || n_targets < 0 || (n_seeds > 0 && (!seeds || !seed_cost)) ||
      (n_targets > 0 && (!targets || !target_cost)))
    return OGR_ERR_ARG;
  if (bytes < ogr_full::workspace_bytes(g->num_nodes, g->num_edges)) return OGR_ERR_CAPACITY;
  *path_len_out = 0;
  if (n_seeds == 0 || n_targets == 0) return OGR_NO_PATH;
  ogr_full::Job job{};
  job.a = *net;
  job.path_out = path_out;
  job.path_cap = path_cap;
  job.stats = reinterpret_cast<unsigned long long*>(stats);
  job.multi = 1;
  job.seeds = seeds;
  job.seed_cost = seed_cost;
  job.n_seeds = n_seeds;
  job.targets = targets;
  job.target_cost = target_cost;
  job.n_targets = n_targets;
  cudaStream_t s = ogr_stream(stream);
  const int rc = ogr_full::launch(*g, *st, job, ws, s);
  if (rc != OGR_OK) return rc;
  int32_t res[4];
  OGR_CUDA_TRY(cudaMemcpyAsync(res, ogr_full::result_words(ws, g->num_nodes, g->num_edges), sizeof(res),
                               cudaMemcpyDeviceToHost, s));
  OGR_CUDA_TRY(cudaStreamSynchronize(s));
  *path_len_out = res[0] == OGR_OK ? res[1] : 0;
  return res[0];
}
