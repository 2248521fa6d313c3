// A1: 3-D Manhattan lattice → CSR, built on the device in closed form.
//
// Row layout of node (x, y, z), sorted by destination id as the reference's
// structured sort leaves it (unified_pathfinder.py:935):
//   [via partners z' < z, ascending] [y-1] [x-1] [x+1] [y+1] [via partners z' > z]
// Lateral arcs exist only on lateral layers and only along the layer's axis
// (plus the other axis when wrong-way arcs are enabled).  A via partner is
// present when (x, y) is a legal site of that layer pair.
#include <string.h>

#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kMaxLayers = 64;
constexpr int kMaxPartners = 64 * 64;

struct LatticeConst {
  int nx, ny, nz;
  float lateral_cost, wrong_way_cost;
  unsigned char axis[kMaxLayers];
  int pptr[kMaxLayers + 1];
};

// The lattice description travels as a kernel argument and its via-partner
// tables live in the build workspace, so builds on different streams (jobs
// of a server) do not share state.
struct LatDev {
  LatticeConst h;
  const int* pz;
  const float* pcost;
  const int* psite;
  bool plain;          // every list ascends, each layer once, without its own
};

__device__ __forceinline__ bool site_ok(int mode, int x, int y) {
  if (mode == 0) return true;
  if (mode == 1) return ((x + y) & 1) == 0;
  return (x % mode) == 0 && (y % mode) == 0;
}

// Whether layer z has arcs along x / along y, and their costs.
struct Axes {
  bool h, v;
  float ch, cv;
  __device__ Axes(const LatticeConst& l, int z) {
    const int ax = l.axis[z];
    const bool ww = ax != 0 && l.wrong_way_cost > 0.f;
    h = ax == 1 || ww;
    v = ax == 2 || ww;
    ch = ax == 1 ? l.lateral_cost : l.wrong_way_cost;
    cv = ax == 2 ? l.lateral_cost : l.wrong_way_cost;
  }
};

// Lateral arcs of (x, y) on a layer with axes ax: all of them, or those that
// come before the one to side (0: y-1, 1: x-1, 2: x+1, 3: y+1).
__device__ __forceinline__ int laterals_before(const LatDev& L, const Axes& ax, int x, int y, int side) {
  int k = 0;
  if (side > 0 && ax.v && y > 0) ++k;
  if (side > 1 && ax.h && x > 0) ++k;
  if (side > 2 && ax.h && x + 1 < L.h.nx) ++k;
  if (side > 3 && ax.v && y + 1 < L.h.ny) ++k;
  return k;
}

// The row of (x, y, z): the via partners listed before the first that is not
// below z, the laterals, the partners above z.  (A list that does not ascend,
// repeats a layer or names z itself is read by the same rule everywhere; of a
// plain one the rule asks for less: 222 us a build of 600x400x12 against 245.)
__device__ __forceinline__ int partners_below(const LatDev& L, int x, int y, int z) {
  int k = 0;
  for (int p = L.h.pptr[z]; p < L.h.pptr[z + 1] && L.pz[p] < z; ++p) k += site_ok(L.psite[p], x, y) ? 1 : 0;
  return k;
}

__device__ __forceinline__ int degree(const LatDev& L, int x, int y, int z) {
  int k = laterals_before(L, Axes(L.h, z), x, y, 4);
  bool below = true;
  for (int p = L.h.pptr[z]; p < L.h.pptr[z + 1]; ++p) {
    const int zz = L.pz[p];
    below = below && zz < z;
    if (L.plain || below || zz > z) k += site_ok(L.psite[p], x, y) ? 1 : 0;
  }
  return k;
}

// Place in the row of (x, y, z) of its first arc to layer `want`; -1: none.
__device__ __forceinline__ int partner_place(const LatDev& L, int x, int y, int z, int want) {
  int k = want > z ? laterals_before(L, Axes(L.h, z), x, y, 4) : 0;
  bool below = true;
  for (int p = L.h.pptr[z]; p < L.h.pptr[z + 1]; ++p) {
    const int zz = L.pz[p];
    const bool ok = site_ok(L.psite[p], x, y);
    if (L.plain) {
      if (zz >= want) return ok && zz == want ? k : -1;
      k += ok ? 1 : 0;
      continue;
    }
    below = below && zz < z;
    if ((below || zz > z) && ok) {
      if (zz == want) return k;
      ++k;
    }
  }
  return -1;
}

// Row starts: degrees and their sums within tiles of kScanTile nodes, the sum
// of the tiles before each (one block), and the sum of both.
constexpr int kScanTile = 4096;
constexpr int kScanThreads = 1024;
constexpr int kScanPer = kScanTile / kScanThreads;

// Exclusive sum over a block of 1024 threads; *total is the block's sum.
__device__ __forceinline__ int block_scan(int v, int* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int t = s_warp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    s_warp[lane] = t;
  }
  __syncthreads();
  *total = s_warp[31];
  const int before = warp > 0 ? s_warp[warp - 1] : 0;
  return before + x - v;
}

__global__ void __launch_bounds__(kScanThreads) scan_tiles(LatDev L, int64_t N, int32_t* out, int32_t* tile_sums) {
  __shared__ int s_warp[32];
  const OgrDiv by_plane((unsigned)(L.h.nx * L.h.ny)), by_nx((unsigned)L.h.nx);
  const int64_t i0 = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanPer;
  int d[kScanPer], sum = 0;
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    d[j] = 0;
    if (i0 + j < N) {
      const unsigned n = (unsigned)(i0 + j), z = by_plane(n), r = n - z * by_plane.d, y = by_nx(r);
      d[j] = degree(L, (int)(r - y * by_nx.d), (int)y, (int)z);
    }
    sum += d[j];
  }
  int total;
  int at = block_scan(sum, s_warp, &total);
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    if (i0 + j < N) out[i0 + j] = at;
    at += d[j];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_tile_sums(int32_t* tile_sums, int64_t ntiles, int32_t* total) {
  __shared__ int s_warp[32];
  int carry = 0;
  for (int64_t base = 0; base < ntiles; base += kScanThreads) {
    const int64_t i = base + threadIdx.x;
    const int v = i < ntiles ? tile_sums[i] : 0;
    int sum;
    const int x = block_scan(v, s_warp, &sum);
    if (i < ntiles) tile_sums[i] = carry + x;
    carry += sum;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void scan_add(int32_t* out, int64_t N, const int32_t* tile_sums, const int32_t* total) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= N;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (i == N) out[N] = *total;
    else out[i] += tile_sums[i / kScanTile];
  }
}

// The rows of a tile of nodes of one layer (blockIdx.y), staged in shared
// memory and copied out in arc order.  A row written by its thread straight to
// memory scattered 18 bytes per arc over six arrays (280 us for 21 M arcs),
// and the reverse arc was found by walking the neighbour's row (132 us): it is
// the neighbour's row start plus a count here, its place in that row.
constexpr int kFillThreads = 128;
__global__ void __launch_bounds__(kFillThreads) fill_kernel(LatDev L, int tile_nodes, const int32_t* __restrict__ indptr, int32_t* indices,
                            float* cost, unsigned char* lay, unsigned char* kind, int32_t* edge_src, int32_t* rev,
                            int cap) {
  extern __shared__ __align__(16) int32_t s_buf[];
  int32_t* s_idx = s_buf;
  float* s_cost = reinterpret_cast<float*>(s_buf + cap);
  int32_t* s_src = s_buf + 2 * cap;
  int32_t* s_rev = s_buf + 3 * cap;
  unsigned char* s_kind = reinterpret_cast<unsigned char*>(s_buf + 4 * cap);
  const int nx = L.h.nx, ny = L.h.ny, z = blockIdx.y;
  const int32_t plane = nx * ny;
  const Axes ax(L.h, z);
  const OgrDiv by_nx((unsigned)nx);
  const int p0 = L.h.pptr[z], p1 = L.h.pptr[z + 1];
  for (int64_t t0 = (int64_t)blockIdx.x * tile_nodes; t0 < plane; t0 += (int64_t)gridDim.x * tile_nodes) {
    const int32_t r0 = (int32_t)t0, r1 = (int32_t)min((int64_t)plane, t0 + tile_nodes);
    const int32_t e0 = indptr[z * plane + r0], e1 = indptr[z * plane + r1];
    for (int32_t i = threadIdx.x; i < r1 - r0; i += kFillThreads) {
      const int32_t r = r0 + i;
      const int y = (int)by_nx((unsigned)r), x = r - y * nx;
      const int32_t n = z * plane + r;
      int k = indptr[n] - e0;
      auto put = [&](int32_t v, float c, int via, int32_t back) {
        s_idx[k] = v;
        s_cost[k] = c;
        s_src[k] = n;
        s_rev[k] = back;
        s_kind[k] = (unsigned char)via;
        ++k;
      };
      auto via = [&](int p, int zz) {
        const int32_t v = zz * plane + r;
        int32_t back = -1;
        if (rev) {
          back = partner_place(L, x, y, zz, z);
          if (back >= 0) back += indptr[v];
        }
        put(v, L.pcost[p], 1, back);
      };
      int p = p0;
      for (; p < p1; ++p) {
        const int zz = L.pz[p];
        if (zz >= z) break;
        if (site_ok(L.psite[p], x, y)) via(p, zz);
      }
      // laterals: the arc back stands on the neighbour's other side
      auto lateral = [&](int dx, int dy, int32_t v, float c, int side) {
        put(v, c, 0, rev ? indptr[v] + partners_below(L, x + dx, y + dy, z) +
                               laterals_before(L, ax, x + dx, y + dy, side)
                         : -1);
      };
      if (ax.v && y > 0) lateral(0, -1, n - nx, ax.cv, 3);
      if (ax.h && x > 0) lateral(-1, 0, n - 1, ax.ch, 2);
      if (ax.h && x + 1 < nx) lateral(1, 0, n + 1, ax.ch, 1);
      if (ax.v && y + 1 < ny) lateral(0, 1, n + nx, ax.cv, 0);
      for (; p < p1; ++p) {
        const int zz = L.pz[p];
        if (zz > z && site_ok(L.psite[p], x, y)) via(p, zz);
      }
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < e1 - e0; i += kFillThreads) {
      indices[e0 + i] = s_idx[i];
      cost[e0 + i] = s_cost[i];
      edge_src[e0 + i] = s_src[i];
      if (rev) rev[e0 + i] = s_rev[i];
      lay[e0 + i] = (unsigned char)z;
      kind[e0 + i] = s_kind[i];
    }
    __syncthreads();
  }
}

// Fills the description; the partner tables are copied on `s` into dev_tab
// (3 * kMaxPartners words of the workspace).
int load_desc(const ogr_lattice_desc* d, int* dev_tab, cudaStream_t s, LatDev* out) {
  if (!d || d->nx < 1 || d->ny < 1 || d->nz < 1 || d->nz > kMaxLayers) return OGR_ERR_ARG;
  LatDev L{};
  LatticeConst& h = L.h;
  h.nx = d->nx; h.ny = d->ny; h.nz = d->nz;
  h.lateral_cost = d->lateral_cost;
  h.wrong_way_cost = d->wrong_way_cost;
  for (int z = 0; z < d->nz; ++z) h.axis[z] = d->layer_axis[z];
  for (int z = 0; z <= d->nz; ++z) h.pptr[z] = d->partner_ptr[z];
  const int np = d->partner_ptr[d->nz];
  if (np > kMaxPartners || np < 0) return OGR_ERR_ARG;
  L.plain = true;
  for (int z = 0; z < d->nz; ++z)
    for (int p = h.pptr[z]; p < h.pptr[z + 1]; ++p)
      L.plain = L.plain && d->partner_z[p] != z && (p == h.pptr[z] || d->partner_z[p] > d->partner_z[p - 1]);
  L.pz = dev_tab;
  L.pcost = nullptr;
  L.psite = nullptr;
  if (np > 0) {
    // one copy of the three tables (the source is pageable, so each copy waits)
    int tab[3 * kMaxPartners];
    memcpy(tab, d->partner_z, np * sizeof(int));
    memcpy(tab + np, d->partner_cost, np * sizeof(float));
    memcpy(tab + 2 * np, d->partner_site, np * sizeof(int));
    L.pcost = reinterpret_cast<const float*>(dev_tab + np);
    L.psite = dev_tab + 2 * np;
    OGR_CUDA_TRY(cudaMemcpyAsync(dev_tab, tab, 3 * np * sizeof(int), cudaMemcpyHostToDevice, s));
  }
  *out = L;
  return OGR_OK;
}

// Host mirror of the per-node arc count (for sizing).
int64_t host_num_edges(const ogr_lattice_desc* d) {
  const int64_t nx = d->nx, ny = d->ny;
  int64_t E = 0;
  for (int z = 0; z < d->nz; ++z) {
    const int ax = d->layer_axis[z];
    const bool ww = d->wrong_way_cost > 0.f;
    if (ax != 0) {
      if (ax == 1 || ww) E += 2 * ny * (nx - 1);
      if (ax == 2 || ww) E += 2 * nx * (ny - 1);
    }
    for (int p = d->partner_ptr[z]; p < d->partner_ptr[z + 1]; ++p) {
      const int mode = d->partner_site[p];
      int64_t sites = 0;
      if (mode == 0) sites = nx * ny;
      else {
        for (int64_t x = 0; x < nx; ++x)
          for (int64_t y = 0; y < ny; ++y)
            if (mode == 1 ? ((x + y) % 2 == 0) : (x % mode == 0 && y % mode == 0)) ++sites;
      }
      E += sites;
    }
  }
  return E;
}

}  // namespace

extern "C" int ogr_csr_num_edges(const ogr_lattice_desc* d, int64_t* num_edges) {
  if (!d || !num_edges || d->nz > kMaxLayers) return OGR_ERR_ARG;
  *num_edges = host_num_edges(d);
  return OGR_OK;
}

extern "C" size_t ogr_csr_workspace_bytes(const ogr_lattice_desc* d) {
  const int64_t N = (int64_t)d->nx * d->ny * d->nz;
  const int64_t tiles = (N + kScanTile - 1) / kScanTile;
  return (size_t)(tiles * 4 + 64) + 3 * sizeof(int) * kMaxPartners + 512;
}

extern "C" int ogr_csr_build(const ogr_lattice_desc* d, int32_t* indptr, int32_t* indices,
                             float* base_costs, uint8_t* edge_layer, uint8_t* edge_kind,
                             int32_t* edge_src, int32_t* rev, void* workspace,
                             size_t workspace_bytes, void* stream) {
  if (!d || d->nz > kMaxLayers || d->nz < 1) return OGR_ERR_ARG;
  const int64_t N = (int64_t)d->nx * d->ny * d->nz;
  if (N >= (int64_t)1 << 31) return OGR_ERR_ARG;
  const int64_t E = host_num_edges(d);
  if (E >= (int64_t)1 << 31) return OGR_ERR_ARG;
  if (workspace_bytes < ogr_csr_workspace_bytes(d) || !workspace) return OGR_ERR_CAPACITY;
  cudaStream_t s = ogr_stream(stream);
  const int64_t tiles = (N + kScanTile - 1) / kScanTile;
  int32_t* tile_sums = reinterpret_cast<int32_t*>(workspace);
  int32_t* total = tile_sums + tiles;
  const size_t tab_off = ((size_t)(tiles * 4 + 64) + 255) & ~(size_t)255;
  LatDev L;
  const int rc = load_desc(d, reinterpret_cast<int*>((char*)workspace + tab_off), s, &L);
  if (rc != OGR_OK) return rc;
  scan_tiles<<<(unsigned)tiles, kScanThreads, 0, s>>>(L, N, indptr, tile_sums);
  OGR_LAUNCH_CHECK();
  scan_tile_sums<<<1, kScanThreads, 0, s>>>(tile_sums, tiles, total);
  OGR_LAUNCH_CHECK();
  scan_add<<<ogr_blocks(N + 1, 256), 256, 0, s>>>(indptr, N, tile_sums, total);
  OGR_LAUNCH_CHECK();
  // A tile's rows have to fit in shared memory: 17 bytes per arc, the layers'
  // longest row times the tile's nodes, at most 48 KB (rows of up to 67 arcs,
  // each layer's partners once: 36,448 bytes at 32 nodes); one row may take more.
  int row = 1;
  for (int z = 0; z < d->nz; ++z) row = std::max(row, d->partner_ptr[z + 1] - d->partner_ptr[z] + 4);
  int tile_nodes = kFillThreads;
  while (tile_nodes > 1 && tile_nodes * row * 17 > 48 * 1024) tile_nodes -= tile_nodes > 32 ? 32 : (tile_nodes + 1) / 2;
  const int cap = tile_nodes * row;
  if (cap * 17 > 48 * 1024)
    OGR_CUDA_TRY(cudaFuncSetAttribute((const void*)fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cap * 17));
  const int64_t plane = (int64_t)d->nx * d->ny;
  const dim3 grid((unsigned)std::min<int64_t>((plane + tile_nodes - 1) / tile_nodes, 65535), (unsigned)d->nz);
  fill_kernel<<<grid, kFillThreads, (size_t)cap * 17, s>>>(L, tile_nodes, indptr, indices, base_costs, edge_layer,
                                                          edge_kind, edge_src, rev, cap);
  OGR_LAUNCH_CHECK();
  return OGR_OK;
}
