// Near-wall cells of a voxel grid and their link tables, built on the device, and the
// memory of grids and voxelizations.
//
// The table holds, for each near-wall cell and direction, how the reference's pull obtains
// the value (lbmCpuReference.ts:189-224), resolved once per voxel grid.  It used to be built
// on the host from copies of the class bytes, the boundary map and q: two copies of 21 MB
// and three passes over the lattice, about 5 ms of a 256x128x128 set-up.  Three kernels over
// the class bytes and the list take 16 us, and the scan of the rows 8: they are bound by the latency of a few
// dependent loads per cell, not by bandwidth.
#include <algorithm>

#include "common.cuh"
#include "engine_internal.h"
#include "lbm_kernels.cuh"

namespace aerosim {

namespace {

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// Whether kept memory serves a need: large enough, and not much larger.
bool fits(size_t cap, size_t need) { return cap >= need && cap - need <= kKeepSlack + need / 8; }

// Near-wall cells per x-row, one warp per row.
__global__ void near_count_kernel(const uint8_t* __restrict__ cls, const Layout L, long long rows, uint32_t* __restrict__ counts) {
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const uint8_t* const c = cls + row * L.pitch;
  int n = 0;
  for (int x0 = 0; x0 < L.nx; x0 += 32) {
    const int x = x0 + lane;
    n += __popc(__ballot_sync(0xffffffffu, x >= 1 && x < L.nx - 1 && (c[x] & CLS_NEAR)));
  }
  if (lane == 0) counts[row] = (uint32_t)n;
}

// Their cell indices in ascending order, from the rows' first positions.
__global__ void near_list_kernel(const uint8_t* __restrict__ cls, const Layout L, long long rows,
                                 const uint32_t* __restrict__ first, int32_t* __restrict__ cells) {
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const uint8_t* const c = cls + row * L.pitch;
  uint32_t at = first[row];
  for (int x0 = 0; x0 < L.nx; x0 += 32) {
    const int x = x0 + lane;
    const bool near = x >= 1 && x < L.nx - 1 && (c[x] & CLS_NEAR);
    const unsigned m = __ballot_sync(0xffffffffu, near);
    if (near) cells[at + __popc(m & ((1u << lane) - 1u))] = (int32_t)(row * L.nx + x);
    at += (uint32_t)__popc(m);
  }
}

// One link: cell t of the list, direction d = blockIdx.y.
__global__ void near_links_kernel(const uint8_t* __restrict__ cls, const int32_t* __restrict__ bmap,
                                  const float* __restrict__ q, const Layout L, const int32_t* __restrict__ cells,
                                  long long n, NearLink* __restrict__ links, NearLinkF* __restrict__ links_f) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int d = blockIdx.y;
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  const int cell = cells[t];
  const int row = cell / nx, ix = cell - row * nx;
  const int iz = row / ny, iy = row - iz * ny;
  // the direction's vector and opposite by arithmetic on a run-time d
  int cx = 0, cy = 0, cz = 0, wd = 0;
#pragma unroll
  for (int e = 1; e < 19; ++e)
    if (e == d) {
      cx = cx_of(e); cy = cy_of(e); cz = cz_of(e); wd = opp_of(e);
    }
  auto flag_at = [&](int x, int y, int z) { return cls[((long long)y + (long long)ny * z) * L.pitch + x] & CLS_FLAG_MASK; };
  auto off = [&](int dir, int x, int y, int z) -> uint32_t {
    int sl = 0;
#pragma unroll
    for (int e = 0; e < 19; ++e)
      if (e == dir) sl = slot_of(e);
    return (uint32_t)(((long long)y + (long long)ny * z) * L.rstride + (long long)sl * L.dstride + x);
  };
  NearLink k;
  k.A = 1.0;
  k.B = 0.0;
  const int sx = clampi(ix - cx, 0, nx - 1), sy = clampi(iy - cy, 0, ny - 1), sz = clampi(iz - cz, 0, nz - 1);
  if (d > 0 && flag_at(sx, sy, sz) == CELL_SOLID) {
    // Bouzidi in the pull, lbmCpuReference.ts:196-221
    const int bi = flag_at(ix, iy, iz) == CELL_BOUNDARY ? bmap[cell] : -1;
    const double qv = bi >= 0 ? (double)q[(long long)bi * 18 + (wd - 1)] : 0.5;
    const double qe = qv > 0.0 ? qv : 0.5;
    const int fx = clampi(ix + cx, 0, nx - 1), fy = clampi(iy + cy, 0, ny - 1), fz = clampi(iz + cz, 0, nz - 1);
    k.o1 = off(wd, ix, iy, iz); k.d1 = (uint32_t)wd;
    k.o2 = k.o1; k.d2 = (uint32_t)wd;
    if (flag_at(fx, fy, fz) != CELL_SOLID) {
      if (qe < 0.5) {
        k.A = 2.0 * qe; k.B = 1.0 - 2.0 * qe;
        k.o2 = off(wd, fx, fy, fz); k.d2 = (uint32_t)wd;
      } else {
        const double inv2q = 1.0 / (2.0 * qe);
        k.A = inv2q; k.B = 1.0 - inv2q;
        k.o2 = off(d, ix, iy, iz); k.d2 = (uint32_t)d;
      }
    }
  } else {
    k.o1 = off(d, sx, sy, sz); k.d1 = (uint32_t)d;
    k.o2 = k.o1; k.d2 = (uint32_t)d;
  }
  const long long i = (long long)d * n + t;
  links[i] = k;
  links_f[i] = NearLinkF{k.o1, k.o2, (float)k.A, (float)k.B};
}

// Exclusive scan in one CTA, tiles of 4096 counts (4 consecutive ones a thread).
__global__ void __launch_bounds__(1024) scan_rows_kernel(uint32_t* __restrict__ counts, long long n, unsigned long long* total) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (long long base = 0; base < n; base += 4096) {
    const long long i = base + threadIdx.x * 4;
    uint32_t v[4], sum = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = i + k < n ? counts[i + k] : 0u;
      sum += v[k];
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t a = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += a;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane];
      const uint32_t own = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += a;
      }
      s_warp[lane] = w - own;
      if (lane == 31) s_tile = w;
    }
    __syncthreads();
    uint32_t run = carry + s_warp[warp] + inc - sum;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < n) counts[i + k] = run;
      run += v[k];
    }
    carry += s_tile;
    __syncthreads();  // s_warp and s_tile are free for the next tile
  }
  if (threadIdx.x == 0) *total = carry;
}

}  // namespace

cudaError_t launch_scan_rows(uint32_t* counts, long long n, unsigned long long* total, cudaStream_t s) {
  scan_rows_kernel<<<1, 1024, 0, s>>>(counts, n, total);
  return cudaGetLastError();
}

cudaError_t build_near_table(const DevGrid& g, const Layout& L, VoxScratch* w, cudaStream_t s, NearTable* t) {
  const long long rows = (long long)g.ny * g.nz;
  cudaError_t e = w->pinned();
  if (e == cudaSuccess) e = w->device(up256((size_t)rows * 4));
  if (e != cudaSuccess) return e;
  uint32_t* const counts = static_cast<uint32_t*>(w->dev);
  const unsigned grid = (unsigned)((rows * 32 + 255) / 256);
  near_count_kernel<<<grid, 256, 0, s>>>(g.cls, L, rows, counts);
  e = launch_scan_rows(counts, rows, w->host, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  const long long n = (long long)w->host[0];
  const size_t cells = up256((size_t)std::max<long long>(n, 1) * 4),
               links = up256((size_t)std::max<long long>(n, 1) * 19 * sizeof(NearLink)),
               links_f = up256((size_t)std::max<long long>(n, 1) * 19 * sizeof(NearLinkF));
  const size_t need = cells + links + links_f;
  if (!fits(t->cap, need)) {
    near_free(t);
    const size_t room = need + need / 8;  // a turned body has a few more cells
    e = cudaMalloc(&t->mem, room);
    if (e != cudaSuccess) {
      t->mem = nullptr;
      return e;
    }
    t->cap = room;
  }
  char* c = static_cast<char*>(t->mem);
  t->cells = reinterpret_cast<int32_t*>(c);
  t->links = reinterpret_cast<NearLink*>(c + cells);
  t->links_f = reinterpret_cast<NearLinkF*>(c + cells + links);
  t->n = n;
  if (n > 0) {
    near_list_kernel<<<grid, 256, 0, s>>>(g.cls, L, rows, counts, t->cells);
    near_links_kernel<<<dim3((unsigned)((n + 127) / 128), 19), 128, 0, s>>>(g.cls, g.bmap, g.q, L, t->cells, n, t->links,
                                                                          t->links_f);
  }
  return cudaGetLastError();
}

void near_free(NearTable* t) {
  cudaFree(t->mem);
  *t = NearTable();
}

cudaError_t grid_cells(DevGrid* g, long long N, size_t cls_bytes) {
  const size_t bf = up256((size_t)N), bc = up256(std::max<size_t>(cls_bytes, 1)), bm = up256((size_t)N * 4);
  if (!fits(g->cell_cap, bf + bc + bm)) {
    cudaFree(g->cell_mem);
    g->cell_mem = nullptr;
    g->cell_cap = 0;
    const cudaError_t e = cudaMalloc(&g->cell_mem, bf + bc + bm);
    if (e != cudaSuccess) {
      g->cell_mem = nullptr;
      return e;
    }
    g->cell_cap = bf + bc + bm;
  }
  char* c = static_cast<char*>(g->cell_mem);
  g->flags = reinterpret_cast<uint8_t*>(c);
  g->cls = reinterpret_cast<uint8_t*>(c + bf);
  g->bmap = reinterpret_cast<int32_t*>(c + bf + bc);
  return cudaSuccess;
}

cudaError_t grid_lists(DevGrid* g, long long B) {
  const size_t n = (size_t)std::max<long long>(B, 1);
  const size_t bc = up256(n * 4), bq = up256(n * 18 * 4), bm = up256(n * 4);
  if (!fits(g->list_cap, bc + bq + bm)) {
    cudaFree(g->list_mem);
    g->list_mem = nullptr;
    g->list_cap = 0;
    const size_t room = bc + bq + bm + (bc + bq + bm) / 8;
    const cudaError_t e = cudaMalloc(&g->list_mem, room);
    if (e != cudaSuccess) {
      g->list_mem = nullptr;
      return e;
    }
    g->list_cap = room;
  }
  char* c = static_cast<char*>(g->list_mem);
  g->bcells = reinterpret_cast<int32_t*>(c);
  g->q = reinterpret_cast<float*>(c + bc);
  g->minq = reinterpret_cast<float*>(c + bc + bq);
  return cudaSuccess;
}

void grid_free(DevGrid* g) {
  cudaFree(g->cell_mem);
  cudaFree(g->list_mem);
  *g = DevGrid();
}

cudaError_t VoxScratch::device(size_t n) {
  if (bytes >= n) return cudaSuccess;
  cudaFree(dev);
  dev = nullptr;
  bytes = 0;
  const cudaError_t e = cudaMalloc(&dev, n);
  if (e != cudaSuccess) {
    dev = nullptr;
    return e;
  }
  bytes = n;
  return cudaSuccess;
}
cudaError_t VoxScratch::pinned() {
  if (host) return cudaSuccess;
  return cudaHostAlloc((void**)&host, 32 * sizeof(unsigned long long), cudaHostAllocMapped);
}
void VoxScratch::release() {
  cudaFree(dev);
  dev = nullptr;
  bytes = 0;
}
void VoxScratch::trim() {
  if (bytes > kKeepSlack) release();
}

}  // namespace aerosim
