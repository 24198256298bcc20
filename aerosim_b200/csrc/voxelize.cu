// GPU voxelizer: voxelizeMeshToLattice (src/geometry/voxelizer.ts:86-281) on sm_100a.
//
// The BVH is the reference's (bvh.ts:34-253: median split of the widest centroid extent,
// leaves of <= 4 triangles), because the node boxes decide which triangles a ray tests; the
// same tree on both sides makes the flags and link lists bit-exact.  Everything runs on the
// device in FP64 with no contraction (this file is compiled with -fmad=false):
//   0. the tree, by one persistent kernel over a queue of nodes (bvh_build_kernel);
//   1. one warp per (iy, iz) scanline of the mesh window: +X ray hits, sorted, even counts
//      fill [x_enter, x_exit], odd counts fall back to the 3-ray vote;
//   2. boundary detection over the window +-1, compacted in ascending cell order by a scan
//      of the x-rows' counts;
//   3. one thread per link of a boundary cell into a solid: Bouzidi q by a segment query.
// At 256x128x128 with 20 224 triangles (B200): tree 188 us, scanlines 21, links 115, the rest
// 30; aerosim_voxelize with the flow reset and the grid copied to the host 15 -> 1.2 ms
// against a tree built on the host, one thread per scanline and arrays allocated anew.
#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "engine_internal.h"

namespace aerosim {

namespace {

constexpr int kStack = 64;    // traversal stack depth (bvh.ts uses Int32Array(64))
constexpr int kMaxHits = 128; // scanline hits kept per ray

// A node of the tree, one 64-byte line: the box, then for an inner node its first child
// (the second follows it) and count 0, for a leaf its first triangle and their count.
// left_turns: left children on the way from the root, which is how many right siblings wait
// on the reference's traversal stack when it visits the node (VOX_ERR_STACK).
struct __align__(64) BvhNode {
  double lo[3], hi[3];
  int32_t first, count, left_turns, pad;
};
// Per triangle: the centroid and the bounds of the build.
struct TriKey {
  double cen[3], lo[3], hi[3];
};

// ---------------------------------------------------------------------------
// Host BVH build, bvh.ts:34-253: where the device build hands back a mesh whose split leaves
// one side empty (the reference then halves the triangles in their current order, which
// depends on every swap so far; it takes centroids a rounding apart, at coordinates above
// 4096, or overflow), where a scanline's hits hold a NaN (scanline_hits_ordered) or a wait in
// it ran out.
// ---------------------------------------------------------------------------
struct HostBvh {
  int tri_count = 0;
  std::vector<double> tri, nb, cen, tb;
  std::vector<int32_t> lof, cnt, tidx;
  double bmin[3] = {INFINITY, INFINITY, INFINITY};
  double bmax[3] = {-INFINITY, -INFINITY, -INFINITY};
  int next = 0;

  static double mn3(double a, double b, double c) { return js_min(js_min(a, b), c); }
  static double mx3(double a, double b, double c) { return js_max(js_max(a, b), c); }

  void node(int n, int first, int count) {
    double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    double clo[3] = {INFINITY, INFINITY, INFINITY}, chi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = first; i < first + count; ++i) {
      const int t = tidx[i];
      for (int a = 0; a < 3; ++a) {
        if (tb[t * 6 + a] < lo[a]) lo[a] = tb[t * 6 + a];
        if (tb[t * 6 + 3 + a] > hi[a]) hi[a] = tb[t * 6 + 3 + a];
        const double c = cen[t * 3 + a];
        if (c < clo[a]) clo[a] = c;
        if (c > chi[a]) chi[a] = c;
      }
    }
    for (int a = 0; a < 3; ++a) {
      nb[n * 6 + a] = lo[a];
      nb[n * 6 + 3 + a] = hi[a];
    }
    if (count <= 4) {
      lof[n] = first;
      cnt[n] = count;
      return;
    }
    int axis = 0;
    double ext = chi[0] - clo[0], split = 0.5 * (clo[0] + chi[0]);
    if (chi[1] - clo[1] > ext) { axis = 1; ext = chi[1] - clo[1]; split = 0.5 * (clo[1] + chi[1]); }
    if (chi[2] - clo[2] > ext) { axis = 2; ext = chi[2] - clo[2]; split = 0.5 * (clo[2] + chi[2]); }
    if (ext <= 1e-12) {
      lof[n] = first;
      cnt[n] = count;
      return;
    }
    int i = first, j = first + count - 1;
    while (i <= j) {
      if (cen[tidx[i] * 3 + axis] < split) ++i;
      else std::swap(tidx[i], tidx[j--]);
    }
    int left = i - first;
    if (left == 0 || left == count) left = count >> 1;
    const int child = next;
    next += 2;
    lof[n] = child;
    cnt[n] = 0;
    node(child, first, left);
    node(child + 1, first + left, count - left);
  }

  void build(const float* pos, int64_t nverts, const int32_t* idx, int64_t nidx, const double* m) {
    tri_count = idx ? (int)(nidx / 3) : (int)(nverts / 3);
    tri.assign((size_t)tri_count * 9, 0.0);
    cen.assign((size_t)tri_count * 3, 0.0);
    tb.assign((size_t)tri_count * 6, 0.0);
    tidx.resize(tri_count);
    for (int t = 0; t < tri_count; ++t) {
      tidx[t] = t;
      double v[3][3];
      for (int k = 0; k < 3; ++k) {
        const int64_t vi = idx ? (int64_t)idx[t * 3 + k] : (int64_t)t * 3 + k;
        double x = pos[vi * 3], y = pos[vi * 3 + 1], z = pos[vi * 3 + 2];
        if (m) {  // THREE.Vector3.applyMatrix4 (column-major elements, perspective divide)
          const double w = 1.0 / (m[3] * x + m[7] * y + m[11] * z + m[15]);
          const double px = (m[0] * x + m[4] * y + m[8] * z + m[12]) * w;
          const double py = (m[1] * x + m[5] * y + m[9] * z + m[13]) * w;
          const double pz = (m[2] * x + m[6] * y + m[10] * z + m[14]) * w;
          x = px; y = py; z = pz;
        }
        v[k][0] = x; v[k][1] = y; v[k][2] = z;
      }
      for (int a = 0; a < 3; ++a) {
        tri[t * 9 + a] = v[0][a];
        tri[t * 9 + 3 + a] = v[1][a] - v[0][a];
        tri[t * 9 + 6 + a] = v[2][a] - v[0][a];
        cen[t * 3 + a] = (v[0][a] + v[1][a] + v[2][a]) / 3.0;
        tb[t * 6 + a] = mn3(v[0][a], v[1][a], v[2][a]);
        tb[t * 6 + 3 + a] = mx3(v[0][a], v[1][a], v[2][a]);
        if (tb[t * 6 + a] < bmin[a]) bmin[a] = tb[t * 6 + a];
        if (tb[t * 6 + 3 + a] > bmax[a]) bmax[a] = tb[t * 6 + 3 + a];
      }
    }
    const int nodes = std::max(1, tri_count * 2);
    nb.assign((size_t)nodes * 6, 0.0);
    lof.assign(nodes, 0);
    cnt.assign(nodes, 0);
    if (tri_count > 0) {
      next = 1;
      node(0, 0, tri_count);
    }
  }
};

struct BvhView {
  const double* tri;
  const BvhNode* nodes;
  const int32_t* tidx;
  int tri_count;
  int host_order;  // the triangles of a leaf stand in the host build's order
};

// VOX_NAN_HITS is no error: a NaN among a scanline's hits, in a tree of the device build.
enum { VOX_ERR_STACK = 1, VOX_ERR_HITS = 2, VOX_NAN_HITS = 4 };

// ---------------------------------------------------------------------------
// Device BVH build.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double min3_js(double a, double b, double c) { return js_min(js_min(a, b), c); }
__device__ __forceinline__ double max3_js(double a, double b, double c) { return js_max(js_max(a, b), c); }

struct Mat16 { double m[16]; };

// Triangle t: world-space vertex and edges, centroid, bounds (bvh.ts:60-139).
__global__ void bvh_triangles_kernel(const float* __restrict__ pos, const int32_t* __restrict__ idx, int n, const Mat16 w,
                                     int has_w, double* __restrict__ tri, TriKey* __restrict__ key,
                                     int32_t* __restrict__ order) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  double v[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const long long vi = idx ? (long long)idx[(long long)t * 3 + k] : (long long)t * 3 + k;
    double x = pos[vi * 3], y = pos[vi * 3 + 1], z = pos[vi * 3 + 2];
    if (has_w) {  // THREE.Vector3.applyMatrix4 (column-major elements, perspective divide)
      const double* const m = w.m;
      const double iw = 1.0 / (m[3] * x + m[7] * y + m[11] * z + m[15]);
      const double px = (m[0] * x + m[4] * y + m[8] * z + m[12]) * iw;
      const double py = (m[1] * x + m[5] * y + m[9] * z + m[13]) * iw;
      const double pz = (m[2] * x + m[6] * y + m[10] * z + m[14]) * iw;
      x = px; y = py; z = pz;
    }
    v[k][0] = x; v[k][1] = y; v[k][2] = z;
  }
  TriKey k;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    tri[(size_t)t * 9 + a] = v[0][a];
    tri[(size_t)t * 9 + 3 + a] = v[1][a] - v[0][a];
    tri[(size_t)t * 9 + 6 + a] = v[2][a] - v[0][a];
    k.cen[a] = (v[0][a] + v[1][a] + v[2][a]) / 3.0;
    k.lo[a] = min3_js(v[0][a], v[1][a], v[2][a]);
    k.hi[a] = max3_js(v[0][a], v[1][a], v[2][a]);
  }
  key[t] = k;
  order[t] = t;
}

// One persistent kernel builds the tree from a queue of nodes.  A CTA that takes a node of
// more than kSubtree triangles reduces its bounds, splits it and goes on with the left
// child, leaving the right one in the queue; a smaller node's whole subtree is built from
// shared memory, a warp per node and level.  The order of the triangles inside a node is
// whatever the compaction leaves: no result depends on it (the nearest hit, the sorted hits
// and their parity do not, and the splits go by predicate), except where a split leaves one
// side empty, which is reported (BVH_DEGENERATE).  A CTA without a node polls the queue;
// no CTA with a node waits for another, and the polls are bounded.
// The top levels bound it: one CTA over all triangles, then two over half of them each.  188
// us for 20 224 triangles and 94 us for 8 784, where the host build took 5.0 and 2.2 ms;
// subtrees of 256 190 / 101 us, CTAs of 1024 threads 197 / 110, of 256 threads 239 / 111.
constexpr int kBuildThreads = 512, kBuildWarps = kBuildThreads / 32;
constexpr int kSubtree = 128;
constexpr int kBuildPolls = 1 << 20;
enum { BVH_DEGENERATE = 1, BVH_TIMEOUT = 2 };

struct BuildTask {
  int node, first, count, left_turns, side;  // side: which of the two order buffers holds it
};
struct BuildState {
  int head, tail, outstanding, next, error;
};
struct BuildArgs {
  const TriKey* key;
  int32_t* order[2];  // triangle order of the open nodes, by side
  int32_t* tidx;      // triangle order of the leaves
  BvhNode* nodes;
  BuildTask* queue;
  int* ready;         // [queue_cap]: the queue entry is written
  BuildState* st;
  int n, queue_cap;
};

// Bounds of a node's triangles: box lo/hi, centroid lo/hi.  NaN coordinates are passed over,
// as the reference's comparisons pass over them.
struct Bounds {
  double v[12];  // lo[3], clo[3] (minima), hi[3], chi[3] (maxima)
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      v[a] = INFINITY;
      v[6 + a] = -INFINITY;
    }
  }
  __device__ __forceinline__ void add(const TriKey& k) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[a] = fmin(v[a], k.lo[a]);
      v[3 + a] = fmin(v[3 + a], k.cen[a]);
      v[6 + a] = fmax(v[6 + a], k.hi[a]);
      v[9 + a] = fmax(v[9 + a], k.cen[a]);
    }
  }
  __device__ __forceinline__ void warp_reduce() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        v[a] = fmin(v[a], __shfl_xor_sync(0xffffffffu, v[a], o));
        v[6 + a] = fmax(v[6 + a], __shfl_xor_sync(0xffffffffu, v[6 + a], o));
      }
    }
  }
};

// The split of bvh.ts:180-205: axis and position, or a leaf (extent <= 1e-12).
__device__ __forceinline__ bool split_of(const double* v, int& axis, double& split) {
  axis = 0;
  double ext = v[9] - v[3];
  split = 0.5 * (v[3] + v[9]);
  if (v[10] - v[4] > ext) { axis = 1; ext = v[10] - v[4]; split = 0.5 * (v[4] + v[10]); }
  if (v[11] - v[5] > ext) { axis = 2; ext = v[11] - v[5]; split = 0.5 * (v[5] + v[11]); }
  return !(ext <= 1e-12);
}

__device__ __forceinline__ void write_node(BvhNode* n, const double* v, int first, int count, int left_turns) {
  BvhNode o;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    o.lo[a] = v[a];
    o.hi[a] = v[6 + a];
  }
  o.first = first;
  o.count = count;
  o.left_turns = left_turns;
  o.pad = 0;
  *n = o;
}

struct SubNode {
  int node, left_turns;
  short first, count;
};

__global__ void __launch_bounds__(kBuildThreads) bvh_build_kernel(const BuildArgs a) {
  __shared__ BuildTask task;
  __shared__ int s_state;  // 1: a task, 0: the tree is done, -1: a wait ran out
  __shared__ double s_bounds[kBuildWarps][12];
  __shared__ int s_left, s_right, s_child;
  __shared__ TriKey s_key[kSubtree];
  __shared__ int32_t s_tri[kSubtree];
  __shared__ short s_list[2][kSubtree];
  __shared__ SubNode s_node[2][kSubtree];
  __shared__ int s_count[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile BuildState* const st = a.st;

  for (;;) {
    if (tid == 0) {
      const int k = atomicAdd(&a.st->head, 1);
      int state = -1;
      for (int i = 0; i < kBuildPolls; ++i) {
        if (k < a.queue_cap && *(volatile int*)&a.ready[k]) {
          __threadfence();
          task = a.queue[k];
          state = 1;
          break;
        }
        if (st->outstanding == 0) {
          state = 0;
          break;
        }
        __nanosleep(64);
      }
      if (state < 0) atomicOr(&a.st->error, BVH_TIMEOUT);
      s_state = state;
    }
    __syncthreads();
    if (s_state <= 0) return;
    BuildTask t = task;
    // ---- nodes above kSubtree triangles: split, go on with the left child ----
    while (t.count > kSubtree) {
      const int32_t* const in = a.order[t.side] + t.first;
      int32_t* const out = a.order[t.side ^ 1] + t.first;
      Bounds b;
      b.clear();
      for (int i = tid; i < t.count; i += kBuildThreads) b.add(a.key[in[i]]);
      b.warp_reduce();
      if (lane == 0) {
#pragma unroll
        for (int c = 0; c < 12; ++c) s_bounds[warp][c] = b.v[c];
      }
      if (tid == 0) s_left = s_right = 0;
      __syncthreads();
      if (tid < 12) {
        double m = s_bounds[0][tid];
        for (int w = 1; w < kBuildWarps; ++w) m = tid < 6 ? fmin(m, s_bounds[w][tid]) : fmax(m, s_bounds[w][tid]);
        s_bounds[0][tid] = m;
      }
      __syncthreads();
      int axis;
      double split;
      const bool inner = split_of(s_bounds[0], axis, split);
      if (!inner) {  // coincident centroids: a leaf of any size
        for (int i = tid; i < t.count; i += kBuildThreads) a.tidx[t.first + i] = in[i];
        if (tid == 0) write_node(&a.nodes[t.node], s_bounds[0], t.first, t.count, t.left_turns);
        t.count = 0;
        break;
      }
      for (int i0 = 0; i0 < t.count; i0 += kBuildThreads) {
        const int i = i0 + tid;
        const bool in_range = i < t.count;
        const int tri = in_range ? in[i] : 0;
        const bool left = in_range && a.key[tri].cen[axis] < split, right = in_range && !left;
        const unsigned ml = __ballot_sync(0xffffffffu, left), mr = __ballot_sync(0xffffffffu, right);
        int bl = 0, br = 0;
        if (lane == 0) {
          bl = atomicAdd(&s_left, __popc(ml));
          br = atomicAdd(&s_right, __popc(mr));
        }
        bl = __shfl_sync(0xffffffffu, bl, 0);
        br = __shfl_sync(0xffffffffu, br, 0);
        const unsigned below = (1u << lane) - 1u;
        if (left) out[bl + __popc(ml & below)] = tri;
        if (right) out[t.count - 1 - (br + __popc(mr & below))] = tri;
      }
      __threadfence();  // the order is read by whichever CTA takes the right child
      __syncthreads();
      const int left = s_left;
      if (left == 0 || left == t.count) {
        if (tid == 0) {
          atomicOr(&a.st->error, BVH_DEGENERATE);
          write_node(&a.nodes[t.node], s_bounds[0], t.first, 0, t.left_turns);
        }
        t.count = 0;
        break;
      }
      if (tid == 0) {
        const int child = atomicAdd(&a.st->next, 2);
        write_node(&a.nodes[t.node], s_bounds[0], child, 0, t.left_turns);
        atomicAdd(&a.st->outstanding, 1);
        const int slot = atomicAdd(&a.st->tail, 1);
        a.queue[slot] = BuildTask{child + 1, t.first + left, t.count - left, t.left_turns, t.side ^ 1};
        __threadfence();
        atomicExch(&a.ready[slot], 1);
        s_child = child;
      }
      __syncthreads();
      t.node = s_child;
      t.count = left;
      t.left_turns += 1;
      t.side ^= 1;
    }
    __syncthreads();
    // ---- the subtree of a small node, level by level ----
    if (t.count > 0) {
      const int32_t* const in = a.order[t.side] + t.first;
      for (int i = tid; i < t.count; i += kBuildThreads) {
        const int tri = in[i];
        s_tri[i] = tri;
        s_key[i] = a.key[tri];
        s_list[0][i] = (short)i;
      }
      if (tid == 0) {
        s_node[0][0] = SubNode{t.node, t.left_turns, 0, (short)t.count};
        s_count[0] = 1;
        s_count[1] = 0;
      }
      __syncthreads();
      for (int level = 0;; ++level) {
        const int cur = level & 1, nodes = s_count[cur];
        if (nodes == 0) break;
        for (int q = warp; q < nodes; q += kBuildWarps) {
          const SubNode nd = s_node[cur][q];
          const short* const li = s_list[cur] + nd.first;
          short* const lo = s_list[cur ^ 1] + nd.first;
          Bounds b;
          b.clear();
          for (int i = lane; i < nd.count; i += 32) b.add(s_key[li[i]]);
          b.warp_reduce();
          int axis;
          double split;
          const bool inner = split_of(b.v, axis, split) && nd.count > 4;
          if (!inner) {
            for (int i = lane; i < nd.count; i += 32) a.tidx[t.first + nd.first + i] = s_tri[li[i]];
            if (lane == 0) write_node(&a.nodes[nd.node], b.v, t.first + nd.first, nd.count, nd.left_turns);
            continue;
          }
          int nl = 0, nr = 0;
          for (int i0 = 0; i0 < nd.count; i0 += 32) {
            const int i = i0 + lane;
            const bool in_range = i < nd.count;
            const short k = in_range ? li[i] : (short)0;
            const bool left = in_range && s_key[k].cen[axis] < split, right = in_range && !left;
            const unsigned ml = __ballot_sync(0xffffffffu, left), mr = __ballot_sync(0xffffffffu, right);
            const unsigned below = (1u << lane) - 1u;
            if (left) lo[nl + __popc(ml & below)] = k;
            if (right) lo[nd.count - 1 - (nr + __popc(mr & below))] = k;
            nl += __popc(ml);
            nr += __popc(mr);
          }
          if (lane == 0) {
            if (nl == 0 || nr == 0) {
              atomicOr(&a.st->error, BVH_DEGENERATE);
              write_node(&a.nodes[nd.node], b.v, t.first + nd.first, 0, nd.left_turns);
            } else {
              const int child = atomicAdd(&a.st->next, 2);
              write_node(&a.nodes[nd.node], b.v, child, 0, nd.left_turns);
              const int at = atomicAdd(&s_count[cur ^ 1], 2);
              s_node[cur ^ 1][at] = SubNode{child, nd.left_turns + 1, nd.first, (short)nl};
              s_node[cur ^ 1][at + 1] = SubNode{child + 1, nd.left_turns, (short)(nd.first + nl), (short)nr};
            }
          }
        }
        __syncthreads();
        if (tid == 0) s_count[cur] = 0;
        __syncthreads();
      }
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicSub(&a.st->outstanding, 1);
    }
  }
}

// One lane of the warp's traversals: a node's box and links as four 16-byte loads.
__device__ __forceinline__ BvhNode load_node(const BvhNode* p) {
  BvhNode n;
  const double2* const q = reinterpret_cast<const double2*>(p);
  const double2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
  const int4 d = __ldg(reinterpret_cast<const int4*>(q + 3));
  n.lo[0] = a.x; n.lo[1] = a.y; n.lo[2] = b.x;
  n.hi[0] = b.y; n.hi[1] = c.x; n.hi[2] = c.y;
  n.first = d.x; n.count = d.y; n.left_turns = d.z; n.pad = d.w;
  return n;
}

// One triangle of bvh.ts:375-457 collectXScanlineHits; x is where the line meets it.
__device__ __forceinline__ bool scanline_hit(const double* T, double py, double pz, double& x) {
  const double ax = T[0], ay = T[1], az = T[2];
  const double e1x = T[3], e1y = T[4], e1z = T[5];
  const double e2x = T[6], e2y = T[7], e2z = T[8];
  const double det = -e1y * e2z + e1z * e2y;
  if (fabs(det) < 1e-13) return false;
  const double inv = 1.0 / det;
  const double ty = py - ay, tz = pz - az;
  const double u = (-ty * e2z + tz * e2y) * inv;
  if (u < 0.0 || u > 1.0) return false;
  const double v = (ty * e1z - tz * e1y) * inv;
  if (v < 0.0 || u + v > 1.0) return false;
  x = ax + u * e1x + v * e2x;
  return true;
}

// bvh.ts:375-457 collectXScanlineHits by a warp: up to 32 waiting nodes at a time, a lane
// each; hits (unsorted) go to shared memory.  With the stack nearly full the warp takes one
// node at a time, depth first, which needs at most kStack - 1 more entries (a deeper path is
// refused as the reference's stack refuses it).  Returns the number of hits, the same for
// every lane.
constexpr int kWarpStack = 512;
__device__ int scanline_hits_warp(const BvhView& b, double y, double z, int* stack, double* hits, int* s_n, int lane, int* err) {
  if (b.tri_count == 0) return 0;
  const double py = y + 1.37e-8, pz = z + 2.93e-8;
  if (lane == 0) {
    stack[0] = 0;
    *s_n = 0;
  }
  __syncwarp();
  int sp = 1;
  bool bad = false;
  while (sp > 0) {
    const int m = sp + 32 <= kWarpStack - 2 * kStack ? min(32, sp) : 1;
    int push = -1;
    if (lane < m) {
      const BvhNode nd = load_node(b.nodes + stack[sp - 1 - lane]);
      if (!(py < nd.lo[1] || py > nd.hi[1] || pz < nd.lo[2] || pz > nd.hi[2])) {
        if (nd.count > 0) {
          for (int i = nd.first; i < nd.first + nd.count; ++i) {
            double x;
            if (!scanline_hit(b.tri + (size_t)b.tidx[i] * 9, py, pz, x)) continue;
            const int at = atomicAdd(s_n, 1);
            if (at < kMaxHits) hits[at] = x;
            else atomicOr(err, VOX_ERR_HITS);
          }
        } else if (nd.left_turns + 2 > kStack) {
          atomicOr(err, VOX_ERR_STACK);
          bad = true;
        } else {
          push = nd.first;
        }
      }
    }
    __syncwarp();
    const unsigned mask = __ballot_sync(0xffffffffu, push >= 0);
    sp -= m;
    if (push >= 0) {
      const int at = sp + 2 * __popc(mask & ((1u << lane) - 1u));
      stack[at] = push + 1;
      stack[at + 1] = push;
    }
    sp += 2 * __popc(mask);
    __syncwarp();
    if (__any_sync(0xffffffffu, bad)) return 0;
  }
  const int n = *s_n;
  return n < kMaxHits ? n : kMaxHits;
}

// The same by one thread, in the reference's order (leaves left to right, triangles as the host
// build left them), and its insertion sort.  Hits that hold a NaN (a vertex without an x, as
// damaged STL files have them) come out of a sort in an order that depends on the one they
// came in, and so does what they fill.
__device__ int scanline_hits_ordered(const BvhView& b, double y, double z, int* stack, double* hits, int* err) {
  const double py = y + 1.37e-8, pz = z + 2.93e-8;
  int sp = 0, n = 0;
  stack[sp++] = 0;
  while (sp > 0) {
    const BvhNode nd = load_node(b.nodes + stack[--sp]);
    if (py < nd.lo[1] || py > nd.hi[1] || pz < nd.lo[2] || pz > nd.hi[2]) continue;
    if (nd.count == 0) {
      if (sp + 2 > kStack) { atomicOr(err, VOX_ERR_STACK); return 0; }
      stack[sp++] = nd.first + 1;
      stack[sp++] = nd.first;
      continue;
    }
    for (int i = nd.first; i < nd.first + nd.count; ++i) {
      double x;
      if (!scanline_hit(b.tri + (size_t)b.tidx[i] * 9, py, pz, x)) continue;
      if (n < kMaxHits) hits[n] = x;
      else atomicOr(err, VOX_ERR_HITS);
      ++n;
    }
  }
  n = n < kMaxHits ? n : kMaxHits;
  for (int i = 1; i < n; ++i) {
    const double key = hits[i];
    int j = i - 1;
    while (j >= 0 && hits[j] > key) { hits[j + 1] = hits[j]; --j; }
    hits[j + 1] = key;
  }
  return n;
}

// bvh.ts:499-589 countRayIntersections
__device__ int count_ray(const BvhView& b, double ox, double oy, double oz, double dx, double dy,
                         double dz, int* err) {
  const double ix = 1.0 / dx, iy = 1.0 / dy, iz = 1.0 / dz;
  int hits = 0;
  int stack[kStack];
  int sp = 0;
  stack[sp++] = 0;
  while (sp > 0) {
    const int n = stack[--sp];
    const BvhNode nd = load_node(b.nodes + n);
    const double tx1 = (nd.lo[0] - ox) * ix, tx2 = (nd.hi[0] - ox) * ix;
    double tmin = js_min(tx1, tx2), tmax = js_max(tx1, tx2);
    const double ty1 = (nd.lo[1] - oy) * iy, ty2 = (nd.hi[1] - oy) * iy;
    tmin = js_max(tmin, js_min(ty1, ty2));
    tmax = js_min(tmax, js_max(ty1, ty2));
    const double tz1 = (nd.lo[2] - oz) * iz, tz2 = (nd.hi[2] - oz) * iz;
    tmin = js_max(tmin, js_min(tz1, tz2));
    tmax = js_min(tmax, js_max(tz1, tz2));
    if (tmax < js_max(0, tmin)) continue;
    const int c = nd.count;
    if (c > 0) {
      const int first = nd.first;
      for (int i = first; i < first + c; ++i) {
        const double* T = b.tri + (size_t)b.tidx[i] * 9;
        const double ax = T[0], ay = T[1], az = T[2];
        const double e1x = T[3], e1y = T[4], e1z = T[5];
        const double e2x = T[6], e2y = T[7], e2z = T[8];
        const double px = dy * e2z - dz * e2y;
        const double py = dz * e2x - dx * e2z;
        const double pz = dx * e2y - dy * e2x;
        const double det = e1x * px + e1y * py + e1z * pz;
        if (fabs(det) < 1e-13) continue;
        const double inv = 1.0 / det;
        const double tx = ox - ax, ty = oy - ay, tz = oz - az;
        const double u = (tx * px + ty * py + tz * pz) * inv;
        if (u < 0.0 || u > 1.0) continue;
        const double qx = ty * e1z - tz * e1y;
        const double qy = tz * e1x - tx * e1z;
        const double qz = tx * e1y - ty * e1x;
        const double v = (dx * qx + dy * qy + dz * qz) * inv;
        if (v < 0.0 || u + v > 1.0) continue;
        const double t = (e2x * qx + e2y * qy + e2z * qz) * inv;
        if (t > 1e-7) ++hits;
      }
    } else {
      if (sp + 2 > kStack) { atomicOr(err, VOX_ERR_STACK); return 0; }
      const int l = nd.first;
      stack[sp++] = l + 1;
      stack[sp++] = l;
    }
  }
  return hits;
}

// bvh.ts:464-497 isPointInside: 3 skew rays, 2-of-3 parity vote.
__device__ bool point_inside(const BvhView& b, double x, double y, double z, int* err) {
  const BvhNode root = load_node(b.nodes);  // the mesh bounds
  if (x < root.lo[0] || x > root.hi[0] || y < root.lo[1] || y > root.hi[1] || z < root.lo[2] || z > root.hi[2])
    return false;
  const double D[3][3] = {{1.0, 0.0137, 0.0293}, {-0.0191, 1.0, 0.0317}, {0.0239, -0.0173, 1.0}};
  int votes = 0;
  for (int d = 0; d < 3; ++d) {
    if ((count_ray(b, x, y, z, D[d][0], D[d][1], D[d][2], err) & 1) == 1) ++votes;
    if (votes >= 2) return true;
    if (d == 1 && votes == 0) return false;
  }
  return votes >= 2;
}

// bvh.ts:265-367 intersectSegment.  The reference pops a node and tests its box; here both
// children's boxes (128 adjacent bytes) are loaded and tested when their parent is visited,
// which halves the chain of dependent loads that bounds the query, and a waiting right child
// keeps its entry distance, so that its test against the nearest hit still happens when its
// turn comes.  The same leaves are visited in the same order with the same nearest hit.
__device__ double segment(const BvhView& b, double ox, double oy, double oz, double dx, double dy,
                          double dz, double maxT, int* err) {
  if (b.tri_count == 0) return -1;
  const double ix = fabs(dx) > 1e-15 ? 1.0 / dx : (dx >= 0 ? 1e15 : -1e15);
  const double iy = fabs(dy) > 1e-15 ? 1.0 / dy : (dy >= 0 ? 1e15 : -1e15);
  const double iz = fabs(dz) > 1e-15 ? 1.0 / dz : (dz >= 0 ? 1e15 : -1e15);
  double closest = maxT + 1e-7;
  bool found = false;
  // the slab test without the nearest hit: false when the box is missed
  auto enter = [&](const BvhNode& nd, double& tmin) {
    const double tx1 = (nd.lo[0] - ox) * ix, tx2 = (nd.hi[0] - ox) * ix;
    tmin = js_min(tx1, tx2);
    double tmax = js_max(tx1, tx2);
    const double ty1 = (nd.lo[1] - oy) * iy, ty2 = (nd.hi[1] - oy) * iy;
    tmin = js_max(tmin, js_min(ty1, ty2));
    tmax = js_min(tmax, js_max(ty1, ty2));
    const double tz1 = (nd.lo[2] - oz) * iz, tz2 = (nd.hi[2] - oz) * iz;
    tmin = js_max(tmin, js_min(tz1, tz2));
    tmax = js_min(tmax, js_max(tz1, tz2));
    return !(tmax < js_max(0, tmin));
  };
  // waiting right children, at most one per left turn of the path: their links and entry
  int4 stack[kStack];
  double wait[kStack];
  int sp = 0;
  int first, count, turns;
  {
    const BvhNode root = load_node(b.nodes);
    double tmin;
    if (!enter(root, tmin) || tmin > closest) return -1;
    first = root.first; count = root.count; turns = root.left_turns;
  }
  for (;;) {
    bool next = false;  // the left child follows its parent
    if (count > 0) {
      for (int i = first; i < first + count; ++i) {
        const double* T = b.tri + (size_t)b.tidx[i] * 9;
        const double ax = T[0], ay = T[1], az = T[2];
        const double e1x = T[3], e1y = T[4], e1z = T[5];
        const double e2x = T[6], e2y = T[7], e2z = T[8];
        const double px = dy * e2z - dz * e2y;
        const double py = dz * e2x - dx * e2z;
        const double pz = dx * e2y - dy * e2x;
        const double det = e1x * px + e1y * py + e1z * pz;
        if (fabs(det) < 1e-13) continue;
        const double inv = 1.0 / det;
        const double tx = ox - ax, ty = oy - ay, tz = oz - az;
        const double u = (tx * px + ty * py + tz * pz) * inv;
        if (u < -1e-7 || u > 1.0 + 1e-7) continue;
        const double qx = ty * e1z - tz * e1y;
        const double qy = tz * e1x - tx * e1z;
        const double qz = tx * e1y - ty * e1x;
        const double v = (dx * qx + dy * qy + dz * qz) * inv;
        if (v < -1e-7 || u + v > 1.0 + 1e-7) continue;
        const double t = (e2x * qx + e2y * qy + e2z * qz) * inv;
        if (t > 1e-7 && t <= closest) {
          closest = t;
          found = true;
        }
      }
    } else {
      if (turns + 2 > kStack) { atomicOr(err, VOX_ERR_STACK); return -1; }
      const BvhNode l = load_node(b.nodes + first), r = load_node(b.nodes + first + 1);
      double tl, tr;
      const bool in_l = enter(l, tl) && !(tl > closest), in_r = enter(r, tr) && !(tr > closest);
      if (in_r) {
        stack[sp] = make_int4(r.first, r.count, r.left_turns, 0);
        wait[sp++] = tr;
      }
      if (in_l) {
        first = l.first; count = l.count; turns = l.left_turns;
        next = true;
      }
    }
    while (!next) {
      if (sp == 0) return found ? js_min(maxT, closest) : -1;
      --sp;
      if (wait[sp] > closest) continue;
      first = stack[sp].x; count = stack[sp].y; turns = stack[sp].z;
      next = true;
    }
  }
}

struct Lattice {
  int nx, ny, nz;
  double h, ox, oy, oz;
  int w[6];  // mesh window minIx, maxIx, minIy, maxIy, minIz, maxIz
};

// STEP 1, voxelizer.ts:127-173.  One warp per (iy, iz) of the window: a thread each left
// 9 CTAs at work on 1152 scanlines, 533 us; a warp's lanes share the nodes, the sort, the
// cells of a filled interval and those of a 3-ray vote (21 us).
constexpr int kScanWarps = 4;
__global__ void __launch_bounds__(kScanWarps * 32) scan_fill_kernel(BvhView b, Lattice L, uint8_t* flags,
                                 unsigned long long* solid_count, int* err) {
  __shared__ int s_stack[kScanWarps][kWarpStack];
  __shared__ double s_hits[kScanWarps][2][kMaxHits];
  __shared__ int s_n[kScanWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wy = L.w[3] - L.w[2] + 1, wz = L.w[5] - L.w[4] + 1;
  const long long t = (long long)blockIdx.x * kScanWarps + warp;
  if (t >= (long long)wy * wz) return;
  const int iy = L.w[2] + (int)(t % wy), iz = L.w[4] + (int)(t / wy);
  const double z = L.oz + (iz + 0.5) * L.h;
  const double y = L.oy + (iy + 0.5) * L.h;
  const int hc = scanline_hits_warp(b, y, z, s_stack[warp], s_hits[warp][0], &s_n[warp], lane, err);
  if (hc == 0) return;
  // ascending numeric sort by rank (equal hits in any order: they are the same number)
  const double* const raw = s_hits[warp][0];
  double* const hits = s_hits[warp][1];
  bool nan = false;
  for (int i = lane; i < hc; i += 32) {
    const double v = raw[i];
    int rank = 0;
    for (int j = 0; j < hc; ++j) rank += raw[j] < v || (raw[j] == v && j < i);
    hits[rank] = v;
    nan |= v != v;
  }
  if (__any_sync(0xffffffffu, nan)) {  // ranks are none
    if (!b.host_order) {  // the host starts over with its own tree
      if (lane == 0) atomicOr(err, VOX_NAN_HITS);
      return;
    }
    if (lane == 0) scanline_hits_ordered(b, y, z, s_stack[warp], hits, err);
  }
  __syncwarp();
  uint8_t* row = flags + (long long)L.nx * (iy + (long long)L.ny * iz);
  unsigned added = 0;
  const int minIx = L.w[0], maxIx = L.w[1];
  if ((hc & 1) == 0) {
    for (int k = 0; k < hc; k += 2) {
      const double xe = hits[k], xx = hits[k + 1];
      if (xx - xe < 1e-7) continue;
      const double s = js_max((double)minIx, ceil((xe - L.ox) / L.h - 0.5));
      const double e = js_min((double)maxIx, floor((xx - L.ox) / L.h - 0.5));
      if (!(s <= e)) continue;
      for (int ix = (int)s + lane; ix <= (int)e; ix += 32) {
        if (row[ix] == CELL_FLUID) {
          row[ix] = CELL_SOLID;
          ++added;
        }
      }
      __syncwarp();  // intervals may share a cell: the next one sees this one's
    }
  } else {
    for (int ix = minIx + lane; ix <= maxIx; ix += 32) {
      const double x = L.ox + (ix + 0.5) * L.h;
      if (x >= hits[0] && x <= hits[hc - 1]) {
        if (point_inside(b, x, y, z, err) && row[ix] == CELL_FLUID) {
          row[ix] = CELL_SOLID;
          ++added;
        }
      }
    }
    __syncwarp();
  }
  added = __reduce_add_sync(0xffffffffu, added);
  if (lane == 0 && added) atomicAdd(solid_count, (unsigned long long)added);
}

// STEP 2, voxelizer.ts:176-212: FLUID cells with an in-bounds SOLID neighbour, one warp per
// x-row of the window.  The first pass counts them, the second (first != null) writes the
// list, the map and the flags from the rows' first positions; it changes only FLUID to
// BOUNDARY, which no test of another cell looks at.
__global__ void boundary_rows_kernel(uint8_t* flags, Lattice L, int sx0, int sy0, int sz0, int wx, int wy, long long rows,
                                     uint32_t* __restrict__ counts, const uint32_t* __restrict__ first,
                                     int32_t* __restrict__ bcells, int32_t* __restrict__ bmap) {
  const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const int iy = sy0 + (int)(r % wy), iz = sz0 + (int)(r / wy);
  const long long row = (long long)L.nx * (iy + (long long)L.ny * iz);
  uint32_t at = first ? first[r] : 0u;
  for (int x0 = 0; x0 < wx; x0 += 32) {
    const int ix = sx0 + x0 + lane;
    bool m = false;
    if (x0 + lane < wx && flags[row + ix] == CELL_FLUID) {
#pragma unroll
      for (int d = 1; d < 19; ++d) {
        const int a = ix + cx_of(d), bb = iy + cy_of(d), c = iz + cz_of(d);
        if (a < 0 || a >= L.nx || bb < 0 || bb >= L.ny || c < 0 || c >= L.nz) continue;
        if (flags[a + (long long)L.nx * (bb + (long long)L.ny * c)] == CELL_SOLID) m = true;
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, m);
    if (first && m) {
      const uint32_t k = at + __popc(mask & ((1u << lane) - 1u));
      flags[row + ix] = CELL_BOUNDARY;
      bcells[k] = (int32_t)(row + ix);
      bmap[row + ix] = (int32_t)k;
    }
    at += (uint32_t)__popc(mask);
  }
  if (!first && lane == 0) counts[r] = at;
}

// STEP 3, voxelizer.ts:221-256 (+ computeSubGridLinkFraction :65-80).  About a third of a
// boundary cell's links end in a solid: a CTA first gathers those of its kLinkCells cells,
// so that every thread of the second part has a query.
constexpr int kLinkThreads = 128, kLinkCells = 16;
__global__ void __launch_bounds__(kLinkThreads) q_links_kernel(BvhView bv, Lattice L, const uint8_t* __restrict__ flags,
                               const int32_t* __restrict__ bcells, long long B, float* __restrict__ q,
                               float* __restrict__ minq, int* err) {
  __shared__ short s_link[kLinkCells * 18];
  __shared__ float s_q[kLinkCells * 18];
  __shared__ int s_n;
  const long long b0 = (long long)blockIdx.x * kLinkCells;
  const int cells = (int)min((long long)kLinkCells, B - b0);
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  auto coords = [&](int cell, int& ix, int& iy, int& iz) {
    const int ci = bcells[b0 + cell];
    const int row = ci / L.nx;
    ix = ci - row * L.nx;
    iz = row / L.ny;
    iy = row - iz * L.ny;
  };
  auto vec = [&](int d, int& cx, int& cy, int& cz) {
    cx = cy = cz = 0;
#pragma unroll
    for (int e = 1; e < 19; ++e)
      if (e == d) {
        cx = cx_of(e); cy = cy_of(e); cz = cz_of(e);
      }
  };
  for (int k = threadIdx.x; k < cells * 18; k += kLinkThreads) {
    int ix, iy, iz, cx, cy, cz;
    coords(k / 18, ix, iy, iz);
    vec(k % 18 + 1, cx, cy, cz);
    const int a = ix + cx, bb = iy + cy, c = iz + cz;
    s_q[k] = -1.0f;
    if (!(a < 0 || a >= L.nx || bb < 0 || bb >= L.ny || c < 0 || c >= L.nz) &&
        flags[a + (long long)L.nx * (bb + (long long)L.ny * c)] == CELL_SOLID)
      s_link[atomicAdd(&s_n, 1)] = (short)k;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < s_n; i += kLinkThreads) {
    const int k = s_link[i];
    int ix, iy, iz, cx, cy, cz;
    coords(k / 18, ix, iy, iz);
    vec(k % 18 + 1, cx, cy, cz);
    const double fx = L.ox + (ix + 0.5) * L.h, fy = L.oy + (iy + 0.5) * L.h,
                 fz = L.oz + (iz + 0.5) * L.h;
    const double tq = segment(bv, fx, fy, fz, cx * L.h, cy * L.h, cz * L.h, 1.0, err);
    double qv = 0.5;
    if (tq > 0 && tq <= 1.0) qv = js_max(1e-4, js_min(1.0, tq));
    s_q[k] = (float)qv;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < cells * 18; k += kLinkThreads) q[b0 * 18 + k] = s_q[k];
  if (threadIdx.x < cells) {
    float m = 1.0f;
    for (int k = 0; k < 18; ++k) {
      const float v = s_q[threadIdx.x * 18 + k];
      if (v > 0.0f && v < m) m = v;
    }
    minq[b0 + threadIdx.x] = m;
  }
}

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// The host build's tree in the device form.
void host_nodes(const HostBvh& hb, std::vector<BvhNode>* out) {
  out->assign(std::max(hb.next, 1), BvhNode{});
  for (int n = 0; n < hb.next; ++n) {
    BvhNode& o = (*out)[n];
    for (int a = 0; a < 3; ++a) {
      o.lo[a] = hb.nb[n * 6 + a];
      o.hi[a] = hb.nb[n * 6 + 3 + a];
    }
    o.first = hb.lof[n];
    o.count = hb.cnt[n];
    if (o.count == 0) {  // children come after their parent
      (*out)[o.first].left_turns = o.left_turns + 1;
      (*out)[o.first + 1].left_turns = o.left_turns;
    }
  }
}

}  // namespace

#define VCHECK(x)                                                              \
  do {                                                                         \
    cudaError_t e_ = (x);                                                      \
    if (e_ != cudaSuccess) {                                                   \
      *err = std::string("voxelizer: ") + #x + ": " + cudaGetErrorString(e_);  \
      return e_ == cudaErrorMemoryAllocation ? -5 : -3;                        \
    }                                                                          \
  } while (0)

int run_voxelizer(const float* pos, int64_t nverts, const int32_t* idx, int64_t nidx,
                  const double* world16, double tunnel_height, int nx, int ny, int nz,
                  cudaStream_t s, VoxScratch* w, DevGrid* g, std::string* err) {
  const auto t0 = std::chrono::steady_clock::now();
  const int T = idx ? (int)(nidx / 3) : (int)(nverts / 3);
  const long long N = (long long)nx * ny * nz;
  const double h = tunnel_height / ny;
  Lattice L{nx, ny, nz, h, -nx * h * 0.5, -ny * h * 0.5, -nz * h * 0.5, {0, 0, 0, 0, 0, 0}};
  // results that the host reads: pinned words, written by copies on the stream
  VCHECK(w->pinned());
  volatile unsigned long long* const total = w->host;                       // boundary cells
  unsigned long long* const h_solid = w->host + 1;
  int* const h_err = reinterpret_cast<int*>(w->host + 2);
  BuildState* const h_build = reinterpret_cast<BuildState*>(w->host + 4);
  BvhNode* const h_root = reinterpret_cast<BvhNode*>(w->host + 8);
  static_assert(sizeof(BuildState) <= 32 && sizeof(BvhNode) == 64, "layout of the pinned results");
  // device scratch: counters, the mesh, the tree, counts of the window's rows
  const int max_nodes = std::max(1, 2 * T);
  const long long max_rows = (long long)ny * nz;
  const size_t b_pos = up256((size_t)std::max<int64_t>(nverts, 1) * 12), b_idx = up256((size_t)(idx ? std::max<int64_t>(nidx, 1) : 1) * 4),
               b_tri = up256((size_t)std::max(T, 1) * 72), b_key = up256((size_t)std::max(T, 1) * sizeof(TriKey)),
               b_ord = up256((size_t)std::max(T, 1) * 4), b_nodes = up256((size_t)max_nodes * sizeof(BvhNode)),
               b_queue = up256((size_t)max_nodes * sizeof(BuildTask)), b_ready = up256((size_t)max_nodes * 4),
               b_rows = up256((size_t)max_rows * 4);
  VCHECK(w->device(512 + b_pos + b_idx + b_tri + b_key + 3 * b_ord + b_nodes + b_queue + b_ready + b_rows));
  char* c = static_cast<char*>(w->dev);
  auto take = [&](size_t b) { char* p = c; c += b; return p; };
  char* const counters = take(512);
  unsigned long long* const d_solid = reinterpret_cast<unsigned long long*>(counters);
  int* const d_err = reinterpret_cast<int*>(counters + 8);
  BuildState* const d_build = reinterpret_cast<BuildState*>(counters + 64);
  int* const d_ready = reinterpret_cast<int*>(take(b_ready));  // cleared with the counters
  float* const d_pos = reinterpret_cast<float*>(take(b_pos));
  int32_t* const d_idx = reinterpret_cast<int32_t*>(take(b_idx));
  double* const d_tri = reinterpret_cast<double*>(take(b_tri));
  TriKey* const d_key = reinterpret_cast<TriKey*>(take(b_key));
  int32_t* const d_ord0 = reinterpret_cast<int32_t*>(take(b_ord));
  int32_t* const d_ord1 = reinterpret_cast<int32_t*>(take(b_ord));
  int32_t* const d_tidx = reinterpret_cast<int32_t*>(take(b_ord));
  BvhNode* const d_nodes = reinterpret_cast<BvhNode*>(take(b_nodes));
  BuildTask* const d_queue = reinterpret_cast<BuildTask*>(take(b_queue));
  uint32_t* const d_rows = reinterpret_cast<uint32_t*>(take(b_rows));

  g->nx = nx; g->ny = ny; g->nz = nz; g->N = N;
  g->h = h; g->ox = L.ox; g->oy = L.oy; g->oz = L.oz;
  VCHECK(grid_cells(g, N, (size_t)make_layout(nx, ny, nz).plane));
  VCHECK(cudaMemsetAsync(g->flags, 0, N, s));
  VCHECK(cudaMemsetAsync(g->bmap, 0xff, N * sizeof(int32_t), s));
  VCHECK(cudaMemsetAsync(counters, 0, 512 + b_ready, s));
  *total = 0;
  *h_solid = 0;
  *h_err = 0;
  BvhView bv{d_tri, d_nodes, d_tidx, T, 0};
  auto host_tree = [&]() -> cudaError_t {
    HostBvh hb;
    hb.build(pos, nverts, idx, nidx, world16);
    std::vector<BvhNode> nodes;
    host_nodes(hb, &nodes);
    cudaError_t e = cudaMemcpyAsync(d_nodes, nodes.data(), nodes.size() * sizeof(BvhNode), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_tidx, hb.tidx.data(), hb.tidx.size() * 4, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *h_root = nodes[0];
    bv.host_order = 1;
    return e;
  };
  double bmin[3] = {INFINITY, INFINITY, INFINITY}, bmax[3] = {-INFINITY, -INFINITY, -INFINITY};
  if (T > 0) {
    VCHECK(cudaMemcpyAsync(d_pos, pos, (size_t)nverts * 12, cudaMemcpyHostToDevice, s));
    if (idx) VCHECK(cudaMemcpyAsync(d_idx, idx, (size_t)nidx * 4, cudaMemcpyHostToDevice, s));
    Mat16 m{};
    if (world16) std::memcpy(m.m, world16, sizeof(m.m));
    bvh_triangles_kernel<<<(unsigned)(((long long)T + 127) / 128), 128, 0, s>>>(d_pos, idx ? d_idx : nullptr, T, m, world16 != nullptr,
                                                                   d_tri, d_key, d_ord0);
    // the root: one task, one node
    BuildState* const init = h_build;
    *init = BuildState{0, 1, 1, 1, 0};
    BuildTask* const root_task = reinterpret_cast<BuildTask*>(w->host + 16);
    *root_task = BuildTask{0, 0, T, 0, 0};
    int* const one = reinterpret_cast<int*>(w->host + 20);
    *one = 1;
    VCHECK(cudaMemcpyAsync(d_build, init, sizeof(BuildState), cudaMemcpyHostToDevice, s));
    VCHECK(cudaMemcpyAsync(d_queue, root_task, sizeof(BuildTask), cudaMemcpyHostToDevice, s));
    VCHECK(cudaMemcpyAsync(d_ready, one, sizeof(int), cudaMemcpyHostToDevice, s));
    BuildArgs ba{};
    ba.key = d_key;
    ba.order[0] = d_ord0; ba.order[1] = d_ord1;
    ba.tidx = d_tidx; ba.nodes = d_nodes; ba.queue = d_queue; ba.ready = d_ready; ba.st = d_build;
    ba.n = T; ba.queue_cap = max_nodes;
    const int ctas = (int)std::min<long long>(148, T / (kSubtree / 2) + 1);
    bvh_build_kernel<<<ctas, kBuildThreads, 0, s>>>(ba);
    VCHECK(cudaGetLastError());
    VCHECK(cudaMemcpyAsync(h_build, d_build, sizeof(BuildState), cudaMemcpyDeviceToHost, s));
    VCHECK(cudaMemcpyAsync(h_root, d_nodes, sizeof(BvhNode), cudaMemcpyDeviceToHost, s));
    VCHECK(cudaStreamSynchronize(s));
    if (h_build->error) VCHECK(host_tree());
    for (int a = 0; a < 3; ++a) {  // the mesh bounds are the root's box
      bmin[a] = h_root->lo[a];
      bmax[a] = h_root->hi[a];
    }
  }
  {
    // a bound outside the int range (or NaN) converts to INT_MIN and wraps, as x86 does it
    auto to_int = [](double v) { return v >= -2147483648.0 && v < 2147483648.0 ? (int)v : INT_MIN; };
    auto add = [](int v, int d) { return (int)((uint32_t)v + (uint32_t)d); };
    auto lo = [&](double v) { return add(to_int(std::floor(v)), -1); };
    auto hi = [&](double v) { return add(to_int(std::ceil(v)), 1); };
    L.w[0] = std::max(0, lo((bmin[0] - L.ox) / h));
    L.w[1] = std::min(nx - 1, hi((bmax[0] - L.ox) / h));
    L.w[2] = std::max(0, lo((bmin[1] - L.oy) / h));
    L.w[3] = std::min(ny - 1, hi((bmax[1] - L.oy) / h));
    L.w[4] = std::max(0, lo((bmin[2] - L.oz) / h));
    L.w[5] = std::min(nz - 1, hi((bmax[2] - L.oz) / h));
  }
  long long brows = 0;
  int sx0 = 0, sy0 = 0, sz0 = 0, wx = 0, wy = 0;
  unsigned bgrid = 0;
  for (;;) {
    if (T > 0) {
      // STEP 1 (window may be empty when the mesh lies outside the lattice)
      const long long rows = ((long long)L.w[3] - L.w[2] + 1) * ((long long)L.w[5] - L.w[4] + 1);
      if (L.w[0] <= L.w[1] && L.w[2] <= L.w[3] && L.w[4] <= L.w[5] && rows > 0) {
        scan_fill_kernel<<<(unsigned)((rows + kScanWarps - 1) / kScanWarps), kScanWarps * 32, 0, s>>>(bv, L, g->flags, d_solid, d_err);
        VCHECK(cudaGetLastError());
      }
      // STEP 2
      sx0 = std::max(0, L.w[0] - 1); sy0 = std::max(0, L.w[2] - 1); sz0 = std::max(0, L.w[4] - 1);
      // cells along each axis of the window +-1, none when the mesh lies outside the lattice
      // along any of them; bounds that leave the int range can make a count wrap, which is
      // refused unless another axis leaves the window empty
      const long long cx = std::min<long long>(nx - 1, (long long)L.w[1] + 1) - sx0 + 1,
                      cy = std::min<long long>(ny - 1, (long long)L.w[3] + 1) - sy0 + 1,
                      cz = std::min<long long>(nz - 1, (long long)L.w[5] + 1) - sz0 + 1;
      const auto none = [](long long n) { return n <= 0 && n >= INT_MIN; };
      const bool empty = none(cx) || none(cy) || none(cz);
      if (!empty && (cx < INT_MIN || cy < INT_MIN || cz < INT_MIN)) {
        *err = "voxelizer: the mesh's bounds are out of range of the lattice's cell indices";
        return -3;
      }
      brows = empty ? 0 : cy * cz;
      wx = (int)cx;
      wy = (int)cy;
      if (brows > 0) {
        bgrid = (unsigned)((brows * 32 + 255) / 256);
        boundary_rows_kernel<<<bgrid, 256, 0, s>>>(g->flags, L, sx0, sy0, sz0, wx, wy, brows, d_rows, nullptr, nullptr, nullptr);
        VCHECK(launch_scan_rows(d_rows, brows, w->host, s));
      }
    }
    // (the error word follows the count on both sides)
    VCHECK(cudaMemcpyAsync(h_solid, d_solid, sizeof(unsigned long long) + sizeof(int), cudaMemcpyDeviceToHost, s));
    VCHECK(cudaStreamSynchronize(s));
    if (!(*h_err & VOX_NAN_HITS)) break;  // the kernel does not set it in a tree of the host
    VCHECK(host_tree());
    VCHECK(cudaMemsetAsync(g->flags, 0, N, s));
    VCHECK(cudaMemsetAsync(counters, 0, 16, s));  // d_solid, d_err
  }
  const long long B = (long long)*total;
  g->B = B;
  g->solid = (long long)*h_solid;
  VCHECK(grid_lists(g, B));
  if (B > 0) {
    boundary_rows_kernel<<<bgrid, 256, 0, s>>>(g->flags, L, sx0, sy0, sz0, wx, wy, brows, nullptr, d_rows, g->bcells, g->bmap);
    // STEP 3
    q_links_kernel<<<(unsigned)((B + kLinkCells - 1) / kLinkCells), kLinkThreads, 0, s>>>(bv, L, g->flags, g->bcells, B, g->q,
                                                                                      g->minq, d_err);
    VCHECK(cudaGetLastError());
  }
  VCHECK(cudaMemcpyAsync(h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, s));
  VCHECK(cudaStreamSynchronize(s));
  if (*h_err) {
    *err = (*h_err & VOX_ERR_STACK) ? "voxelizer: BVH deeper than the 64-entry traversal stack"
                                    : "voxelizer: more than 128 hits on one scanline";
    return -4;
  }
  g->window[0] = L.w[0]; g->window[1] = L.w[1]; g->window[2] = L.w[2];
  g->window[3] = L.w[3]; g->window[4] = L.w[4]; g->window[5] = L.w[5];
  g->vox_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return 0;
}

}  // namespace aerosim
