// The two-cells-per-thread step of a single lattice (pair_kernel) and the item loop it
// shares with the batched step: FP32 arithmetic, with MLP the learned closure as warp tiles,
// rows of 4 and more cells (a batch: of an even count).  With ODD the pairs cover cells
// 0 .. nx-2 and the outlet cell nx-1 follows the last of them.
//
// A work item is R consecutive x-rows; its pairs of cells form one list, and each consumer
// warp takes chunks of 32 consecutive pairs of it, across row ends, dealt cyclically (the
// dealing goes on where the previous item stopped).  So every lane has a pair whatever the
// row length: the loop this replaces gave a warp 64 cells of one row, which left 2 of 8
// warps without rows at 192 cells and a quarter of the lanes idle at 140.  Slots of the
// shared-memory ring have the layout of the row blocks in memory, so one 32-bit offset per
// lane addresses both, and what a warp needs to know of a row (is it a wall?) is a byte the
// producer leaves beside it.  A chunk of plain fluid (one vote) has no per-cell tests.
//
// What bounds it (ncu, 256x128x128): with 16-bit storage issue and fixed latencies at 20 warps
// per SM (36.7 M warp instructions, 2.35 of 4 per cycle, DRAM 53 %), with FP32 DRAM (72 % cold,
// 0.97 of the copy peak in a run of steps).  Microseconds per step, before -> with this kernel:
// 256x128x128 F16S 68.5 -> 58.2, BF16S 69.5 -> 58.5, F16C 73.1 -> 63.6, FP32 101.6 -> 101.0;
// 160x80x80 F16S 28.2 -> 21.3; 200x100x96 F16S 43.1 -> 36.4; 128x64x64 FP32 20.3 -> 16.5;
// 64x32x32 FP32 11.4 -> 9.3; 191x95x97 (one cell per thread before) BF16S 43.8 -> 33.8, FP32
// 58.4 -> 50.1.  What made the difference: the bulk copies issued by one elected
// lane from uniform registers, 37 an item of 4 rows (by 32 lanes they are replayed one by one,
// about 20 instructions each, and the producer warp was the limit: 63.5 us), the flat pair
// list (the row ends on a helper warp were 6 M of 44 M instructions, on the critical path) and
// the near-wall cells at the start of the step, while the ring fills.  Not kept: 14 to 19
// consumer warps in one CTA per SM (93-96 us: one producer cannot feed an SM); a tail of
// one-row items (59.5 us here, but 9.7 -> 10.3 at 64x32x32).
#pragma once
#include "lbm_kernels.cuh"

namespace aerosim {

constexpr int kMaxPairRows = 16;  // rows per item
constexpr int kPairWarps = 9;                // consumer warps
constexpr int kPairProducer = kPairWarps;    // and the producer
constexpr int kPairThreads = (kPairWarps + 1) * 32;

// ceil(2^32 / d): n / d = umulhi(n, magic) for n d < 2^32 (pairs of an item: n < 2^16)
__host__ __device__ inline uint32_t pair_magic(int d) { return (uint32_t)((0x100000000ull + (uint32_t)d - 1) / (uint32_t)d); }

// Rows per item: about `pairs` pairs, and not so many that some CTAs get no item.
__host__ inline int pair_rows(int nx, long long rows, int pairs, long long ctas) {
  int r = pairs / (nx / 2);
  const long long share = (rows + ctas - 1) / ctas;
  if (r > share) r = (int)share;
  return r < 1 ? 1 : (r > kMaxPairRows ? kMaxPairRows : r);
}

// Dynamic shared memory: a guard (a pull of cell 0's or nx-1's outer neighbour reads past
// the row); the ring slots (R row blocks, then their class bytes); a guard; the barriers; the
// inlet tables; the direction table of the row ends, a scratch row per consumer warp, the
// directions' slots; per slot the rows' wall flags; the closure's weights, biases and a staging
// block per consumer warp.
constexpr int kEndScratch = 23;
__host__ __device__ inline size_t pair_smem_bytes(int pitch, int ny, int rows, int stages, size_t elem, bool mlp = false) {
  return kSmemGuard + (size_t)stages * rows * pitch * (19 * elem + 1) + kSmemGuard + 16 * (size_t)stages +
         2 * (size_t)ny * sizeof(double) + 19 * sizeof(float4) + kPairWarps * kEndScratch * sizeof(float) + 19 +
         (size_t)stages * rows + 16 + (mlp ? 16 + (kMlpFragWords * 32 + kMlpBias + kPairWarps * 128) * 4 : 0);
}

// p rounded up to 16 bytes, by its offset in the (aligned) shared memory: going through an
// integer would leave the compiler with generic loads.
__device__ __forceinline__ unsigned char* align16(unsigned char* base, void* p) {
  return base + (((uint32_t)(static_cast<unsigned char*>(p) - base) + 15u) & ~15u);
}

// What a consumer warp needs of an item beyond its slot.
template <class T>
struct PairItem {
  T* dst;           // destination of the item's first row block
  int r0, nr;       // first row, rows
  int nx, np, pitch;
  uint32_t magic;   // pair_magic(np)
  int ny, nz, ground_no_slip, write_macro;
  float tau0, k_smag;
  float2 dec;
};

// The row ends of a chunk (:323-371), lane-transposed: lane d writes direction d of the inlet
// cell 0 or the outlet cell nx-1, one end after the other, after a __syncwarp that orders it
// behind the lanes' own stores (in a plain chunk a row end's lane stores its pair as if both
// cells were its own).  Sources: the density of cell 1, or the post-collision, pre-wall cell nx-2, staged in
// the warp's scratch row xo.  Near-wall sources defer the end to the near-wall pass.
struct EndTables {
  const float4* dcw;    // direction table (c_x, c_y, c_z, w)
  const uint8_t* dslot;
  float* xo;            // the warp's scratch row
};
template <class S, bool ODD, class InletFn>
__device__ __forceinline__ void chunk_ends(const float2 (&v)[19], float2 r, float2 ux, float2 uy, float2 uz, bool lo, bool hi,
                                           uint32_t cls2 /* of the pair and, nx odd, of cell nx-1 */, int yy,
                                           typename S::T* dst, int pitch, int nx, int ny, int r0, bool write_macro,
                                           const StepArgs& m, const EndTables& e, InletFn inlet, int lane,
                                           long long& my_sum, int& my_nan) {
  using T = typename S::T;
  for (unsigned left = __ballot_sync(0xffffffffu, lo || hi); left; left &= left - 1) {
    const int src = __ffs(left) - 1;
    const bool is_hi = __shfl_sync(0xffffffffu, (int)hi, src) != 0;
    const int cls3 = __shfl_sync(0xffffffffu, (int)cls2, src), ry = __shfl_sync(0xffffffffu, yy, src);
    // the end's class and its neighbour's
    const int ce = (is_hi ? (ODD ? cls3 >> 16 : cls3 >> 8) : cls3) & 0xff,
              cn = (is_hi ? (ODD ? cls3 >> 8 : cls3) : cls3 >> 8) & 0xff;
    const bool solid_n = (cn & CLS_FLAG_MASK) == CELL_SOLID;
    if ((ce & CLS_FLAG_MASK) == CELL_SOLID || ((cn & CLS_NEAR) && !solid_n)) continue;
    T* const blk = dst + ry * (19 * pitch);
    const int sl = lane < 19 ? e.dslot[lane] : 0;
    const float4 cw = e.dcw[lane < 19 ? lane : 0];
    float rho, mx, my, mz = 0.0f, q;
    if (is_hi) {  // outlet (:354-371); a solid nx-2 gives what fDst holds there
      if (lane == src) {
#pragma unroll
        for (int d = 0; d < 19; ++d) e.xo[slot_of(d)] = ODD ? v[d].y : v[d].x;
        e.xo[19] = ODD ? r.y : r.x; e.xo[20] = ODD ? ux.y : ux.x;
        e.xo[21] = ODD ? uy.y : uy.x; e.xo[22] = ODD ? uz.y : uz.x;
      }
      __syncwarp();
      rho = end_rho(solid_n ? 1.0f : e.xo[19]);
      mx = solid_n ? 0.0f : e.xo[20]; my = solid_n ? 0.0f : e.xo[21]; mz = solid_n ? 0.0f : e.xo[22];
      const float prev = solid_n ? S::raw(blk[sl * pitch + nx - 2]) : e.xo[sl];
      q = outlet_blend(prev, end_eq<S>(dot_lane(cw, mx, my, mz), cw.w, rho, end_A(rho, mx, my, mz)));
    } else {  // inlet (:328-352); a solid cell 1 has density 1 (:177)
      const float r1 = __shfl_sync(0xffffffffu, r.y, src);
      rho = end_rho(solid_n ? 1.0f : r1);
      const int iy = (r0 + ry) % ny;
      const double2 ui = inlet(iy);
      mx = (float)ui.x;
      my = (float)ui.y;
      q = end_eq<S>(dot_lane(cw, mx, my, 0.0f), cw.w, rho, end_A(rho, mx, my, 0.0f));
      __syncwarp();
    }
    if (lane >= 19) q = 0.0f;
    q = compensate_lanes<S>(q, lane);
    if (lane < 19) blk[sl * pitch + (is_hi ? nx - 1 : 0)] = S::store(q);
    if (is_hi) __syncwarp();  // the scratch row is free for the next end
    if (lane == 0) {
      if (rho == rho) my_sum += rho_fixed(rho);
      else my_nan = 1;
      if (write_macro) {
        const long long ic = (long long)(r0 + ry) * nx + (is_hi ? nx - 1 : 0);
        m.mux[ic] = mx; m.muy[ic] = my; m.muz[ic] = mz; m.mrho[ic] = rho;
      }
    }
  }
}

// One consumer warp's chunks of an item: pull, release of the slot after the last pull,
// collision, stores, density sum, row ends.  (After the release only registers may be used:
// the next fill overwrites the slot and the rows' flags.)  Near-wall cells are left to the
// near-wall pass, solids are never written.
template <class S, int P, bool ODD = false, bool MLP = false, class InletFn>
__device__ __forceinline__ void pair_item(const PairItem<typename S::T>& it, const StepArgs& m, const typename S::T* slot,
                                          const uint8_t* cls, const uint8_t* wall, int first, uint64_t* empty,
                                          const EndTables& ends, InletFn inlet, int lane, long long& my_sum,
                                          int& my_nan, const PairMlp* mlp = nullptr) {
  using T = typename S::T;
  constexpr bool FUSE = ODD || MLP;  // the arithmetic of the one-cell kernels
  const int pitch = P ? P : it.pitch;
  const int total = it.nr * it.np;
  for (int base = first * 32; base < total; base += kPairWarps * 32) {
    const int p = min(base + lane, total - 1);
    const int yy = (int)__umulhi((uint32_t)p, it.magic);
    const int x0 = 2 * (p - yy * it.np);
    const bool act = base + lane < total;
    const int off = yy * (19 * pitch) + x0;
    const T* const sp = slot + off;
    const uint32_t cls2 = *reinterpret_cast<const uint16_t*>(cls + yy * pitch + x0);
    const bool wall_row = wall[yy] != 0;
    // the row ends: cell 0 in its pair; cell nx-1 in its pair (nx even) or after the last
    // pair, which then ends with its source nx-2 (nx odd)
    const bool lo = act && x0 == 0, hi = act && x0 + (ODD ? 3 : 2) == it.nx;
    const uint32_t end_cls = ODD ? cls[yy * pitch + it.nx - 1] : 0u;
    float2 v[19];
#pragma unroll
    for (int d = 0; d < 19; ++d) {  // pull-stream (lbmCpuReference.ts:189-231)
      const T* q = sp + slot_of(d) * pitch;
      if (cx_of(d) == 0) v[d] = load_pair<S>(q);
      else v[d] = make_float2(S::raw(q[-cx_of(d)]), S::raw(q[1 - cx_of(d)]));
    }
    if (base + kPairWarps * 32 >= total) {  // the warp's last pull of this slot: release it
      __syncwarp();
      if (lane == 0) mbar_arrive(empty);
    }
    float2 r, ux, uy, uz;
    collide_fast2<S, FUSE, MLP>(v, r, ux, uy, uz, it.tau0, it.k_smag, it.dec, mlp, cls2, lane);  // v: storage domain
    T* const out = it.dst + off;
    if (!__any_sync(0xffffffffu, act && ((cls2 & 0x0707u) != 0u || wall_row)) && !it.write_macro) {
      if (act) {
        if constexpr (S::kCompensate) {
          __half2 hv[19];
          compensate_pair<S, FUSE>(v, r, hv);
#pragma unroll
          for (int d = 0; d < 19; ++d) *reinterpret_cast<__half2*>(out + slot_of(d) * pitch) = hv[d];
        } else {
#pragma unroll
          for (int d = 0; d < 19; ++d) store_pair<S>(out + slot_of(d) * pitch, v[d]);
        }
        // a NaN density counts 0 in the sum (the conversion's result) and sets the flag
        const bool end1 = !ODD && hi;  // the pair's second cell is the outlet
        my_sum += (lo ? 0 : __float2int_rn(r.x * 33554432.0f)) + (end1 ? 0 : __float2int_rn(r.y * 33554432.0f));
        const float t = (lo ? 1.0f : r.x) + (end1 ? 1.0f : r.y);
        if (t != t) my_nan = 1;
      }
      if (__any_sync(0xffffffffu, lo || hi))
        chunk_ends<S, ODD>(v, r, ux, uy, uz, lo, hi, cls2 | (end_cls << 16), yy, it.dst, pitch, it.nx, it.ny, it.r0,
                           false, m, ends, inlet, lane, my_sum, my_nan);
      continue;
    }
    // the row ends first: the outlet reads cell nx-2 before any wall condition
    if (__any_sync(0xffffffffu, lo || hi))
      chunk_ends<S, ODD>(v, r, ux, uy, uz, lo, hi, cls2 | (end_cls << 16), yy, it.dst, pitch, it.nx, it.ny, it.r0,
                         it.write_macro, m, ends, inlet, lane, my_sum, my_nan);
    const int f0 = cls2 & CLS_FLAG_MASK, f1 = (cls2 >> 8) & CLS_FLAG_MASK;
    const bool own0 = act && f0 != CELL_SOLID && !(cls2 & CLS_NEAR) && !lo;
    const bool own1 = act && f1 != CELL_SOLID && !(cls2 & (CLS_NEAR << 8)) && (ODD || !hi);
    if (wall_row) {  // floor, ceiling, then sides (:375-429), fluid cells only
      const int row = it.r0 + yy, iz = row / it.ny, iy = row - iz * it.ny;
      if (iy == 0) {
        if (it.ground_no_slip) { ux = f2(0.0f); uz = f2(0.0f); }
        uy = f2(0.0f);
      }
      if (iy == it.ny - 1) uy = f2(0.0f);
      if (it.nz > 4 && (iz == 0 || iz == it.nz - 1)) uz = f2(0.0f);
      heq_pair<S, FUSE>(v, r, ux, uy, uz);
    }
    if constexpr (S::kCompensate) {
      __half2 hv[19];
      compensate_pair<S, FUSE>(v, r, hv);
      if (own0 && own1) {
#pragma unroll
        for (int d = 0; d < 19; ++d) *reinterpret_cast<__half2*>(out + slot_of(d) * pitch) = hv[d];
      } else if (own0 || own1) {
#pragma unroll
        for (int d = 0; d < 19; ++d) {
          if (own0) out[slot_of(d) * pitch] = __low2half(hv[d]);
          if (own1) out[slot_of(d) * pitch + 1] = __high2half(hv[d]);
        }
      }
    } else if (own0 && own1) {
#pragma unroll
      for (int d = 0; d < 19; ++d) store_pair<S>(out + slot_of(d) * pitch, v[d]);
    } else if (own0 || own1) {
#pragma unroll
      for (int d = 0; d < 19; ++d) {
        if (own0) out[slot_of(d) * pitch] = S::store(v[d].x);
        if (own1) out[slot_of(d) * pitch + 1] = S::store(v[d].y);
      }
    }
    if (own0) {
      if (r.x == r.x) my_sum += rho_fixed(r.x);
      else my_nan = 1;
    }
    if (own1) {
      if (r.y == r.y) my_sum += rho_fixed(r.y);
      else my_nan = 1;
    }
    if (it.write_macro && act) {
      const long long di = (long long)(it.r0 + yy) * it.nx + x0;
      if (f0 == CELL_SOLID) {  // solid macro (:173-179)
        m.mux[di] = 0.0f; m.muy[di] = 0.0f; m.muz[di] = 0.0f; m.mrho[di] = 1.0f;
      } else if (own0) {
        m.mux[di] = ux.x; m.muy[di] = uy.x; m.muz[di] = uz.x; m.mrho[di] = r.x;
      }
      if (f1 == CELL_SOLID) {
        m.mux[di + 1] = 0.0f; m.muy[di + 1] = 0.0f; m.muz[di + 1] = 0.0f; m.mrho[di + 1] = 1.0f;
      } else if (own1) {
        m.mux[di + 1] = ux.y; m.muy[di + 1] = uy.y; m.muz[di + 1] = uz.y; m.mrho[di + 1] = r.y;
      }
      if (ODD && hi && (end_cls & CLS_FLAG_MASK) == CELL_SOLID) {
        m.mux[di + 2] = 0.0f; m.muy[di + 2] = 0.0f; m.muz[di + 2] = 0.0f; m.mrho[di + 2] = 1.0f;
      }
    }
  }
}

// Coordinates of the row k rows after (iy, iz).
__device__ __forceinline__ int2 row_after(int iy, int iz, int k, int ny) {
  for (iy += k; iy >= ny; iy -= ny) ++iz;
  return make_int2(iy, iz);
}
// The producer's note on a row: whether a wall condition holds there.
__device__ __forceinline__ uint8_t wall_flag(int iy, int iz, int ny, int nz) {
  return iy == 0 || iy == ny - 1 || (nz > 4 && (iz == 0 || iz == nz - 1));
}

// One thread of a converged warp (the same one each time): its bulk copies take their
// operands from uniform registers, where copies issued by several lanes are replayed lane by
// lane.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}" : "=r"(p));
  return p != 0;
}

// The producer warp's fill of a ring slot with rows r0 .. r0 + nr - 1: their source rows in
// direction groups, their class bytes and wall flags.  publish() runs in one lane, before the
// slot can complete.
template <class T, class Publish>
__device__ __forceinline__ void pair_fill(int lane, const T* fs, const uint8_t* cls, int r0, int nr, int ny, int nz, int pitch,
                                          T* sp, uint8_t* sc, uint8_t* wall, uint64_t* full, Publish publish) {
  const uint32_t slot_bytes = (uint32_t)(pitch * sizeof(T));
  const int iz0 = r0 / ny, iy0 = r0 - iz0 * ny;
  if (lane < nr) {
    const int2 yz = row_after(iy0, iz0, lane, ny);
    wall[lane] = wall_flag(yz.x, yz.y, ny, nz);
  }
  __syncwarp();
  if (elect_one()) {
    publish();
    mbar_arrive_expect_tx(full, (uint32_t)nr * (19u * slot_bytes + (uint32_t)pitch));
    bulk_load(sc, cls + (long long)r0 * pitch, (uint32_t)(nr * pitch), full);
  }
  if (iy0 > 0 && iy0 + nr < ny && iz0 > 0 && iz0 < nz - 1) {
    // no clamped source: the nine source rows of a row lie at fixed distances from it
    if (elect_one()) {
      const long long plane = (long long)ny * (19 * pitch);  // elements between rows of neighbouring iz
      const T* src = fs + (long long)r0 * (19 * pitch);
      T* dst = sp;
      for (int yy = 0; yy < nr; ++yy, src += 19 * pitch, dst += 19 * pitch) {
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
          bulk_load(dst + group_first(g) * pitch, src + (group_first(g) * pitch - group_cy(g) * (19 * pitch) - group_cz(g) * plane),
                    (uint32_t)group_count(g) * slot_bytes, full);
      }
    }
  } else {
    // copy c: row yy = c / 9, direction group g = c % 9
    __syncwarp();  // after the expected bytes
    for (int c = lane; c < nr * kGroups; c += 32) {
      const int yy = c / kGroups, g = c - yy * kGroups;
      const int2 yz = row_after(iy0, iz0, yy, ny);
      const long long sr =
          clampi(yz.x - group_cy(g), 0, ny - 1) + (long long)ny * clampi(yz.y - group_cz(g), 0, nz - 1);
      const int first = group_first(g);
      bulk_load(sp + (size_t)(yy * 19 + first) * pitch, fs + (sr * 19 + first) * pitch,
                (uint32_t)group_count(g) * slot_bytes, full);
    }
  }
  __syncwarp();
}

// The lanes' direction table of the row ends.
__device__ __forceinline__ void fill_end_tables(float4* dcw, uint8_t* dslot) {
  if (threadIdx.x < 19) {
#pragma unroll
    for (int d = 0; d < 19; ++d)
      if (d == (int)threadIdx.x) {
        dcw[d] = make_float4((float)cx_of(d), (float)cy_of(d), (float)cz_of(d), wf_of(d));
        dslot[d] = (uint8_t)slot_of(d);
      }
  }
}

// One time step of one lattice: a producer warp fills the ring, the consumer warps first take
// their near-wall cells, while the first slots fill, and then the chunks of the items; the
// last CTA takes the rescale decision.
template <class S, int P, bool ODD = false, bool MLP = false>
__global__ void __launch_bounds__(kPairThreads, 2) pair_kernel(const __grid_constant__ StepArgs a) {
  using T = typename S::T;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ long long red[kPairWarps + 1];
  __shared__ int nan_flag;
  __shared__ int s_first[8];  // first row of the item in ring slot s (-1: none left)

  const int nx = a.L.nx, ny = a.L.ny, nz = a.L.nz;
  const int pitch = P ? P : a.L.pitch;
  const int S_ = a.stages, R = a.item_rows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = ny * nz;
  const int n_items = (rows + R - 1) / R;
  // Odd steps take the items last to first: a step then begins on the rows the step before
  // wrote last, while they are still in L2.  Every cell's update reads only the source
  // lattice and the density sums are fixed-point, so the order changes no result.
  const bool reverse = (a.step_index & 1) != 0;

  T* const spop = reinterpret_cast<T*>(smem_raw + kSmemGuard);
  uint8_t* const scls = smem_raw + kSmemGuard + (size_t)S_ * R * 19 * pitch * sizeof(T);
  // (the class bytes end on a multiple of 32)
  uint64_t* const full = reinterpret_cast<uint64_t*>(scls + (size_t)S_ * R * pitch + kSmemGuard);
  uint64_t* const empty = full + S_;
  double* const s_uxi = reinterpret_cast<double*>(empty + S_);
  double* const s_uyi = s_uxi + ny;
  float4* const s_dcw = reinterpret_cast<float4*>(align16(smem_raw, s_uyi + ny));          // [19]
  float* const s_xo = reinterpret_cast<float*>(s_dcw + 19);                                // [kPairWarps][kEndScratch]
  uint8_t* const s_dslot = reinterpret_cast<uint8_t*>(s_xo + kPairWarps * kEndScratch);    // [19]
  uint8_t* const s_wall = s_dslot + 19;                                                    // [S_][R]

  uint32_t* const s_mfrag = reinterpret_cast<uint32_t*>(align16(smem_raw, s_wall + S_ * R));  // [24 * 32]
  float* const s_mbias = reinterpret_cast<float*>(s_mfrag + kMlpFragWords * 32);   // [kMlpBias]
  uint32_t* const s_mstage = reinterpret_cast<uint32_t*>(s_mbias + kMlpBias);      // [kPairWarps][128]
  if constexpr (MLP) {
    for (int i = threadIdx.x; i < kMlpFragWords * 32; i += blockDim.x) s_mfrag[i] = a.mlp_frag[i];
    for (int i = threadIdx.x; i < kMlpBias; i += blockDim.x) s_mbias[i] = a.mlp_bias[i];
  }

  const T* const fs = static_cast<const T*>(a.fsrc);
  T* const fd = static_cast<T*>(a.fdst);
  const int cur_slot = a.step_index & 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S_; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kPairWarps);
    }
    nan_flag = 0;
    mbar_fence_init();
  }
  fill_end_tables(s_dcw, s_dslot);
  // inlet velocity per iy (:334-342)
  for (int i = threadIdx.x; i < ny; i += blockDim.x) {
    double uxi = a.u_inlet;
    if (a.ground_no_slip) uxi = a.u_inlet * a.abl[i];
    double uyi = 0.0;
    if (a.step_index < 120) uyi = 0.015 * a.u_inlet * a.sin_tab[(long long)a.step_index * ny + i];
    s_uxi[i] = uxi;
    s_uyi[i] = uyi;
  }
  __syncthreads();
  // Programmatic dependent launch: everything above wrote only shared memory and read only
  // inputs the host copied in; wait for the previous step, then let the next one's CTAs in.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  long long my_sum = 0;
  int my_nan = 0;
  bool failed = false;
  const int stride_first = (int)gridDim.x;

  if (warp == kPairProducer) {
    int issued = 0;
    int end_slot = -1;  // the slot that took the end mark
    int s = 0;
    uint32_t ph = 0;  // parity of the slot's current fill
    for (int j = 0;; ++j) {
      int k;  // this fill's item
      if (a.dynamic_items) {  // from the step's counter
        unsigned int t = 0;
        if (lane == 0) t = atomicAdd(&a.st->next_item[cur_slot], 1u);
        t = __shfl_sync(0xffffffffu, t, 0);
        k = t < (unsigned)n_items ? (int)t : -1;
      } else {  // round-robin
        const long long t = blockIdx.x + (long long)j * stride_first;
        k = t < n_items ? (int)t : -1;
      }
      const int r0 = k < 0 ? -1 : (reverse ? n_items - 1 - k : k) * R;
      if (j >= S_) {  // the slot's previous fill must have been consumed
        const bool ok = mbar_wait(&empty[s], ph ^ 1u, a.wait_limit);
        if (!__any_sync(0xffffffffu, ok)) {
          failed = true;
          break;
        }
      }
      if (r0 < 0) {  // no items left: the other warps leave when they reach this slot
        if (lane == 0) {
          s_first[s] = -1;
          mbar_arrive(&full[s]);
        }
        end_slot = s;
        break;
      }
      const int nr = min(rows - r0, R);
      pair_fill(lane, fs, a.cls, r0, nr, ny, nz, pitch, spop + (size_t)s * R * 19 * pitch, scls + (size_t)s * R * pitch,
                s_wall + s * R, &full[s], [&] { s_first[s] = r0; });
      issued = j + 1;
      if (++s == S_) { s = 0; ph ^= 1u; }
    }
    if (failed && lane == 0) atomicOr(&a.st->error, STEP_ERR_PIPELINE_TIMEOUT);
    // no copy may still be in flight when the CTA exits (see main_kernel)
    if (lane == 0) {
      for (int k = 0; k < S_ && k < issued; ++k) {
        if (k == end_slot) continue;
        const int last = k + ((issued - 1 - k) / S_) * S_;
        mbar_wait(&full[k], (uint32_t)((last / S_) & 1), kWaitLimit);
      }
    }
  } else {
    const int pslot = (a.step_index + 1) & 1;  // pending rescale of the previous step
    const double corr = a.st->apply[pslot] ? a.st->corr[pslot] : 1.0;
    auto inlet = [&](int y) { return make_double2(s_uxi[y], s_uyi[y]); };
    constexpr int kForm = S::kCompensate && (ODD || MLP) ? 2 : (sizeof(T) == 2 || ODD || MLP) ? 1 : 0;
    for (long long t = ((long long)warp * gridDim.x + blockIdx.x) * 32 + lane; t < a.n_near;
         t += (long long)gridDim.x * (kPairWarps * 32))
      my_sum += near_cell<S, MODE_FAST, P, kForm>(a, a.fsrc, a.fdst, a.write_macro, t, corr, inlet, &my_nan);
    const float corrf = (float)corr;
    PairItem<T> it;
    it.nx = nx; it.np = nx / 2; it.pitch = pitch; it.magic = a.pair_magic;
    it.ny = ny; it.nz = nz; it.ground_no_slip = a.ground_no_slip; it.write_macro = a.write_macro;
    it.tau0 = (float)a.tau0; it.k_smag = (float)a.k_smag;
    it.dec = make_float2(corrf * S::kRawScale, corrf - 1.0f);  // raw-moment decode
    const EndTables ends{s_dcw, s_dslot, s_xo + warp * kEndScratch};
    const PairMlp mlp{s_mfrag, s_mbias, s_mstage + warp * 128, a.mlp_nu0};
    int s = 0;
    uint32_t ph = 0;
    int deal = warp;  // this warp's first chunk of the item
    for (;;) {
      const bool ok = mbar_wait(&full[s], ph, a.wait_limit);
      if (!__any_sync(0xffffffffu, ok)) {
        failed = true;
        break;
      }
      it.r0 = s_first[s];
      if (it.r0 < 0) break;
      it.nr = min(rows - it.r0, R);
      it.dst = fd + (long long)it.r0 * (19 * pitch);
      const int chunks = (it.nr * it.np + 31) >> 5;
      if (deal < chunks) {
        pair_item<S, P, ODD, MLP>(it, a, spop + (size_t)s * R * 19 * pitch, scls + (size_t)s * R * pitch, s_wall + s * R, deal,
                                  &empty[s], ends, inlet, lane, my_sum, my_nan, &mlp);
      } else {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
      }
      deal -= chunks % kPairWarps;  // the dealing goes on where this item stopped
      if (deal < 0) deal += kPairWarps;
      if (++s == S_) { s = 0; ph ^= 1u; }
    }
    if (__any_sync(0xffffffffu, my_nan) && lane == 0) nan_flag = 1;
    if (failed && lane == 0) atomicOr(&a.st->error, STEP_ERR_PIPELINE_TIMEOUT);
  }

#pragma unroll
  for (int o = 16; o > 0; o >>= 1) my_sum += __shfl_down_sync(0xffffffffu, my_sum, o);
  if (lane == 0) red[warp] = my_sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long s = 0;
    for (int w = 0; w <= kPairWarps; ++w) s += red[w];
    if (nan_flag) a.st->nan_seen = 1;
    finish_step(a, s);
  }
}

}  // namespace aerosim
