// Transport sweep (short characteristics) and the coupled radiation-hydro step.
//
// The reference sweeps every direction on the CPU in the order of a precomputed
// graph (sorted_graph: (cell, out-face) pairs) with precomputed node distances
// (vec_x0), solvers/illum/src/mpi/multi_gpu/illum_multi_gpu_face_calc.cpp:91-190.
// Here the order is built on the device once per mesh and direction set as
// levels per direction: level 0 holds the cells whose in-faces are all on the
// boundary, level L+1 those whose last upwind neighbour is in level L.  A sweep
// is one kernel: a CTA per direction, or a cluster of them where directions are few and their
// fronts wide, walks its direction's levels, one thread per cell and a barrier between levels.
//
// One value per cell.  The reference gives every out-face the mean over its three
// interpolation nodes of the intensity traced back from the node to the in-face it
// came through: the in-face h with the smallest t_h = lam_h r_h (r_h = H_h / -cos_h,
// H_h the height of the cell over face h, lam_h the node's barycentric weight of the
// vertex opposite h: 2/3 at the node's own vertex, 1/6 at the others).  Let b1 be the
// in-face with the smallest r / 6 and b2 the next.  A node of a vertex v other than b1's
// sees t = r_b1 / 6 at b1 and at least min(2/3 r_v, r / 6) >= r_b1 / 6 elsewhere, so it is
// traced to b1; only the node at b1's own vertex compares 2/3 r_b1 with r_b2 / 6.  A face j
// holds the nodes of the three vertices other than j, and an out-face is not b1, so every
// out-face holds the special node and two ordinary ones: all out-faces of a cell carry the
// SAME value, (A + A + B) / 3.  The sweep therefore keeps one outgoing value per (cell,
// direction), two attenuations at most, and forms the cell value (ReCalcIllumOpt, an
// area-weighted face mean) in the same thread from the in-face values and that one value.
//
// A cell's outgoing value lives from its level to the last level of its downwind
// neighbours; the plan gives it a slot for that time (a free list per direction), so a
// direction needs about as many slots as its front is wide (9,400 on the 48^3 x 6 mesh)
// and no face-value array exists.  Slots sit in shared memory when they fit, else (or where
// a cluster shares them) in a per-direction array that stays in L2.
//
// What a thread reads of its item comes in sweep order: a 16-byte record (cell, face
// choice, slots) and, where memory holds them, the two distances and the weights; by cell index
// it reads the source record of the step and the scattering integral.
// Compiled with --fmad=false: in double precision every value is the oracle's operation
// for operation, but for exp, exp(-4x) = exp(-x)^4 and the order of the face sums.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <cub/device/device_radix_sort.cuh>
#include <type_traits>
#include <vector>

#include "coupled.h"
#include "ctx.h"
#include "dirs.h"
#include "hydro_phys.cuh"
#include "rad_phys.cuh"
#include "rrhd_internal.h"

using namespace rrhd;

namespace {

// Per-cell geometry record (RW words), read by the plan and, in a sweep without the
// distance stream, by every item: 0-11 outward normals n_j, 12-15 heights H_j, then the
// neighbours (4 x int32, -1 on the boundary).
template <class T>
struct Rec {
  static constexpr int NBR = 16;                        // word offset of the neighbours
  static constexpr int RW = 16 + 16 / (int)sizeof(T);  // words: 144 B in double, 80 B in float
};
// Per-cell source record (SW words): {k, betta/k, alpha Q_g/k}, one Q for all groups where
// they share it (the coupled step).  In float with one or two groups the cell's weights follow at
// word kSrcW: an item's record and weights are one 32-byte access.
constexpr int kSrcQ = 2, kSrcW = 4;
template <class T>
constexpr bool weights_in_record(int G) {
  return sizeof(T) == 4 && (G == 1 || G == 2);
}
template <class T>
constexpr int source_words(int G, bool one_q) {
  return weights_in_record<T>(G) ? 8 : one_q ? 4 : (kSrcQ + G + 3) / 4 * 4;
}

template <class T>
__device__ __forceinline__ void load_vec(const T *r, T *g, int n) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int q = 0; q < n; q += V) {
    if constexpr (sizeof(T) == 8) {
      const double2 v = __ldg(reinterpret_cast<const double2 *>(r) + q / 2);
      g[q] = v.x;
      g[q + 1] = v.y;
    } else {
      const float4 v = __ldg(reinterpret_cast<const float4 *>(r) + q / 4);
      g[q] = v.x;
      g[q + 1] = v.y;
      g[q + 2] = v.z;
      g[q + 3] = v.w;
    }
  }
}
template <class T>
__device__ __forceinline__ void load_nbr(const T *r, int *nbr) {
  const int4 n = __ldg(reinterpret_cast<const int4 *>(r + Rec<T>::NBR));
  nbr[0] = n.x, nbr[1] = n.y, nbr[2] = n.z, nbr[3] = n.w;
}

__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double ex(double x) { return exp(x); }
__device__ __forceinline__ float ex(float x) { return __expf(x); }
__device__ __forceinline__ double dv(double a, double b) { return a / b; }
__device__ __forceinline__ float dv(float a, float b) { return __fdividef(a, b); }

template <class T>
__device__ __forceinline__ void face_cos(const T *g, T wx, T wy, T wz, T *cosf) {
#pragma unroll
  for (int j = 0; j < 4; j++) cosf[j] = (g[3 * j] * wx + g[3 * j + 1] * wy) + g[3 * j + 2] * wz;
}

// Code word of an item:
//   bits 0-1, 2-3, 4-5  the in-faces (cos < 0) b1, b2 and the third, as far as there are
//   bits 6-7            their number (at most three: the four outward normals weighted by
//                       the face areas sum to zero)
//   bits 8-11           out-faces (cos > 0)
//   bit 12              the node at b1's vertex is traced to b2 (else to b1, lam = 2/3)
//   bit 13              the weights come from the cell: some face is neither (parallel to the
//                       direction), or the out-faces are small (out_weight)
constexpr uint32_t kCodeB2 = 1u << 12, kCodeCell = 1u << 13;

// Code word and distances of one (cell, direction) from the cell's normals and heights
// g[16]: tA = r_b1 / 6, tB = r_b2 / 6 (bit 12; else 0).  b1, b2: the smallest by (t, face
// index), as the restatement compares them; an equal 2/3 r_b1 = r_b2 / 6 goes to the lower
// face index.
template <class T>
__device__ __forceinline__ uint32_t item_geometry(const T *g, const T *cosf, T &tA, T &tB) {
  uint32_t out = 0;
  int b1 = -1, b2 = -1, n = 0, sum = 0;
  T tb1 = 0, tb2 = 0, rb1 = 0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (cosf[f] < 0) {
      const T r = dv(g[12 + f], -cosf[f]);
      const T t1 = (T)(1.0 / 6.0) * r;
      n++;
      sum += f;
      if (b1 < 0 || t1 < tb1) {
        b2 = b1;
        tb2 = tb1;
        b1 = f;
        tb1 = t1;
        rb1 = r;
      } else if (b2 < 0 || t1 < tb2) {
        b2 = f;
        tb2 = t1;
      }
    } else if (cosf[f] > 0) {
      out |= 1u << f;
    }
  }
  n = min(n, 3);  // four only on a mesh whose cells do not close
  tA = tb1;
  tB = (T)0;
  uint32_t code = out << 8 | (uint32_t)n << 6;
  if (n + __popc(out) != 4) code |= kCodeCell;
  if (n >= 1) code |= (uint32_t)b1;
  if (n >= 2) {
    code |= (uint32_t)b2 << 2;
    const T t4 = (T)(2.0 / 3.0) * rb1;
    if (!(t4 < tb2 || (t4 == tb2 && b1 < b2))) {
      code |= kCodeB2;
      tB = tb2;
    }
  }
  if (n >= 3) code |= (uint32_t)((sum - b1 - b2) & 3) << 4;
  return code;
}

// Weights of an item: w of the in-faces b1, b2 and the third (0 where there is none), wo of all
// out-faces together, from the cell's four (area_j / sum of the areas).  wo is the sum of the
// out-faces' weights: as one minus the others it would lose the digits of a small out-face, and
// with them the value of a cell that takes nothing from its in-faces.
template <class T>
__device__ __forceinline__ void item_weights(const T (&f)[4], uint32_t code, T (&w)[3], T &wo) {
  const int nin = (int)(code >> 6) & 3;
  const auto pick = [&](uint32_t j) { return j & 2 ? (j & 1 ? f[3] : f[2]) : (j & 1 ? f[1] : f[0]); };
  w[0] = nin > 0 ? pick(code & 3) : (T)0;
  w[1] = nin > 1 ? pick((code >> 2) & 3) : (T)0;
  w[2] = nin > 2 ? pick((code >> 4) & 3) : (T)0;
  wo = (T)0;
#pragma unroll
  for (int j = 0; j < 4; j++) wo += (code >> (8 + j)) & 1u ? f[j] : (T)0;
}

// In double the out-faces' weight is what the in-faces leave of one, so that the four sum to one and
// a smooth intensity does not feel their roundings (error of the cell values 2.46e-16 in the 2-norm,
// 2.52e-16 with each weight rounded by itself); the stream keeps the in-faces'.  It is good to 2^-52 / its
// size, so below 1/16 the item takes all from the cell (no item of the jittered Kuhn meshes is).
__device__ __forceinline__ double out_weight(const double (&w)[3]) { return (1.0 - w[0]) - (w[1] + w[2]); }
constexpr double kOutMin = 1.0 / 16.0;

// 32 bytes of global memory in one access (32-byte aligned)
__device__ __forceinline__ void ld_32(const double *p, double &a, double &b, double &c, double &d) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a), "=d"(b), "=d"(c), "=d"(d) : "l"(p) : "memory");
}
__device__ __forceinline__ void ld_32(const float *p, float &a, float &b, float &c, float &d, float (&e)[4]) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a), "=f"(b), "=f"(c), "=f"(d), "=f"(e[0]), "=f"(e[1]), "=f"(e[2]), "=f"(e[3])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void st_32(double *p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

__device__ __forceinline__ void ld_cell_weights(const double *p, double (&f)[4]) { ld_32(p, f[0], f[1], f[2], f[3]); }
__device__ __forceinline__ void ld_cell_weights(const float *p, float (&f)[4]) {
  const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
  f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
}

// G values at p (contiguous), vectorised for 2 and 4 groups; GMEM: p is in global memory,
// 32-byte aligned when the values are 32 bytes
template <bool GMEM, class T, int G>
__device__ __forceinline__ void ld_groups(const T *p, T (&v)[G]) {
  if constexpr (GMEM && sizeof(T) == 8 && G == 4) {
    ld_32(p, v[0], v[1], v[2], v[3]);
  } else if constexpr (sizeof(T) == 8 && G % 2 == 0) {
#pragma unroll
    for (int q = 0; q < G / 2; q++) {
      const double2 x = reinterpret_cast<const double2 *>(p)[q];
      v[2 * q] = x.x;
      v[2 * q + 1] = x.y;
    }
  } else if constexpr (sizeof(T) == 4 && G == 4) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
  } else {
#pragma unroll
    for (int q = 0; q < G; q++) v[q] = p[q];
  }
}
template <bool GMEM, class T, int G>
__device__ __forceinline__ void st_groups(T *p, const T (&v)[G]) {
  if constexpr (GMEM && sizeof(T) == 8 && G == 4) {
    st_32(p, v[0], v[1], v[2], v[3]);
  } else if constexpr (sizeof(T) == 8 && G % 2 == 0) {
#pragma unroll
    for (int q = 0; q < G / 2; q++) reinterpret_cast<double2 *>(p)[q] = make_double2(v[2 * q], v[2 * q + 1]);
  } else if constexpr (sizeof(T) == 4 && G == 4) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int q = 0; q < G; q++) p[q] = v[q];
  }
}

// T: records, slots and the transport arithmetic; S and I come and go as TI.
template <class T, class TI>
struct SweepArgs {
  int64_t N;
  int d0, G, SW;
  int qs;                   // 1: Q per group, 0: one for all
  const uint4 *ord;         // [M][N] items in sweep order {cell, code, own | in0 << 16, in1 | in2 << 16}
  const uint2 *ord_hi;      // [M][N] upper halves of the slots (WIDE)
  const T *dist;            // [M][N][2] {tA, tB} (GEO >= 1)
  const T *wgt, *wgt3;      // [M][N][2], [M][N] weights (GEO 2)
  const T *rec, *w, *wt;    // geometry records and directions (GEO 0), face weights [N][4]
  const int32_t *lvl;       // level offsets of every direction
  const int64_t *lvl_base;  // [M] first entry in lvl
  const int32_t *depth;     // [M] levels
  const T *src;             // [N][SW]
  T *slots;                 // [directions of the launch][nhigh][G]: slots from `cap` on
  uint32_t cap;             // slots in shared memory
  int cl;                   // CTAs a direction
  int64_t nhigh;
  const TI *S;              // S and I element (cell c, direction d0 + x, group g) at q * sc + x * sd + g,
  TI *I;                    // q the item's position in sweep order (by_pos) or its cell
  int64_t sc, sd;
  bool by_pos;
  T bc;
};

// Asks L2 for n bytes at p (both multiples of 16 after rounding p down).
template <class P>
__device__ __forceinline__ void bulk_prefetch(const P *p, uint32_t n) {
  const uint64_t b = reinterpret_cast<uint64_t>(p);
  const uint32_t skip = (uint32_t)(b & 15);
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(b - skip), "r"((n + skip) & ~15u) : "memory");
}

// One CTA (or cluster) per direction.  GT: compile-time group count (1, 2 or 4; S and I in the sweep's own
// layout), 0 for any other.  HIGH: slots from a.cap on are in global memory (the others in
// shared memory).  GEO: from the stream come 0 nothing (distances and weights from the cell's
// records), 1 the distances (weights from the cell's sector), 2 the weights as well (double).
// Slots 0 and 1 hold the boundary value and zero (for in-faces an item does not have); an item
// whose own slot is 0 has no downwind neighbour and writes none.
//
// Only the slot values depend on the levels before.  A thread loads the record and distances of
// its item after the next, and the source record of its next one, while it works on one item;
// one thread asks L2 for the streams' lines four CTA widths ahead.  What an SM can send of
// uncoalesced accesses (a request every few cycles when each misses L1) decides the rest: per
// item one 32-byte source record, and by cell also S and I.
// Measured (whole sweep with its copies; before: one launch per level of all directions, face
// values in HBM): 48^3 x 6 cells x 256 directions FP64, one group, 28.1 -> 5.0 ms; 12^3 x 6 x
// 64, 269 -> 84 us; coupled step's sweep 32^3 x 256 x 4 FP64 12.6 -> 3.9 ms, 48^3 x 256 x 4 mixed 37.0 -> 10.2.
// With every load from L1 it would take half of that: issue slots and the latency of the FP64
// chains at 16 warps an SM, and the wait at each level's barrier.
//
// CLUSTER: a.cl CTAs of a cluster share a direction's levels (few directions with long fronts);
// slots 2 and up are in global memory, where a level's values pass from CTA to CTA over the
// cluster barrier.
// A sweep in float with one group: 64 registers let two CTAs of 512 threads share an SM (14^3 x 6 cells
// x 256 x 1 0.30 ms, 0.50 with the 72 it would take; 36^3 x 128 x 1 1.42 and 1.53).
template <class T, int GT, bool HIGH, int NB>
constexpr int kResident = sizeof(T) == 4 && GT == 1 && !HIGH ? 2 : NB;
template <class T, class TI, int GT, bool HIGH, bool WIDE, int GEO, int NT, int NB, bool CLUSTER>
__global__ void __launch_bounds__(NT, (kResident<T, GT, HIGH, NB>)) k_sweep(const SweepArgs<T, TI> a) {
  extern __shared__ __align__(16) uint8_t sweep_smem[];
  constexpr int GR = GT > 0 ? GT : 1;
  constexpr bool WGT = GEO == 2;
  constexpr bool AHEAD = sizeof(T) == 4;  // the cell's weights an item ahead, where they take few registers
  const int cl = CLUSTER ? a.cl : 1, x = (int)blockIdx.x / cl, d = a.d0 + x;
  const int first = CLUSTER ? ((int)blockIdx.x - x * cl) * NT + (int)threadIdx.x : (int)threadIdx.x;  // in a level
  const int step = cl * NT, kAhead = 4 * step;
  const int G = GT > 0 ? GT : a.G;
  T *const low = reinterpret_cast<T *>(sweep_smem);
  T *const high = HIGH ? a.slots + (int64_t)x * a.nhigh * G : nullptr;
  auto get_slot = [&](uint32_t q, T (&v)[GR]) {
    if (HIGH && q >= a.cap)
      ld_groups<true>(high + (int64_t)(q - a.cap) * GR, v);
    else
      ld_groups<false>(low + q * GR, v);
  };
  auto slot = [&](uint32_t q) {
    if (HIGH && q >= a.cap) return high + (int64_t)(q - a.cap) * G;
    return low + q * (uint32_t)G;
  };
  const int64_t at = (int64_t)d * a.N;
  const uint4 *const ord = a.ord + at;
  const T *const dist = a.dist + 2 * at, *const wgt = a.wgt + 2 * at, *const wgt3 = a.wgt3 + at;
  const int32_t *lvl = a.lvl + a.lvl_base[d];
  const int depth = a.depth[d];
  const TI *const S = a.S + x * a.sd;
  TI *const I = a.I + x * a.sd;
  const char *const src = reinterpret_cast<const char *>(a.src);
  const uint32_t src_bytes = (uint32_t)(a.SW * (int)sizeof(T));
  const int N = (int)a.N;
  T wx = 0, wy = 0, wz = 0;
  if (!GEO) wx = a.w[3 * d], wy = a.w[3 * d + 1], wz = a.w[3 * d + 2];
  for (int g = threadIdx.x; g < 2 * G; g += NT) low[g] = g < G ? a.bc : (T)0;
  __syncthreads();

  struct Item {
    uint4 o;
    uint2 hi;
    T tA, tB;
    T k, bk, q0, q1;  // q1: of the second group where each has its own
    T cw[AHEAD ? 4 : 1];
  };
  auto load_record = [&](int i, Item &it) {
    it.o = __ldcs(ord + i);
    if constexpr (WIDE) it.hi = __ldcs(a.ord_hi + at + i);
    if constexpr (GEO) {
      if constexpr (sizeof(T) == 8) {
        const double2 t = __ldcs(reinterpret_cast<const double2 *>(dist) + i);
        it.tA = t.x, it.tB = t.y;
      } else {
        const float2 t = __ldcs(reinterpret_cast<const float2 *>(dist) + i);
        it.tA = t.x, it.tB = t.y;
      }
    }
  };
  auto load_cell = [&](Item &it) {
    const T *sr = reinterpret_cast<const T *>(src + (uint64_t)it.o.x * src_bytes);
    if constexpr (sizeof(T) == 8) {
      ld_32(sr, it.k, it.bk, it.q0, it.q1);
    } else if constexpr (weights_in_record<T>(GT)) {
      ld_32(sr, it.k, it.bk, it.q0, it.q1, it.cw);
    } else {
      const float4 t = __ldg(reinterpret_cast<const float4 *>(sr));
      it.k = t.x, it.bk = t.y, it.q0 = t.z, it.q1 = t.w;
      ld_cell_weights(a.wt + 4 * (uint64_t)it.o.x, it.cw);
    }
  };
  // one thread asks L2 for the streams' lines some levels ahead
  int fetched = 0;
  auto fetch = [&](int to) {
    to = min(to, N) & ~1;  // whole 16-byte pieces
    if (to <= fetched) return;
    const int64_t q = fetched;
    const uint32_t n = (uint32_t)(to - fetched);
    bulk_prefetch(ord + q, 16 * n);
    if (GEO) {
      bulk_prefetch(dist + 2 * q, 2 * (uint32_t)sizeof(T) * n);
    }
    if (WGT) {
      bulk_prefetch(wgt + 2 * q, 2 * (uint32_t)sizeof(T) * n);
      bulk_prefetch(wgt3 + q, (uint32_t)sizeof(T) * n);
    }
    if (a.by_pos && sizeof(TI) * G % 8 == 0) bulk_prefetch(S + (int64_t)fetched * G, (uint32_t)sizeof(TI) * G * n);
    fetched = to;
  };

  // this thread's items in order, two ahead of the one in work: position p in the level that
  // ends at p_hi (the next one at p_hi2); N when there are none left
  int p = first, p_lvl = 0, p_hi = lvl[1], p_hi2 = lvl[min(2, depth)];
  auto settle = [&]() {
    while (p >= p_hi && p_hi < N) {
      p = p_hi + first;
      p_lvl++;
      p_hi = p_hi2;
      p_hi2 = lvl[min(p_lvl + 2, depth)];
    }
  };
  Item it, next;
  settle();
  int i = p;
  if (p < N) {
    load_record(p, it);
    load_cell(it);
    p += step;
    settle();
    if (p < N) load_record(p, next);
  }
  int hi = lvl[1], hi2 = lvl[min(2, depth)];
  for (int L = 0; L < depth; L++) {
    if (first == 0) fetch(hi + kAhead);
    while (i < hi) {
      const Item now = it;
      const int at_i = i;
      const uint32_t iq = a.by_pos ? (uint32_t)i : now.o.x;
      i = p;
      it = next;
      if (p < N) {
        load_cell(it);
        p += step;
        settle();
        if (p < N) load_record(p, next);
      }
      const uint64_t c = now.o.x;
      const uint32_t code = now.o.y;
      T w[3], wo, cw[4];  // cw: the cell's weights, where there is no stream of them
      TI sv[GR];
      if constexpr (GT > 0) ld_groups<true>(S + (uint64_t)iq * (uint32_t)GT, sv);
      if constexpr (WGT) {
        const double2 u = __ldcs(reinterpret_cast<const double2 *>(wgt) + at_i);
        w[0] = u.x, w[1] = u.y;
        w[2] = __ldcs(wgt3 + at_i);
      } else if constexpr (AHEAD) {
#pragma unroll
        for (int q = 0; q < 4; q++) cw[q] = now.cw[q];
      } else {
        ld_cell_weights(a.wt + 4 * c, cw);
      }
      uint32_t own = now.o.z & 0xffffu, s0 = now.o.z >> 16, s1 = now.o.w & 0xffffu, s2 = now.o.w >> 16;
      if constexpr (WIDE) {
        own |= now.hi.x << 16;
        s0 |= now.hi.x & 0xffff0000u;
        s1 |= now.hi.y << 16;
        s2 |= now.hi.y & 0xffff0000u;
      }
      T tA, tB;
      if constexpr (GEO) {
        tA = now.tA, tB = now.tB;
      } else {
        T g[16], cosf[4];
        load_vec<T>(a.rec + c * Rec<T>::RW, g, 16);
        face_cos(g, wx, wy, wz, cosf);
        (void)item_geometry<T>(g, cosf, tA, tB);  // the code word is the plan's
      }
      const T k = now.k, bk = now.bk;
      const bool two = (code & kCodeB2) != 0;
      const T EA = ex(-k * tA);
      const T E2 = EA * EA, EX = ex(-k * tB);  // formed in any case: the two chains overlap
      const T EB = two ? EX : E2 * E2;
      T v0[GR], v1[GR], v2[GR];
      if constexpr (GT > 0) {  // asked for before the branch below
        get_slot(s0, v0);
        get_slot(s1, v1);
        get_slot(s2, v2);
      }
      if constexpr (!WGT) item_weights(cw, code, w, wo);
      if constexpr (sizeof(T) == 8) wo = out_weight(w);  // the same bits with and without the stream
      T par = (T)0;  // a face parallel to the direction holds the boundary value
      if (code & kCodeCell) {
        const int nin = (int)(code >> 6) & 3;
        uint32_t seen = (code >> 8) & 15u;
        if (nin > 0) seen |= 1u << (code & 3);
        if (nin > 1) seen |= 1u << ((code >> 2) & 3);
        if (nin > 2) seen |= 1u << ((code >> 4) & 3);
        T all[4];
        ld_cell_weights(a.wt + 4 * c, all);
        item_weights(all, code, w, wo);
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (!((seen >> j) & 1u)) par += all[j] * a.bc;
      }
      auto value = [&](T v0, T v1, T v2, T rhs, T &cell) {
        const T A = fma_rn(EA, v0 - rhs, rhs);
        const T B = fma_rn(EB, (two ? v1 : v0) - rhs, rhs);
        const T o = fma_rn((T)2, A, B) * (T)0.3333333333333333;
        cell = fma_rn(v0, w[0], fma_rn(v1, w[1], fma_rn(v2, w[2], fma_rn(o, wo, par))));
        return o;
      };
      if constexpr (GT > 0) {
        TI iv[GT];
        T o[GT];
#pragma unroll
        for (int g = 0; g < GT; g++) {
          T q = now.q0, cell;
          if (g > 0 && a.qs)
            q = g == 1 ? now.q1 : __ldg(reinterpret_cast<const T *>(src + c * src_bytes) + kSrcQ + g);
          o[g] = value(v0[g], v1[g], v2[g], fma_rn(bk, (T)sv[g], q), cell);
          iv[g] = (TI)cell;
        }
        if (HIGH && own >= a.cap)
          st_groups<true>(high + (int64_t)(own - a.cap) * GR, o);
        else if (own)
          st_groups<false>(low + own * GR, o);
        st_groups<true>(I + (uint64_t)iq * (uint32_t)GT, iv);
      } else {
        const T *sr = a.src + c * a.SW + kSrcQ;
        const TI *Sc = S + (int64_t)iq * a.sc;
        TI *Ic = I + (int64_t)iq * a.sc;
        for (int g = 0; g < G; g++) {
          const T v0 = slot(s0)[g];
          const T v1 = slot(s1)[g];
          const T v2 = slot(s2)[g];
          T cell;
          const T o = value(v0, v1, v2, fma_rn(bk, (T)Sc[g], sr[g * a.qs]), cell);
          if (own) slot(own)[g] = o;
          Ic[g] = (TI)cell;
        }
      }
    }
    hi = hi2;
    hi2 = lvl[min(L + 3, depth)];
    if constexpr (CLUSTER) {
      __syncwarp();  // the barrier wants whole warps, whose lanes have left the loop one by one
      asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
      __syncthreads();
    }
  }
}

// The sweep's own layout is [direction][item][G], items in sweep order (pos: the position of
// each cell [M][N]) or, without pos, cells in context numbering.  These tiles of 32 rows x DX
// directions of values of type V bring an array there and back through shared memory,
// directions d0 .. d0 + nd - 1, gw values of V a cell:
//   rows [rows][M] in caller numbering (perm; row = cell * gw + g, V = TI, gw = G), or
//   [cells][M][G] in context numbering (perm null; V = the G values of a cell and direction,
//   gw = 1).
// The caller's side moves whole lines.  On the other side the cells of a tile, neighbours in
// Morton order, lie in few runs (a level holds its cells in that order), and the tiles around
// it fill up the same lines while they are in L2: the scattered accesses are here, where 64
// warps an SM hide them, and not in the sweep, whose warps could not send them fast enough
// (a front's S by cell held them up 2 of 5 ms at 32^3 x 256 x 4 FP64).  All indices are loaded
// before the first value.
struct alignas(8) Bytes8 { uint32_t w[2]; };
struct alignas(16) Bytes16 { uint32_t w[4]; };
struct alignas(32) Bytes32 { double w[4]; };

// one access a value in global memory, 32 bytes included
template <class V>
__device__ __forceinline__ V ld_value(const V *p) {
  if constexpr (sizeof(V) == 32) {
    V v;
    ld_32(reinterpret_cast<const double *>(p), v.w[0], v.w[1], v.w[2], v.w[3]);
    return v;
  } else {
    return *p;
  }
}
template <class V>
__device__ __forceinline__ void st_value(V *p, const V &v) {
  if constexpr (sizeof(V) == 32)
    st_32(reinterpret_cast<double *>(p), v.w[0], v.w[1], v.w[2], v.w[3]);
  else
    *p = v;
}
template <class V>
constexpr int kTileDirs = sizeof(V) <= 8 ? 64 : 32;
template <class V, bool IMPORT>
__global__ void __launch_bounds__(256) k_tile(int64_t N, int gw, int M, int d0, int nd, const int32_t *perm,
                                              const uint32_t *pos, const V *in, V *out) {
  constexpr int DX = kTileDirs<V>;
  __shared__ V tile[DX][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t rows = N * gw;
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int x0 = blockIdx.y * DX;
  int64_t line[4];        // offset of row ty + 8 k on the caller's side
  int64_t item[DX / 8];   // offset of (row tx, direction ty + 8 k) on the sweep's side
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int64_t r = r0 + ty + 8 * k;
    line[k] = -1;
    if (r < rows) {
      const int64_t c = gw == 1 ? r : r / gw;
      line[k] = ((perm ? (int64_t)perm[c] : c) * gw + (r - c * gw)) * M + d0 + x0;
    }
  }
  {
    const int64_t r = r0 + tx, c = gw == 1 ? r : r / gw;
#pragma unroll
    for (int k = 0; k < DX / 8; k++) {
      const int x = x0 + ty + 8 * k;
      item[k] = -1;
      if (r < rows && x < nd) item[k] = x * rows + (pos ? (int64_t)pos[(d0 + x) * N + c] : c) * gw + (r - c * gw);
    }
  }
  if (IMPORT) {
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int h = 0; h < DX; h += 32)
        if (line[k] >= 0 && x0 + h + tx < nd) tile[h + tx][ty + 8 * k] = ld_value(in + line[k] + h + tx);
  } else {
#pragma unroll
    for (int k = 0; k < DX / 8; k++)
      if (item[k] >= 0) tile[ty + 8 * k][tx] = ld_value(in + item[k]);
  }
  __syncthreads();
  if (IMPORT) {
#pragma unroll
    for (int k = 0; k < DX / 8; k++)
      if (item[k] >= 0) st_value(out + item[k], tile[ty + 8 * k][tx]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int h = 0; h < DX; h += 32)
        if (line[k] >= 0 && x0 + h + tx < nd) st_value(out + line[k] + h + tx, tile[h + tx][ty + 8 * k]);
  }
}

// ---------------------------------------------------------------- plan
constexpr int kPlanThreads = 1024;

// Levels of every cell for one direction per CTA (breadth first: a cell joins the queue
// when its last upwind neighbour has been taken).  level [nd][N]; indeg, queue [nd][N]
// scratch; depth, count [nd]: levels and cells reached (fewer than N: a cycle).
template <class T>
__global__ void __launch_bounds__(kPlanThreads) k_plan_levels(int64_t N, int d0, const T *w, const T *rec,
                                                              uint32_t *indeg_all, uint32_t *queue_all,
                                                              uint32_t *level_all, int32_t *depth, int32_t *count) {
  __shared__ int tail;
  const int x = blockIdx.x, d = d0 + x;
  uint32_t *indeg = indeg_all + x * N, *queue = queue_all + x * N, *level = level_all + x * N;
  const T wx = w[3 * d], wy = w[3 * d + 1], wz = w[3 * d + 2];
  if (threadIdx.x == 0) tail = 0;
  __syncthreads();
  auto faces = [&](int64_t c, T *cosf, int *nbr) {
    T g[12];
    load_vec<T>(rec + c * Rec<T>::RW, g, 12);
    load_nbr<T>(rec + c * Rec<T>::RW, nbr);
    face_cos(g, wx, wy, wz, cosf);
  };
  for (int64_t c = threadIdx.x; c < N; c += kPlanThreads) {
    T cosf[4];
    int nbr[4];
    faces(c, cosf, nbr);
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) n += (cosf[j] < 0 && nbr[j] >= 0) ? 1u : 0u;
    indeg[c] = n;
    if (n == 0) {
      level[c] = 0;
      queue[atomicAdd(&tail, 1)] = (uint32_t)c;
    }
  }
  __syncthreads();
  int lo = 0, hi = tail, L = 0;
  __syncthreads();  // every thread has read tail before it moves on
  while (lo < hi) {
    L++;
    for (int i = lo + (int)threadIdx.x; i < hi; i += kPlanThreads) {
      T cosf[4];
      int nbr[4];
      faces(queue[i], cosf, nbr);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (cosf[j] > 0 && nbr[j] >= 0 && atomicSub(indeg + nbr[j], 1u) == 1u) {
          level[nbr[j]] = (uint32_t)L;
          queue[atomicAdd(&tail, 1)] = (uint32_t)nbr[j];
        }
    }
    __syncthreads();
    lo = hi;
    hi = tail;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    depth[d] = L;
    count[d] = lo;
  }
}

// sort keys (direction << lbits | level) and cells of nd directions
__global__ void k_plan_keys(int64_t N, int64_t total, int lbits, const uint32_t *level, uint32_t *key,
                            uint32_t *cell) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  const uint32_t x = (uint32_t)(i / N);
  key[i] = x << lbits | level[i];
  cell[i] = (uint32_t)(i - x * N);
}

// level offsets from the sorted keys of directions d0 .. (every level holds a cell)
__global__ void k_plan_offsets(int64_t N, int64_t total, int lbits, int d0, const uint32_t *key,
                               const int64_t *lvl_base, int32_t *lvl) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int64_t x = i / N, k = i - x * N;
  int32_t *o = lvl + lvl_base[d0 + x];
  const uint32_t mask = (1u << lbits) - 1u, L = key[i] & mask;
  if (k == 0 || (key[i - 1] & mask) != L) o[L] = (int32_t)k;
  if (k == N - 1) o[L + 1] = (int32_t)N;
}

// Items of one direction per CTA in sweep order: face choice and slots.  Within a
// level the cells' own slots are taken first (from the free list, or a new one), then the
// slots whose last reader sits in this level go back, so a slot is never written in a level
// that reads it.  Slots below cap2 (the shared memory of one CTA of two per SM) are preferred,
// then those below cap1 (of a CTA that has the SM alone): the free lists of these two sit at
// the front of `freed` and from cap2 on, that of the rest at its end (there are never more
// slots than cells).  need [M]: one more than a direction's largest slot.
template <class T>
__global__ void __launch_bounds__(kPlanThreads)
    k_plan_items(int64_t N, int d0, const T *w, const T *rec, const int32_t *lvl_all, const int64_t *lvl_base,
                 const int32_t *depth, const uint32_t *order_all, uint32_t *slot_all, uint32_t *readers_all,
                 uint32_t *freed_all, uint4 *ord_all, uint2 *hi_all, const T *wt, int cap2, int cap1, int32_t *need) {
  __shared__ int top[3], next[3];  // free list and next new slot below cap2, below cap1, beyond
  const int x = blockIdx.x, d = d0 + x;
  const uint32_t *order = order_all + x * N;
  uint32_t *slot_of = slot_all + x * N, *readers = readers_all + x * N, *freed = freed_all + x * N;
  uint4 *ord = ord_all + (int64_t)d * N;
  uint2 *hi16 = hi_all ? hi_all + (int64_t)d * N : nullptr;
  const int32_t *lvl = lvl_all + lvl_base[d];
  const T wx = w[3 * d], wy = w[3 * d + 1], wz = w[3 * d + 2];
  if (threadIdx.x == 0) {
    top[0] = top[1] = top[2] = 0;
    next[0] = 2;  // slots 0 and 1 hold the boundary value and zero
    next[1] = cap2;
    next[2] = cap1;
  }
  __syncthreads();
  int lo = 0;
  for (int L = 0; L < depth[d]; L++) {
    const int hi = lvl[L + 1];
    for (int i = lo + (int)threadIdx.x; i < hi; i += kPlanThreads) {
      const int64_t c = order[i];
      T g[16], cosf[4], tA, tB;
      int nbr[4];
      load_vec<T>(rec + c * Rec<T>::RW, g, 16);
      load_nbr<T>(rec + c * Rec<T>::RW, nbr);
      face_cos(g, wx, wy, wz, cosf);
      uint32_t code = item_geometry<T>(g, cosf, tA, tB);
      uint32_t n = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) n += (cosf[j] > 0 && nbr[j] >= 0) ? 1u : 0u;
      uint32_t own = 0;
      if (n) {
        int q = atomicSub(&top[0], 1) - 1;
        if (q >= 0) {
          own = freed[q];
        } else if ((q = atomicAdd(&next[0], 1)) < cap2) {
          own = (uint32_t)q;
        } else if ((q = atomicSub(&top[1], 1) - 1) >= 0) {
          own = freed[cap2 + q];
        } else if ((q = atomicAdd(&next[1], 1)) < cap1) {
          own = (uint32_t)q;
        } else {
          q = atomicSub(&top[2], 1) - 1;
          own = q >= 0 ? freed[N - 1 - q] : (uint32_t)atomicAdd(&next[2], 1);
        }
        slot_of[c] = own;
        readers[c] = n;
      }
      const int nin = (int)(code >> 6) & 3;
      uint32_t s[3] = {0u, 1u, 1u};  // no such in-face (a cell without any starts from the boundary value)
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const int f = (int)(code >> (2 * q)) & 3;
        const int b = f == 0 ? nbr[0] : f == 1 ? nbr[1] : f == 2 ? nbr[2] : nbr[3];
        if (q < nin) s[q] = b >= 0 ? slot_of[b] : 0u;
      }
      if constexpr (sizeof(T) == 8) {
        T f[4], wq[3], wo;
        ld_cell_weights(wt + 4 * c, f);
        item_weights(f, code, wq, wo);
        if (!(wo >= kOutMin)) code |= kCodeCell;
      }
      ord[i] = make_uint4((uint32_t)c, code, (own & 0xffffu) | s[0] << 16, (s[1] & 0xffffu) | s[2] << 16);
      if (hi16) hi16[i] = make_uint2(own >> 16 | (s[0] & 0xffff0000u), s[1] >> 16 | (s[2] & 0xffff0000u));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int q = 0; q < 3; q++) top[q] = max(top[q], 0);
      next[0] = min(next[0], cap2);
      next[1] = min(next[1], cap1);
    }
    __syncthreads();
    for (int i = lo + (int)threadIdx.x; i < hi; i += kPlanThreads) {
      const int64_t c = order[i];
      T g[12], cosf[4];
      int nbr[4];
      load_vec<T>(rec + c * Rec<T>::RW, g, 12);
      load_nbr<T>(rec + c * Rec<T>::RW, nbr);
      face_cos(g, wx, wy, wz, cosf);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (cosf[j] < 0 && nbr[j] >= 0 && atomicSub(readers + nbr[j], 1u) == 1u) {
          const uint32_t q = slot_of[nbr[j]];
          if (q < (uint32_t)cap2)
            freed[atomicAdd(&top[0], 1)] = q;
          else if (q < (uint32_t)cap1)
            freed[cap2 + atomicAdd(&top[1], 1)] = q;
          else
            freed[N - 1 - atomicAdd(&top[2], 1)] = q;
        }
    }
    lo = hi;
    __syncthreads();
  }
  if (threadIdx.x == 0) need[d] = next[2] > cap1 ? next[2] : next[1] > cap2 ? next[1] : next[0];
}

// The geometry stream of all items from their order: distances and positions (dist), weights
// (wgt; double), each where it is not null.
template <class T>
__global__ void k_fill_stream(int64_t N, int64_t total, const uint4 *ord, const T *w, const T *rec, const T *wt,
                              T *dist, uint32_t *pos, T *wgt, T *wgt3) {
  const int64_t at = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (at >= total) return;
  const int64_t d = at / N;
  const uint4 o = __ldcs(ord + at);
  const int64_t c = o.x;
  if (dist) {
    T g[16], cosf[4], tA, tB;
    load_vec<T>(rec + c * Rec<T>::RW, g, 16);
    face_cos(g, w[3 * d], w[3 * d + 1], w[3 * d + 2], cosf);
    (void)item_geometry<T>(g, cosf, tA, tB);
    dist[2 * at] = tA;
    dist[2 * at + 1] = tB;
    pos[d * N + c] = (uint32_t)(at - d * N);
  }
  if (wgt) {
    T f[4], wq[3], wo;
    ld_cell_weights(wt + 4 * c, f);
    item_weights(f, o.y, wq, wo);
    wgt[2 * at] = wq[0];
    wgt[2 * at + 1] = wq[1];
    wgt3[at] = wq[2];
  }
}

// Source record {k = alpha + betta, betta / k, alpha Q_g / k} of each context cell
// (rhs_g = alpha Q_g / k + (betta / k) S_g, GetRhsOpt with the division by k
// distributed) from caller arrays (caller numbering) ...
template <class T, class TA>
__global__ void k_dyn_from_arrays(int64_t N, int G, int SW, const int32_t *perm, const TA *alpha, const TA *betta,
                                  const TA *Q, const T *wt, T *src) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= N) return;
  const int64_t p = perm[c];
  const T al = (T)alpha[p], be = (T)betta[p];
  T *o = src + (int64_t)SW * c;
  const T k = al + be;
  o[0] = k;
  o[1] = be / k;
  for (int g = 0; g < G; g++) o[kSrcQ + g] = (al * (T)Q[p * G + g]) / k;
  if (weights_in_record<T>(G))
    for (int j = 0; j < 4; j++) o[kSrcW + j] = wt[4 * c + j];
}

// ... or from the solver state: alpha = a rho, betta = b rho, Q_g = B(T) / kRadiation / G.
template <class T>
__global__ void k_dyn_from_state(int64_t N, int G, int SW, const double *state, double a_coef, double b_coef,
                                 Emission em, const T *wt, T *src) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= N) return;
  const double rho = state[10 * c + 5], prs = state[10 * c + 9];
  const T al = (T)(a_coef * rho), be = (T)(b_coef * rho);
  const T q = (T)(planck_B(em, rho, prs) / em.rad_unit / (double)G);
  T *o = src + (int64_t)SW * c;
  const T k = al + be;
  o[0] = k;
  o[1] = be / k;
  o[kSrcQ] = (al * q) / k;
  if (weights_in_record<T>(G))
    for (int j = 0; j < 4; j++) o[kSrcW + j] = wt[4 * c + j];
}

// ---------------------------------------------------------------- coupled step
// 4-force from the moments summed over the groups.  FP64 moments per row: E
// [rows], F [rows][3], T [rows][9]; FP32 moments: [rows][16] = {E, F, Txx, Txy,
// Txz, Tyy, Tyz, Tzz, ...}.
__global__ void k_source(int64_t N, int G, const double *state, double a_coef, double b_coef, Emission em,
                         const double *mE, const double *mF, const double *mT, const float *mom, double *G4) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= N) return;
  double E = 0, F[3] = {0, 0, 0}, Tm[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int g = 0; g < G; g++) {
    const int64_t r = c * G + g;
    if (mom) {
      const float4 *m4 = reinterpret_cast<const float4 *>(mom + 16 * r);
      const float4 a = m4[0], b = m4[1], cc = m4[2];
      const double t9[9] = {b.x, b.y, b.z, b.y, b.w, cc.x, b.z, cc.x, cc.y};
      E += a.x;
      F[0] += a.y;
      F[1] += a.z;
      F[2] += a.w;
#pragma unroll
      for (int q = 0; q < 9; q++) Tm[q] += t9[q];
    } else {
      E += mE[r];
#pragma unroll
      for (int q = 0; q < 3; q++) F[q] += mF[3 * r + q];
#pragma unroll
      for (int q = 0; q < 9; q++) Tm[q] += mT[9 * r + q];
    }
  }
  double w[5];
#pragma unroll
  for (int q = 0; q < 5; q++) w[q] = state[10 * c + 5 + q];
  double out[4];
  rad_source_cell(em, w, a_coef * w[0], b_coef * w[0], E, F, Tm, out);
#pragma unroll
  for (int q = 0; q < 4; q++) G4[4 * c + q] = out[q];
}

// U.E += tau G0, U.S += tau G (radRHD_main.cpp:117-126), then GetPhysValueStab
// from its own guess without fallback (its status is ignored there as well).
// cnt: {ok, failed, newton iterations, max iterations}.
__global__ void k_source_c2p(int64_t N, Eos eos, double *state, const double *G4, double tau,
                             unsigned long long *cnt) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  unsigned long long ok = 0, failed = 0, iters = 0;
  if (c < N) {
    double u[5], w[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      u[q] = state[10 * c + q];
      w[q] = state[10 * c + 5 + q];
    }
    u[4] += tau * G4[4 * c];
    u[1] += tau * G4[4 * c + 1];
    u[2] += tau * G4[4 * c + 2];
    u[3] += tau * G4[4 * c + 3];
    int it = 0;
    const int code = c2p_from(eos, u, w, 0.0, false, &it);
    ok = code == 0;
    failed = code != 0;
    iters = (unsigned long long)it;
#pragma unroll
    for (int q = 0; q < 5; q++) {
      state[10 * c + q] = u[q];
      state[10 * c + 5 + q] = w[q];
    }
  }
  unsigned long long mx = iters;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ok += __shfl_xor_sync(0xffffffffu, ok, o);
    failed += __shfl_xor_sync(0xffffffffu, failed, o);
    iters += __shfl_xor_sync(0xffffffffu, iters, o);
    const unsigned long long m2 = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = m2 > mx ? m2 : mx;
  }
  if ((threadIdx.x & 31) == 0 && (ok | failed)) {
    atomicAdd(cnt + 0, ok);
    atomicAdd(cnt + 1, failed);
    atomicAdd(cnt + 2, iters);
    atomicMax(cnt + 3, mx);
  }
}

template <class T>
__global__ void k_rows_to_host_order(int64_t N, int64_t width, const int32_t *perm, const T *src, double *dst) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N * width) return;
  const int64_t c = i / width, k = i - c * width;
  dst[(int64_t)perm[c] * width + k] = (double)src[i];
}

unsigned grid_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

Eos eos_of(const rrhd_ctx *c) {
  Eos e;
  e.eos = c->eos;
  e.g1 = c->gamma;
  e.gg = c->gamma / (c->gamma - 1.0);
  return e;
}

// ---------------------------------------------------------------- launches
// Shared memory of a sweep's CTA.  With more directions than SMs two CTAs of 256 threads share
// an SM, so that one works while the other waits at its level's barrier, where their half of
// it holds all but a few of the slots and S and I are in sweep order; else one of 512 threads
// has it alone.  The slots beyond are in global memory.  32^3 x 256 directions, four groups
// FP64 (7 % of the slots beyond half an SM): 4.0 ms with two, 4.5 with one; 48^3, four groups
// mixed (57 % beyond): 14.4 and 10.2; 48^3, one group FP64 (none beyond, but S by cell: twice
// the directions at work push each other's lines out of L2): 9.5 and 5.5.  More threads an SM
// run out of registers (1024: 8.1 ms in the first).
constexpr int kSweepSMs = 148, kSmemTwo = 113 * 1024, kSmemOne = 226 * 1024;
constexpr double kTwoBeyond = 0.1;  // slots that may be beyond half an SM

int slot_cap(const RadState &R, bool two) {  // slots a CTA's shared memory can hold
  const size_t tv = R.prec == RRHD_RAD_FP32 ? sizeof(float) : sizeof(double);
  return (int)((two ? kSmemTwo : kSmemOne) / (tv * R.G));
}

// CTAs that share a direction: a power of two up to the portable eight.
// One where its slots take no more than half of an SM's shared memory: the values stay there (48^3 x
// 6 cells x 8 and 16 directions, one group FP64: 2.1 and 2.2 ms; 2.5 and 2.3 with two CTAs).
// Two at least where they take more than kRoomy of it: what does not fit is read back from L2 (48^3 x 8,
// four groups: 6.0; 3.6, 3.7 and 3.9 with 2, 4 and 8), and where it just fits, the L1 that is left holds
// hardly a load in flight (80^3 x 4, 206 KB: 20.3; 8.0, 6.1 and 6.0; 48^3 x 1 x 4, 197 KB: 6.9, 4.7 with two;
// 36^3 x 24 x 4, 194 KB: 2.3, 2.7 with two), but for levels of a few hundred items (24^3 x 64 x 8: 3.3, 3.7).
// All slots are in global memory then and a level's barrier costs more, so each CTA gets about a
// round of the level that the average item is in: 640 items, or 460 for four where one is not open
// (36^3 x 8 x 3, 1,050 items: 2.2 ms with one, 2.8 with two; 64^3 x 8 x 4, 3,300: 6.9, 5.8 and 6.5 with
// 2, 4 and 8; 64^3 x 1 x 4, 1,900: 8.1, 7.5 and 7.5; 96^3 x 8, 7,000: 12.4, 8.9 and 7.8).  Near all SMs they
// take bandwidth from one another: where one is open up to 64 of them (64^3 x 16 5.5 -> 3.7 ms with four
// each, 64^3 x 36 6.6 -> 6.7 with two), and eight each only where that leaves half (80^3 x 18: 9.3, 6.8
// with four).
constexpr int kRoomy = 196 * 1024;
// off: the level offsets of all directions.
int cluster_size(const RadState &R, int64_t slots, const std::vector<int32_t> &off) {
  if (slots <= slot_cap(R, true)) return 1;
  const int64_t bytes = (R.prec == RRHD_RAD_FP32 ? sizeof(float) : sizeof(double)) * R.G * slots;
  const bool roomy = bytes <= kRoomy, fits = slots <= slot_cap(R, false);
  double items = 0, squares = 0;
  for (int d = 0; d < R.M; d++)
    for (int L = 0; L < R.depth[d]; L++) {
      const double n = off[R.lvl_base[d] + L + 1] - off[R.lvl_base[d] + L];
      items += n;
      squares += n * n;
    }
  const double width = squares / items;
  int cl = 1;
  for (int next = 2; next <= 8; next *= 2) {
    const int most = roomy ? kSweepSMs * 7 / 16 : next == 8 ? kSweepSMs / 2 : kSweepSMs;
    const int each = roomy || next == 8 ? 640 : next == 4 ? 460 : fits ? 400 : 0;
    if (next * R.M > most || width < next * each) break;
    cl = next;
  }
  return cl;
}

template <class T, class TI, int GT, bool HIGH, bool WIDE, int GEO, int NT, int NB>
cudaError_t launch_sweep_kernel(const SweepArgs<T, TI> &a, int nd, size_t smem, cudaStream_t st) {
  if constexpr (HIGH && NT == 512) {
    if (a.cl > 1) {
      cudaLaunchAttribute cluster;
      cluster.id = cudaLaunchAttributeClusterDimension;
      cluster.val.clusterDim.x = (unsigned)a.cl;
      cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(nd * a.cl));
      cfg.blockDim = dim3(NT);
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cfg.attrs = &cluster;
      cfg.numAttrs = 1;
      return cudaLaunchKernelEx(&cfg, k_sweep<T, TI, GT, HIGH, WIDE, GEO, NT, NB, true>, a);
    }
  }
  auto *k = k_sweep<T, TI, GT, HIGH, WIDE, GEO, NT, NB, false>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<nd, NT, smem, st>>>(a);
  return cudaGetLastError();
}

template <class T, class TI, int GT, bool HIGH, bool WIDE, int NT, int NB>
cudaError_t launch_sweep_geo(const SweepArgs<T, TI> &a, int nd, size_t smem, cudaStream_t st) {
  if constexpr (sizeof(T) == 8)
    if (a.wgt) return launch_sweep_kernel<T, TI, GT, HIGH, WIDE, 2, NT, NB>(a, nd, smem, st);
  return a.dist ? launch_sweep_kernel<T, TI, GT, HIGH, WIDE, 1, NT, NB>(a, nd, smem, st)
                : launch_sweep_kernel<T, TI, GT, HIGH, WIDE, 0, NT, NB>(a, nd, smem, st);
}

// How the slots lie at a launch: two CTAs an SM only with S and I in sweep order.
struct Shape {
  bool two;
  int cap;
  int64_t low, high;
};
Shape shape_of(const RadState &R) {
  Shape q;
  q.two = R.two && R.d_pos;
  q.cap = R.cl > 1 ? 2 : slot_cap(R, q.two);
  q.low = std::min<int64_t>(R.slots, q.cap);
  q.high = std::max<int64_t>(0, R.slots - q.cap);
  return q;
}

template <class T, class TI, int GT>
cudaError_t launch_sweep_groups(const SweepArgs<T, TI> &a, int64_t low, bool two, int nd, cudaStream_t st) {
  const size_t smem = sizeof(T) * (size_t)low * a.G;
  if (two) {
    if (a.ord_hi) return launch_sweep_geo<T, TI, GT, true, true, 256, 2>(a, nd, smem, st);
    if (a.nhigh) return launch_sweep_geo<T, TI, GT, true, false, 256, 2>(a, nd, smem, st);
    return launch_sweep_geo<T, TI, GT, false, false, 256, 2>(a, nd, smem, st);
  }
  if constexpr (sizeof(T) == 4 && GT == 2) {
    // The same with two groups, at a cost (64 registers of 77), so where it fills SMs twice and the
    // lines of twice as many fronts are few times what L2 holds: 14^3 x 256 x 2 0.49 -> 0.33 ms, 40^3
    // 4.0 -> 3.7, but 44^3 (360 MB) 5.1 -> 6.9, 48^3 6.5 -> 10.6, and 24^3 x 100 0.78 -> 0.82.
    if (!a.nhigh && nd > kSweepSMs && 2 * smem <= kSmemOne &&
        low * 128 * std::min(nd, 2 * kSweepSMs) <= (int64_t)320 << 20)
      return launch_sweep_geo<T, TI, GT, false, false, 512, 2>(a, nd, smem, st);
  }
  if (a.ord_hi) return launch_sweep_geo<T, TI, GT, true, true, 512, 1>(a, nd, smem, st);
  if (a.nhigh) return launch_sweep_geo<T, TI, GT, true, false, 512, 1>(a, nd, smem, st);
  return launch_sweep_geo<T, TI, GT, false, false, 512, 1>(a, nd, smem, st);
}

// directions d0 .. d0 + nd - 1; S and I: element (cell, d0 + x, group) at q * sc + x * sd + group,
// q the cell or its position in the direction's sweep order
template <class T, class TI>
rrhd_status launch_sweep(rrhd_ctx *c, int d0, int nd, const void *S, void *I, int64_t sc, int64_t sd, bool by_pos,
                         bool one_q) {
  RadState &R = c->rad;
  SweepArgs<T, TI> a;
  a.N = c->N;
  a.d0 = d0;
  a.G = R.G;
  a.ord = R.d_ord;
  a.ord_hi = R.d_ord_hi;
  a.dist = (const T *)R.d_dist;
  a.wgt = (const T *)R.d_wgt;
  a.wgt3 = (const T *)R.d_wgt3;
  a.qs = one_q ? 0 : 1;
  a.SW = source_words<T>(R.G, one_q);
  a.wt = (const T *)R.d_wt;
  a.rec = (const T *)R.d_rec;
  a.w = (const T *)R.d_w;
  a.lvl = R.d_lvl;
  a.lvl_base = R.d_lvl_base;
  a.depth = R.d_depth;
  a.src = (const T *)R.d_src;
  a.slots = (T *)R.d_slots;
  const Shape q = shape_of(R);
  a.cap = (uint32_t)q.cap;
  a.cl = R.cl;
  a.nhigh = q.high;
  a.S = (const TI *)S;
  a.I = (TI *)I;
  a.sc = sc;
  a.sd = sd;
  a.by_pos = by_pos;
  a.bc = (T)R.bc;
  cudaError_t e;
  switch (R.G) {
    case 1: e = launch_sweep_groups<T, TI, 1>(a, q.low, q.two, nd, c->stream); break;
    case 2: e = launch_sweep_groups<T, TI, 2>(a, q.low, q.two, nd, c->stream); break;
    case 4: e = launch_sweep_groups<T, TI, 4>(a, q.low, q.two, nd, c->stream); break;
    default: e = launch_sweep_groups<T, TI, 0>(a, q.low, q.two, nd, c->stream); break;
  }
  RRHD_CUDA(e);
  return RRHD_OK;
}

// S and I in sweep order when a (cell, direction)'s values fill half a sector or more (32^3 x
// 256 x 4 FP64, kernel and tiles 4.8 -> 4.0 ms); else by cell: values of 8 bytes of neighbouring
// cells share sectors, and the coalesced tiles save more (48^3 x 256 x 1 FP64 6.1 -> 5.5 ms)
template <class TI>
bool by_position(const RadState &R) {
  return R.d_pos != nullptr && sizeof(TI) * R.G >= 16;
}

template <class TI, class V, bool IMPORT>
cudaError_t launch_tile(rrhd_ctx *c, int gw, int d0, int nd, const int32_t *perm, const void *in, void *out) {
  const dim3 tiles((unsigned)((c->N * gw + 31) / 32), (unsigned)((nd + kTileDirs<V> - 1) / kTileDirs<V>));
  const uint32_t *pos = by_position<TI>(c->rad) ? c->rad.d_pos : nullptr;
  k_tile<V, IMPORT><<<tiles, 256, 0, c->stream>>>(c->N, gw, c->rad.M, d0, nd, perm, pos, (const V *)in, (V *)out);
  return cudaGetLastError();
}

// S or I between the caller's arrays (rows, or [N][M][G] when cdg) and the sweep's layout
template <class TI, bool IMPORT>
cudaError_t move_tiles(rrhd_ctx *c, int d0, int nd, const void *in, void *out, bool cdg) {
  const RadState &R = c->rad;
  if (!cdg) return launch_tile<TI, TI, IMPORT>(c, R.G, d0, nd, c->d_perm, in, out);
  switch (sizeof(TI) * R.G) {
    case 4: return launch_tile<TI, float, IMPORT>(c, 1, d0, nd, nullptr, in, out);
    case 8: return launch_tile<TI, Bytes8, IMPORT>(c, 1, d0, nd, nullptr, in, out);
    case 16: return launch_tile<TI, Bytes16, IMPORT>(c, 1, d0, nd, nullptr, in, out);
    case 32: return launch_tile<TI, Bytes32, IMPORT>(c, 1, d0, nd, nullptr, in, out);
    default: return cudaErrorNotSupported;
  }
}

// ---------------------------------------------------------------- memory
// Beyond its plan a sweep keeps, where memory allows, in the order they are taken:
//   the scratch in the sweep's layout, of all directions or of as many as run at once (one at
//     least: without it a caller's sweep cannot run);
//   the first part of the geometry stream, distances (2 values an item) and positions (4 bytes),
//     which spares an item its cell's 144-byte record and brings S and I into sweep order;
//   the second part, weights (3 values an item, in double; a sweep in float takes the cell's).
// 96^3 x 6 cells x 256 directions x 4 groups in double, 21.7 GB of plan and 43.5 GB an array:
// with both parts (27.2 and 32.6 GB) a coupled step's sweep takes 204 ms, 234 with the first alone,
// 389 with none; a caller's sweep 294 with the first and 446 with none.  All results are the same bits.
// At setup they are kept beside the two arrays of the intensity's size that a coupled step or a
// caller will make; once those exist (first sweep, coupled step), beside a sixteenth of the device's
// memory, which is the caller's.  c->rad_keep bounds their sum where the caller has set it.
void drop_weights(RadState &R) {
  for (void **p : {&R.d_wgt, &R.d_wgt3}) {
    cudaFree(*p);
    *p = nullptr;
  }
}
void drop_stream(RadState &R) {
  drop_weights(R);
  for (void **p : {&R.d_dist, (void **)&R.d_pos}) {
    cudaFree(*p);
    *p = nullptr;
  }
}
void drop_scratch(RadState &R) {
  cudaFree(R.d_x);
  R.d_x = nullptr;
  R.xdirs = 0;
}

struct Sizes {
  size_t x;            // scratch of one direction
  size_t geo, wgt;     // the stream's parts
  size_t kept;         // what is kept now
};
Sizes sizes_of(const rrhd_ctx *c) {
  const RadState &R = c->rad;
  const size_t tv = R.prec == RRHD_RAD_FP32 ? sizeof(float) : sizeof(double), total = (size_t)c->N * R.M;
  Sizes z;
  z.x = (R.prec == RRHD_RAD_FP64 ? sizeof(double) : sizeof(float)) * (size_t)c->N * R.G;
  z.geo = (2 * tv + sizeof(uint32_t)) * total;
  z.wgt = R.prec == RRHD_RAD_FP32 ? 0 : 3 * tv * total;
  z.kept = (R.d_x ? z.x * R.xdirs : 0) + (R.d_dist ? z.geo : 0) + (R.d_wgt ? z.wgt : 0);
  return z;
}

// Bytes that may be taken: what is free beside `reserve` (negative: a sixteenth of the device's
// memory), within the caller's bound.
rrhd_status room_of(const rrhd_ctx *c, int64_t reserve, size_t &room) {
  size_t free_b = 0, all_b = 0;
  RRHD_CUDA(cudaMemGetInfo(&free_b, &all_b));
  const size_t hold = all_b / 16 + (reserve < 0 ? 0 : (size_t)reserve);
  room = free_b > hold ? free_b - hold : 0;
  if (c->rad_keep >= 0) {
    const size_t kept = sizes_of(c).kept, keep = (size_t)c->rad_keep;
    room = std::min(room, keep > kept ? keep - kept : (size_t)0);
  }
  return RRHD_OK;
}

bool take(void **p, size_t bytes) {
  if (cudaMalloc(p, bytes) == cudaSuccess) return true;
  cudaGetLastError();
  *p = nullptr;
  return false;
}

// directions of a sweep that run at once
int at_once(const RadState &R) { return std::min(R.M, R.two ? 2 * kSweepSMs : kSweepSMs); }

template <class T>
rrhd_status fill_t(rrhd_ctx *c, int64_t reserve, bool scratch) {
  RadState &R = c->rad;
  const Sizes z = sizes_of(c);
  size_t room = 0;
  rrhd_status s = room_of(c, reserve, room);
  if (s) return s;
  const auto held = [&](bool got, size_t bytes) {
    if (got) room -= bytes;
    return got;
  };
  if (scratch && !R.d_x) {
    const size_t geo = R.d_dist ? 0 : z.geo;
    const int dirs = z.x * R.M + geo <= room ? R.M : z.x * at_once(R) <= room ? at_once(R) : 0;
    if (dirs && held(take(&R.d_x, z.x * dirs), z.x * dirs)) R.xdirs = dirs;
  }
  const size_t tv = sizeof(T), total = (size_t)c->N * R.M;
  bool geo = false, wgt = false;
  if (!R.d_dist && z.geo <= room) {
    geo = take(&R.d_dist, 2 * tv * total) && take((void **)&R.d_pos, sizeof(uint32_t) * total);
    if (!held(geo, z.geo)) drop_stream(R);
  }
  if (z.wgt && R.d_dist && !R.d_wgt && z.wgt <= room) {
    wgt = take(&R.d_wgt, 2 * tv * total) && take(&R.d_wgt3, tv * total);
    if (!held(wgt, z.wgt)) drop_weights(R);
  }
  if (geo || wgt) {
    k_fill_stream<T><<<grid_for((int64_t)total, 256), 256, 0, c->stream>>>(
        c->N, (int64_t)total, R.d_ord, (const T *)R.d_w, (const T *)R.d_rec, (const T *)R.d_wt,
        geo ? (T *)R.d_dist : nullptr, R.d_pos, wgt ? (T *)R.d_wgt : nullptr, (T *)R.d_wgt3);
    RRHD_CUDA(cudaGetLastError());
  }
  return RRHD_OK;
}
rrhd_status fill(rrhd_ctx *c, int64_t reserve, bool scratch) {
  return c->rad.prec == RRHD_RAD_FP32 ? fill_t<float>(c, reserve, scratch) : fill_t<double>(c, reserve, scratch);
}

// Frees, in steps, what a sweep can do without: the scratch (a later sweep makes another), the
// weights, the rest of the stream.
rrhd_status give_back(rrhd_ctx *c, bool &freed) {
  RadState &R = c->rad;
  freed = R.d_x || R.d_dist;
  if (!freed) return RRHD_OK;
  RRHD_CUDA(cudaStreamSynchronize(c->stream));
  if (R.d_x)
    drop_scratch(R);
  else if (R.d_wgt)
    drop_weights(R);
  else
    drop_stream(R);
  return RRHD_OK;
}

// The scratch of a caller's sweep: of all directions, or of whole runs of as many as run at once;
// the stream makes room for one such run, and if it is still too much the number is halved down to one.
rrhd_status make_scratch(rrhd_ctx *c) {
  RadState &R = c->rad;
  const Sizes z = sizes_of(c);
  const int run = at_once(R);
  size_t room = 0;
  rrhd_status s = room_of(c, -1, room);
  if (s) return s;
  int dirs = (int)std::min<size_t>(R.M, room / z.x);
  if (dirs < R.M) dirs = std::max(run, dirs - dirs % run);
  if (c->rad_keep >= 0)
    dirs = (int)std::min<size_t>(dirs, std::max<size_t>(1, ((size_t)c->rad_keep - std::min((size_t)c->rad_keep, z.kept)) / z.x));
  while (!take(&R.d_x, z.x * dirs)) {
    if (dirs <= run && R.d_dist) {
      bool freed = false;
      if ((s = give_back(c, freed))) return s;
      continue;
    }
    if (dirs == 1) return rrhd_fail(RRHD_ERR_OOM, "sweep scratch allocation failed");
    dirs = dirs > run ? (dirs - 1) / run * run : (dirs + 1) / 2;
  }
  R.xdirs = dirs;
  return RRHD_OK;
}

// One sweep of every direction on the caller's rows [N*G][M], swept in place in the scratch, as
// many directions at a time as it holds.
template <class T, class TI>
rrhd_status run_sweep_rows(rrhd_ctx *c, const void *S, void *I) {
  RadState &R = c->rad;
  rrhd_status s;
  if (!R.settled) {  // the caller's arrays exist by now
    const bool short_of = !R.d_x || !R.d_dist || (sizeof(T) == 8 && !R.d_wgt);
    if (short_of && (s = fill(c, -1, true))) return s;
    R.settled = true;
  }
  if (!R.d_x && (s = make_scratch(c))) return s;
  for (int d0 = 0; d0 < R.M; d0 += R.xdirs) {
    const int nd = std::min(R.xdirs, R.M - d0);
    RRHD_CUDA((move_tiles<TI, true>(c, d0, nd, S, R.d_x, false)));
    if ((s = launch_sweep<T, TI>(c, d0, nd, R.d_x, R.d_x, R.G, c->N * R.G, by_position<TI>(R), false))) return s;
    RRHD_CUDA((move_tiles<TI, false>(c, d0, nd, R.d_x, I, false)));
  }
  return RRHD_OK;
}
rrhd_status run_sweep_rows(rrhd_ctx *c, const void *S, void *I) {
  switch (c->rad.prec) {
    case RRHD_RAD_FP64: return run_sweep_rows<double, double>(c, S, I);
    case RRHD_RAD_MIXED: return run_sweep_rows<double, float>(c, S, I);
    default: return run_sweep_rows<float, float>(c, S, I);
  }
}

// ... and on the coupled step's arrays [N][M][G] in context numbering.  Neither is needed again as
// it is, so the old intensity is the scratch, the result takes the place of the old scattering
// integral, and the two change places.  Where a (cell, direction) is not a whole access (8 groups
// and more) S is read and I written as they lie.
template <class T, class TI>
rrhd_status run_sweep_coupled(rrhd_ctx *c) {
  RadState &R = c->rad;
  const size_t cd = sizeof(TI) * R.G;
  if (!(cd == 4 || cd == 8 || cd == 16 || cd == 32))
    return launch_sweep<T, TI>(c, 0, R.M, R.d_S, R.d_I, (int64_t)R.M * R.G, R.G, false, true);
  RRHD_CUDA((move_tiles<TI, true>(c, 0, R.M, R.d_S, R.d_I, true)));
  const rrhd_status s =
      launch_sweep<T, TI>(c, 0, R.M, R.d_I, R.d_I, R.G, c->N * R.G, by_position<TI>(R), true);
  if (s) return s;
  RRHD_CUDA((move_tiles<TI, false>(c, 0, R.M, R.d_I, R.d_S, true)));
  std::swap(R.d_I, R.d_S);
  return RRHD_OK;
}
rrhd_status run_sweep_coupled(rrhd_ctx *c) {
  switch (c->rad.prec) {
    case RRHD_RAD_FP64: return run_sweep_coupled<double, double>(c);
    case RRHD_RAD_MIXED: return run_sweep_coupled<double, float>(c);
    default: return run_sweep_coupled<float, float>(c);
  }
}

// ---------------------------------------------------------------- plan, host side
struct Scratch {  // device memory of the plan build, freed on every way out
  std::vector<void *> p;
  ~Scratch() {
    for (void *q : p) cudaFree(q);
  }
  void *get(size_t bytes) {
    void *q = nullptr;
    if (cudaMalloc(&q, bytes) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    p.push_back(q);
    return q;
  }
};

int bits_for(int64_t n) {  // bits that hold 0 .. n - 1
  int b = 0;
  while ((int64_t(1) << b) < n) b++;
  return b;
}

// The sweep order, items and slots of every direction (R.d_ord, level offsets).
template <class T>
rrhd_status build_plan(rrhd_ctx *c) {
  RadState &R = c->rad;
  const int64_t N = c->N, total = N * (int64_t)R.M;
  cudaStream_t st = c->stream;
  const rrhd_status oom = RRHD_ERR_OOM;
  if (cudaMalloc(&R.d_ord, sizeof(uint4) * total) != cudaSuccess) {
    cudaGetLastError();
    R.d_ord = nullptr;
    return rrhd_fail(oom, "sweep plan allocation failed (%lld bytes)", (long long)(sizeof(uint4) * total));
  }
  // directions of a build pass: six 32-bit words a pair (and a sort's) in at most half of the free
  // memory, within the caller's bound
  size_t free_b = 0, all_b = 0;
  RRHD_CUDA(cudaMemGetInfo(&free_b, &all_b));
  int64_t build = (int64_t)(free_b / 2);
  if (c->rad_keep >= 0) build = std::min(build, c->rad_keep);
  const int B = (int)std::max<int64_t>(1, std::min<int64_t>(R.M, build / (28 * N)));
  R.build_dirs = B;
  Scratch mem;
  uint32_t *buf[6];
  for (uint32_t *&b : buf)
    if (!(b = (uint32_t *)mem.get(sizeof(uint32_t) * (size_t)N * B))) return rrhd_fail(oom, "sweep plan scratch");
  uint32_t *const level = buf[0], *const key = buf[1], *const cell = buf[2], *const key2 = buf[3],
           *const order = buf[4], *const indeg = buf[5], *const queue = key;
  int32_t *d_count = (int32_t *)mem.get(sizeof(int32_t) * R.M);
  int32_t *d_need = (int32_t *)mem.get(sizeof(int32_t) * R.M);
  if (!d_count || !d_need || cudaMalloc(&R.d_depth, sizeof(int32_t) * R.M) != cudaSuccess ||
      cudaMalloc(&R.d_lvl_base, sizeof(int64_t) * R.M) != cudaSuccess)
    return rrhd_fail(oom, "sweep plan scratch");
  size_t sort_bytes = 0;
  RRHD_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, key, key2, cell, order, N * B, 0, 32, st));
  void *sort_tmp = mem.get(sort_bytes);
  if (!sort_tmp) return rrhd_fail(oom, "sweep plan scratch");
  R.depth.assign(R.M, 0);
  R.lvl_base.assign(R.M, 0);
  std::vector<int32_t> count(R.M), need(R.M, 0);
  const T *w = (const T *)R.d_w, *rec = (const T *)R.d_rec;
  // levels of every direction first: their number decides the sort keys and the offsets
  auto levels_of = [&](int d0, int nd) -> rrhd_status {
    k_plan_levels<T><<<nd, kPlanThreads, 0, st>>>(N, d0, w, rec, indeg, queue, level, R.d_depth, d_count);
    RRHD_CUDA(cudaGetLastError());
    RRHD_CUDA(cudaMemcpyAsync(R.depth.data() + d0, R.d_depth + d0, sizeof(int32_t) * nd, cudaMemcpyDeviceToHost, st));
    RRHD_CUDA(cudaMemcpyAsync(count.data() + d0, d_count + d0, sizeof(int32_t) * nd, cudaMemcpyDeviceToHost, st));
    RRHD_CUDA(cudaStreamSynchronize(st));
    return RRHD_OK;
  };
  rrhd_status s;
  for (int d0 = 0; d0 < R.M; d0 += B)
    if ((s = levels_of(d0, std::min(B, R.M - d0)))) return s;
  int64_t entries = 0;
  for (int d = 0; d < R.M; d++) {
    if (count[d] != N)
      return rrhd_fail(RRHD_ERR_STATE, "sweep dependency cycle: %lld of %lld cells have, in direction %d, an upwind "
                                       "neighbour that depends on them", (long long)(N - count[d]), (long long)N, d);
    R.lvl_base[d] = entries;
    entries += R.depth[d] + 1;
  }
  if (cudaMalloc(&R.d_lvl, sizeof(int32_t) * entries) != cudaSuccess) {
    cudaGetLastError();
    R.d_lvl = nullptr;
    return rrhd_fail(oom, "sweep plan allocation failed");
  }
  RRHD_CUDA(cudaMemcpyAsync(R.d_lvl_base, R.lvl_base.data(), sizeof(int64_t) * R.M, cudaMemcpyHostToDevice, st));
  for (int d0 = 0; d0 < R.M; d0 += B) {
    const int nd = std::min(B, R.M - d0);
    if (B < R.M && (s = levels_of(d0, nd))) return s;  // the scratch held another batch's levels
    const int lbits = std::max(1, bits_for(*std::max_element(R.depth.begin() + d0, R.depth.begin() + d0 + nd)));
    // directions per sort: its keys are 32-bit
    const int ns = (int)std::min<int64_t>(nd, lbits < 31 ? int64_t(1) << (32 - lbits) : 1);
    for (int x = 0; x < nd; x += ns) {
      const int n = std::min(ns, nd - x);
      const int64_t at = N * x, pairs = N * n;
      k_plan_keys<<<grid_for(pairs, 256), 256, 0, st>>>(N, pairs, lbits, level + at, key + at, cell + at);
      RRHD_CUDA(cudaGetLastError());
      RRHD_CUDA(cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, key + at, key2 + at, cell + at, order + at,
                                                pairs, 0, std::min(32, lbits + bits_for(n)), st));
      k_plan_offsets<<<grid_for(pairs, 256), 256, 0, st>>>(N, pairs, lbits, d0 + x, key2 + at, R.d_lvl_base, R.d_lvl);
      RRHD_CUDA(cudaGetLastError());
    }
    auto items = [&]() -> rrhd_status {
      k_plan_items<T><<<nd, kPlanThreads, 0, st>>>(N, d0, w, rec, R.d_lvl, R.d_lvl_base, R.d_depth, order, indeg, key,
                                                   cell, R.d_ord, R.d_ord_hi, (const T *)R.d_wt, slot_cap(R, true),
                                                   slot_cap(R, false), d_need);
      RRHD_CUDA(cudaGetLastError());
      RRHD_CUDA(cudaMemcpyAsync(need.data() + d0, d_need + d0, sizeof(int32_t) * nd, cudaMemcpyDeviceToHost, st));
      RRHD_CUDA(cudaStreamSynchronize(st));
      return RRHD_OK;
    };
    if ((s = items())) return s;
    if (*std::max_element(need.begin(), need.end()) > 65536 && !R.d_ord_hi) {
      // slots beyond 16 bits: their upper halves in a second array (zero for the batches before)
      if (cudaMalloc(&R.d_ord_hi, sizeof(uint2) * total) != cudaSuccess) {
        cudaGetLastError();
        R.d_ord_hi = nullptr;
        return rrhd_fail(oom, "sweep plan allocation failed");
      }
      RRHD_CUDA(cudaMemsetAsync(R.d_ord_hi, 0, sizeof(uint2) * total, st));
      if ((s = items())) return s;
    }
  }
  std::vector<int32_t> off((size_t)entries);
  RRHD_CUDA(cudaMemcpyAsync(off.data(), R.d_lvl, sizeof(int32_t) * entries, cudaMemcpyDeviceToHost, st));
  RRHD_CUDA(cudaStreamSynchronize(st));
  const int cap2 = slot_cap(R, true);
  int64_t all = 0, beyond = 0, most = 0;
  for (int32_t n : need) {
    all += n;
    beyond += std::max(0, n - cap2);
    most = std::max<int64_t>(most, n);
  }
  const size_t ti = R.prec == RRHD_RAD_FP64 ? sizeof(double) : sizeof(float);
  R.slots = most;
  R.cl = cluster_size(R, most, off);
  R.two = R.cl == 1 && R.M > kSweepSMs && ti * R.G >= 16 && (double)beyond <= kTwoBeyond * (double)all;
  // rrhd_rad_plan_info: levels and the largest level over batches of R.DB directions
  R.levels = R.max_level = 0;
  for (int d0 = 0; d0 < R.M; d0 += R.DB) {
    std::vector<int64_t> items;
    for (int d = d0; d < std::min(R.M, d0 + R.DB); d++) {
      const int32_t *o = off.data() + R.lvl_base[d];
      if ((int)items.size() < R.depth[d]) items.resize(R.depth[d], 0);
      for (int L = 0; L < R.depth[d]; L++) items[L] += o[L + 1] - o[L];
    }
    R.levels += (int64_t)items.size();
    for (int64_t n : items) R.max_level = std::max(R.max_level, n);
  }
  return RRHD_OK;
}

}  // namespace

void rrhd_rad_release(rrhd_ctx *c) {
  RadState &R = c->rad;
  void *ptrs[] = {R.d_w,     R.d_rec, R.d_src, R.d_ord, R.d_ord_hi, R.d_dist, R.d_wgt, R.d_wgt3, R.d_wt, R.d_pos, R.d_lvl, R.d_lvl_base, R.d_depth,
                  R.d_slots, R.d_x,   R.d_I,   R.d_S,   R.d_G4,     R.d_mE,  R.d_mF,  R.d_mT,       R.d_mom,
                  R.d_cnt};
  for (void *p : ptrs) cudaFree(p);
  for (cudaEvent_t e : R.ev)
    if (e) cudaEventDestroy(e);
  if (R.side) cudaStreamDestroy(R.side);
  if (R.tc) rrhd_scatter_tc_destroy(R.tc);
  R = RadState();
}

// T: the records (geometry, opacities and sources), directions, slots and arithmetic.
template <class T>
static rrhd_status rad_setup_t(rrhd_ctx *c) {
  RadState &R = c->rad;
  const int64_t N = c->N;
  constexpr int W = Rec<T>::RW;
  R.SW = source_words<T>(R.G, false);
  std::vector<T> rec((size_t)W * N, (T)0), wt((size_t)4 * N), w(3 * R.M);
  std::vector<int32_t> iperm(N);
  for (int64_t i = 0; i < N; i++) iperm[c->h_perm[i]] = (int32_t)i;
  for (int64_t cn = 0; cn < N; cn++) {
    const int64_t p = c->h_perm[cn];
    T *r = rec.data() + (size_t)W * cn;
    int32_t nbr[4];
    double area = 0.0;
    for (int j = 0; j < 4; j++) {
      const int32_t fc = c->h_cell_faces[4 * p + j];
      const bool out = (c->h_cell_sign[p] >> j) & 1;
      for (int x = 0; x < 3; x++) {
        const double v = c->h_face_n[3 * (int64_t)fc + x];
        r[3 * j + x] = (T)(out ? v : -v);
      }
      r[12 + j] = (T)(3.0 * c->h_cell_V[p] / c->h_face_area[fc]);
      area += c->h_face_area[fc];
      const int32_t l = c->h_face_l[fc], rr = c->h_face_r[fc];
      const int32_t o = (l == p) ? rr : l;
      nbr[j] = o < 0 ? -1 : iperm[o];
    }
    std::memcpy(r + Rec<T>::NBR, nbr, sizeof nbr);
    // ReCalcIllumOpt (illum_utils.cpp:415-430): the plain mean for the caller's last cell
    for (int j = 0; j < 4; j++)
      wt[4 * cn + j] = p == N - 1 ? (T)0.25 : (T)(c->h_face_area[c->h_cell_faces[4 * p + j]] / area);
  }
  for (int q = 0; q < 3 * R.M; q++) w[q] = (T)R.dirs->h_w[q];
  auto up = [&](void **dst, const void *from, size_t bytes) -> rrhd_status {
    if (cudaMalloc(dst, bytes) != cudaSuccess) {
      cudaGetLastError();
      *dst = nullptr;
      return rrhd_fail(RRHD_ERR_OOM, "sweep allocation failed");
    }
    RRHD_CUDA(cudaMemcpy(*dst, from, bytes, cudaMemcpyHostToDevice));
    return RRHD_OK;
  };
  rrhd_status s;
  if ((s = up(&R.d_rec, rec.data(), sizeof(T) * rec.size())) || (s = up(&R.d_w, w.data(), sizeof(T) * w.size())) ||
      (s = up(&R.d_wt, wt.data(), sizeof(T) * wt.size())))
    return s;
  if (cudaMalloc(&R.d_src, sizeof(T) * (size_t)R.SW * N) != cudaSuccess) {
    cudaGetLastError();
    R.d_src = nullptr;
    return rrhd_fail(RRHD_ERR_OOM, "sweep allocation failed");
  }
  if ((s = build_plan<T>(c))) return s;
  Shape q = shape_of(R);  // without positions: one CTA an SM
  int64_t high = q.high;
  if (R.two) high = std::max<int64_t>(high, R.slots - slot_cap(R, true));
  if (high) {
    const size_t bytes = sizeof(T) * (size_t)high * R.G * R.M;
    if (!take(&R.d_slots, bytes))
      return rrhd_fail(RRHD_ERR_OOM, "sweep slot allocation failed (%lld bytes)", (long long)bytes);
  }
  const size_t ti = R.prec == RRHD_RAD_FP64 ? sizeof(double) : sizeof(float);
  const size_t arrays = 2 * ti * (size_t)N * R.M * R.G + 128 * (size_t)N * (R.G + 1);
  if ((s = fill(c, (int64_t)arrays, true))) return s;
  RRHD_CUDA(cudaStreamSynchronize(c->stream));
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_setup(rrhd_ctx *c, const rrhd_dirs *dirs, const rrhd_rad_opts *o) {
  RRHD_CHECK_ARG(c && dirs && o, "null argument");
  RRHD_CHECK_ARG(o->groups >= 1 && o->groups <= 64, "groups must be in [1, 64]");
  RRHD_CHECK_ARG(o->precision == RRHD_RAD_FP64 || o->precision == RRHD_RAD_FP32 || o->precision == RRHD_RAD_MIXED,
                 "bad precision");
  RRHD_CHECK_ARG(dirs->device == c->device, "direction set lives on another device");
  RRHD_CHECK_ARG(o->item_geometry == 0 || o->item_geometry == 1, "item_geometry: 0 or 1");
  RRHD_CHECK_ARG(o->item_geometry == 0 || o->precision != RRHD_RAD_FP64,
                 "item_geometry needs RRHD_RAD_FP32 or RRHD_RAD_MIXED");
  int DB = o->dirs_per_batch;
  RRHD_CHECK_ARG(DB == 0 || (DB > 0 && DB <= 256 && (DB & (DB - 1)) == 0), "dirs_per_batch: power of two <= 256");
  RRHD_CUDA(cudaSetDevice(c->device));
  RRHD_CUDA(cudaStreamSynchronize(c->stream));
  rrhd_rad_release(c);
  RadState &R = c->rad;
  R.dirs = dirs;
  R.M = dirs->M;
  R.G = o->groups;
  if (DB == 0) {
    DB = 1;
    while (DB < std::min(R.M, 64)) DB <<= 1;
  }
  R.DB = DB;
  const int shift = bits_for(c->N);
  if (shift > 31 || ((int64_t)DB << shift) > (int64_t)UINT32_MAX + 1)
    return rrhd_fail(RRHD_ERR_LIMIT, "dirs_per_batch x 2^ceil(log2 cells) must stay within 2^32");
  R.prec = o->precision;
  R.bc = o->boundary_value;
  const rrhd_status s = R.prec == RRHD_RAD_FP32 ? rad_setup_t<float>(c) : rad_setup_t<double>(c);
  if (s) {
    rrhd_rad_release(c);
    return s;
  }
  R.ready = true;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_plan_info(const rrhd_ctx *c, int64_t *levels, int64_t *max_level_items) {
  RRHD_CHECK_ARG(c, "null context");
  if (!c->rad.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  if (levels) *levels = c->rad.levels;
  if (max_level_items) *max_level_items = c->rad.max_level;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_plan_form(const rrhd_ctx *c, rrhd_rad_form *form) {
  RRHD_CHECK_ARG(c && form, "null argument");
  const RadState &R = c->rad;
  if (!R.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  const Shape q = shape_of(R);
  form->cluster = R.cl;
  form->ctas_per_sm = q.two ? 2 : 1;
  form->wide_slots = R.d_ord_hi ? 1 : 0;
  form->stream = !R.d_dist ? 0 : R.prec == RRHD_RAD_FP32 || R.d_wgt ? 2 : 1;
  form->scratch_dirs = R.d_x ? R.xdirs : 0;
  form->build_dirs = R.build_dirs;
  form->slots_shared = q.low;
  form->slots_global = q.high;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_memory(rrhd_ctx *c, int64_t bytes) {
  RRHD_CHECK_ARG(c, "null context");
  c->rad_keep = bytes < 0 ? -1 : bytes;
  RadState &R = c->rad;
  if (!R.ready) return RRHD_OK;
  RRHD_CUDA(cudaSetDevice(c->device));
  R.settled = false;  // a wider bound is used by the next sweep
  if (R.d_x && R.xdirs < R.M) {
    RRHD_CUDA(cudaStreamSynchronize(c->stream));
    drop_scratch(R);
  }
  bool freed = true;
  while (c->rad_keep >= 0 && freed && sizes_of(c).kept > (size_t)c->rad_keep) {
    const rrhd_status s = give_back(c, freed);
    if (s) return s;
  }
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_plan_levels(const rrhd_ctx *c, int32_t *levels) {
  RRHD_CHECK_ARG(c && levels, "null argument");
  const RadState &R = c->rad;
  if (!R.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  RRHD_CUDA(cudaSetDevice(c->device));
  const int64_t N = c->N;
  std::vector<uint4> ord((size_t)N);
  std::vector<int32_t> off;
  RRHD_CUDA(cudaStreamSynchronize(c->stream));
  for (int d = 0; d < R.M; d++) {
    off.resize(R.depth[d] + 1);
    RRHD_CUDA(cudaMemcpy(ord.data(), R.d_ord + (int64_t)d * N, sizeof(uint4) * N, cudaMemcpyDeviceToHost));
    RRHD_CUDA(cudaMemcpy(off.data(), R.d_lvl + R.lvl_base[d], sizeof(int32_t) * off.size(), cudaMemcpyDeviceToHost));
    for (int L = 0; L < R.depth[d]; L++)
      for (int32_t k = off[L]; k < off[L + 1]; k++) levels[(int64_t)d * N + c->h_perm[ord[k].x]] = L;
  }
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_sweep(rrhd_ctx *c, const void *alpha, const void *betta, const void *Q, const void *S,
                                  void *I) {
  RRHD_CHECK_ARG(c && alpha && betta && Q && S && I, "null argument");
  RadState &R = c->rad;
  if (!R.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  RRHD_CUDA(cudaSetDevice(c->device));
  const int64_t N = c->N;
  if (R.prec == RRHD_RAD_FP64)
    k_dyn_from_arrays<double, double><<<grid_for(N, 256), 256, 0, c->stream>>>(
        N, R.G, R.SW, c->d_perm, (const double *)alpha, (const double *)betta, (const double *)Q,
        (const double *)R.d_wt, (double *)R.d_src);
  else if (R.prec == RRHD_RAD_MIXED)  // float arrays, double records
    k_dyn_from_arrays<double, float><<<grid_for(N, 256), 256, 0, c->stream>>>(
        N, R.G, R.SW, c->d_perm, (const float *)alpha, (const float *)betta, (const float *)Q,
        (const double *)R.d_wt, (double *)R.d_src);
  else
    k_dyn_from_arrays<float, float><<<grid_for(N, 256), 256, 0, c->stream>>>(
        N, R.G, R.SW, c->d_perm, (const float *)alpha, (const float *)betta, (const float *)Q,
        (const float *)R.d_wt, (float *)R.d_src);
  RRHD_CUDA(cudaGetLastError());
  return run_sweep_rows(c, S, I);
}

// ---------------------------------------------------------------- coupled step
namespace {
// I or S of the caller's cells p0 .. p0 + n - 1 as rows [n * G][M]
template <class T>
__global__ void k_cdg_to_rows(int64_t p0, int64_t n, int M, int G, const int32_t *iperm, const T *src, double *dst) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t per = (int64_t)M * G;
  if (i >= n * per) return;
  const int64_t p = i / per, rem = i - p * per;
  const int g = (int)(rem / M), d = (int)(rem - (int64_t)g * M);
  dst[i] = (double)src[((int64_t)iperm[p0 + p] * M + d) * G + g];
}

// Moments of the last scattering per row (cell * G + g), caller order, as
// {E, F0, F1, F2, T00, T01, T02, T11, T12, T22}: from the FP64 arrays (E [rows],
// F [rows][3], T [rows][9] column-major) or the FP32 [rows][16] columns.
__global__ void k_mom_to_rows(int64_t N, int G, const int32_t *perm, const double *mE, const double *mF,
                              const double *mT, const float *mom, double *dst) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= N * G) return;
  const int64_t c = r / G, g = r - c * G;
  double *o = dst + ((int64_t)perm[c] * G + g) * 10;
  if (mom) {
    for (int k = 0; k < 10; k++) o[k] = (double)mom[16 * r + k];
    return;
  }
  o[0] = mE[r];
  for (int k = 0; k < 3; k++) o[1 + k] = mF[3 * r + k];
  const int ij[6][2] = {{0, 0}, {0, 1}, {0, 2}, {1, 1}, {1, 2}, {2, 2}};
  for (int k = 0; k < 6; k++) o[4 + k] = mT[9 * r + 3 * ij[k][1] + ij[k][0]];
}

template <class T>
__global__ void k_rows_to_cdg(int64_t p0, int64_t n, int M, int G, const int32_t *iperm, const double *src, T *dst) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t per = (int64_t)M * G;
  if (i >= n * per) return;
  const int64_t p = i / per, rem = i - p * per;
  const int g = (int)(rem / M), d = (int)(rem - (int64_t)g * M);
  dst[((int64_t)iperm[p0 + p] * M + d) * G + g] = (T)src[i];
}

// I or S between the context and the caller's host rows [N * G][M], a piece of the caller's
// cells at a time through a buffer of at most kPieceBytes (one cell at least): at 96^3 x 6
// cells, 256 directions and 4 groups a whole array is 43.5 GB, more than a coupled step leaves.
// What bounds it is the copy to or from the host; a piece's kernel moves its bytes once on the device.
constexpr size_t kPieceBytes = (size_t)256 << 20;
rrhd_status move_rows(rrhd_ctx *c, void *array, double *to, const double *from) {
  const RadState &R = c->rad;
  const int64_t N = c->N, per = (int64_t)R.M * R.G;
  int64_t cells = std::min<int64_t>(N, std::max<int64_t>(1, (int64_t)(kPieceBytes / (sizeof(double) * per))));
  double *tmp = nullptr;
  while (cudaMalloc(&tmp, sizeof(double) * cells * per) != cudaSuccess) {
    cudaGetLastError();
    if (cells == 1) return rrhd_fail(RRHD_ERR_OOM, "transfer buffer allocation failed");
    cells = (cells + 1) / 2;
  }
  cudaError_t e = cudaSuccess;
  for (int64_t p = 0; p < N && e == cudaSuccess; p += cells) {
    const int64_t n = std::min(cells, N - p);
    const unsigned nb = grid_for(n * per, 256);
    const size_t bytes = sizeof(double) * n * per;
    if (to) {
      if (R.prec == RRHD_RAD_FP64)
        k_cdg_to_rows<double><<<nb, 256, 0, c->stream>>>(p, n, R.M, R.G, c->d_iperm, (const double *)array, tmp);
      else
        k_cdg_to_rows<float><<<nb, 256, 0, c->stream>>>(p, n, R.M, R.G, c->d_iperm, (const float *)array, tmp);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(to + p * per, tmp, bytes, cudaMemcpyDeviceToHost, c->stream);
    } else {
      e = cudaMemcpyAsync(tmp, from + p * per, bytes, cudaMemcpyHostToDevice, c->stream);
      if (e != cudaSuccess) break;
      if (R.prec == RRHD_RAD_FP64)
        k_rows_to_cdg<double><<<nb, 256, 0, c->stream>>>(p, n, R.M, R.G, c->d_iperm, tmp, (double *)array);
      else
        k_rows_to_cdg<float><<<nb, 256, 0, c->stream>>>(p, n, R.M, R.G, c->d_iperm, tmp, (float *)array);
      e = cudaGetLastError();
    }
  }
  const cudaError_t e2 = cudaStreamSynchronize(c->stream);
  cudaFree(tmp);
  RRHD_CUDA(e);
  RRHD_CUDA(e2);
  return RRHD_OK;
}
}  // namespace

namespace {
void drop_coupled(RadState &R) {
  for (void **p : {&R.d_I, &R.d_S, (void **)&R.d_G4, (void **)&R.d_mE, (void **)&R.d_mF, (void **)&R.d_mT,
                   (void **)&R.d_mom, (void **)&R.d_cnt}) {
    cudaFree(*p);
    *p = nullptr;
  }
  for (cudaEvent_t &e : R.ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (R.side) cudaStreamDestroy(R.side);
  R.side = nullptr;
}

// The arrays, events and side stream of the coupled step, zeroed: all of them, or (R.d_I is null) none.
rrhd_status make_coupled(rrhd_ctx *c) {
  RadState &R = c->rad;
  const size_t N = (size_t)c->N, rows = N * R.G;
  const bool fp64 = R.prec == RRHD_RAD_FP64;
  const size_t big = (fp64 ? sizeof(double) : sizeof(float)) * rows * R.M;
  const struct {
    void **p;
    size_t bytes;
  } parts[] = {{&R.d_I, big},
               {&R.d_S, big},
               {(void **)&R.d_G4, sizeof(double) * 4 * N},
               {(void **)&R.d_cnt, sizeof(unsigned long long) * 8},
               {(void **)&R.d_mE, fp64 ? sizeof(double) * rows : 0},
               {(void **)&R.d_mF, fp64 ? sizeof(double) * 3 * rows : 0},
               {(void **)&R.d_mT, fp64 ? sizeof(double) * 9 * rows : 0},
               {(void **)&R.d_mom, fp64 ? 0 : sizeof(float) * 16 * rows}};
  // a coupled step sweeps in its own arrays: the scratch is the first of them, or in the way
  if (R.d_x && R.xdirs == R.M) {
    std::swap(R.d_I, R.d_x);
    R.xdirs = 0;
  } else if (R.d_x) {
    RRHD_CUDA(cudaStreamSynchronize(c->stream));
    drop_scratch(R);
  }
  for (const auto &q : parts) {
    if (!q.bytes) continue;
    while (!*q.p && !take(q.p, q.bytes)) {
      bool freed = false;
      const rrhd_status s = give_back(c, freed);
      if (s) return s;
      if (!freed) return rrhd_fail(RRHD_ERR_OOM, "coupled-step allocation failed (%lld bytes)", (long long)q.bytes);
    }
    RRHD_CUDA(cudaMemsetAsync(*q.p, 0, q.bytes, c->stream));
  }
  for (cudaEvent_t &e : R.ev) RRHD_CUDA(cudaEventCreate(&e));
  RRHD_CUDA(cudaStreamCreateWithFlags(&R.side, cudaStreamNonBlocking));
  return fill(c, -1, false);  // with the arrays made, what else of the stream fits
}
rrhd_status alloc_coupled(rrhd_ctx *c) {
  const rrhd_status s = make_coupled(c);
  if (s) {
    cudaStreamSynchronize(c->stream);  // the zeroing of what is freed
    drop_coupled(c->rad);
  }
  return s;
}
}  // namespace

extern "C" rrhd_status rrhd_coupled_step(rrhd_ctx *c, double tau, const rrhd_coupled_opts *o, rrhd_step_stats *hs,
                                         rrhd_c2p_stats *ss) {
  RRHD_CHECK_ARG(c && o, "null argument");
  RRHD_CHECK_ARG(tau > 0, "tau must be > 0");
  RRHD_CHECK_ARG(c->part_world == 1, "the coupled step runs on a whole mesh (no rrhd_hydro_set_part split)");
  RadState &R = c->rad;
  if (!R.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  const bool fp64 = R.prec == RRHD_RAD_FP64;         // intensity and scattering integral in double
  const bool rec64 = R.prec != RRHD_RAD_FP32;        // records (geometry, opacities, sources) in double
  const bool lowrank = o->scatter == RRHD_SCATTER_LOWRANK;
  RRHD_CHECK_ARG(lowrank || (fp64 ? o->scatter == RRHD_SCATTER_FP64
                                  : (o->scatter >= RRHD_TC_BF16X3 && o->scatter <= RRHD_TC_BF16)),
                 "scatter form does not match the sweep precision");
  RRHD_CHECK_ARG((fp64 && !lowrank) ? (64 % R.G == 0) : (R.G == 1 || R.G == 2 || R.G == 4),
                 "coupled step groups: a divisor of 64 (FP64 direct sum) or 1, 2, 4 (tensor cores, low rank)");
  const int k_stall = o->k_stall ? o->k_stall : 12;
  RRHD_CHECK_ARG(k_stall > 0 && k_stall <= 40, "k_stall must be in [1, 40]");
  RRHD_CUDA(cudaSetDevice(c->device));
  rrhd_status s;
  if (!R.d_I && (s = alloc_coupled(c))) return s;
  if (!fp64 && !lowrank && (!R.tc || R.tc_form != o->scatter)) {
    if (R.tc) rrhd_scatter_tc_destroy(R.tc);
    R.tc = nullptr;
    if ((s = rrhd_scatter_tc_create(R.dirs, o->scatter, &R.tc))) return s;
    R.tc_form = o->scatter;
  }
  cudaStream_t st = c->stream;
  const int64_t N = c->N;
  // a previous step that returned early may have left its source term on the side stream
  RRHD_CUDA(cudaStreamWaitEvent(st, R.ev[4], 0));
  RRHD_CUDA(cudaEventRecord(R.ev[0], st));
  // 1. hydro step (flux, update, con2prim with fallback)
  rrhd_step_stats hst;
  const rrhd_status hstat = rrhd_hydro_step(c, tau, hs ? &hst : nullptr);
  if (hstat && hstat != RRHD_ERR_C2P) return hstat;
  if (hs) *hs = hst;
  RRHD_CUDA(cudaEventRecord(R.ev[1], st));
  double *state = c->d_state[c->cur];
  const Emission em{o->emission.temp_coef, o->emission.sigma_sb, o->emission.pi, o->emission.rad_unit};
  // 2. opacities and emission from the new primitives
  if (rec64)
    k_dyn_from_state<double><<<grid_for(N, 256), 256, 0, st>>>(N, R.G, source_words<double>(R.G, true), state,
                                                                o->absorption, o->scattering, em,
                                                                (const double *)R.d_wt, (double *)R.d_src);
  else
    k_dyn_from_state<float><<<grid_for(N, 256), 256, 0, st>>>(N, R.G, source_words<float>(R.G, true), state,
                                                               o->absorption, o->scattering, em,
                                                               (const float *)R.d_wt, (float *)R.d_src);
  RRHD_CUDA(cudaGetLastError());
  // 4. 4-force from the previous intensity's moments and the source con2prim, on the side
  // stream beside the sweep: they read the state after the opacities were taken from it and
  // the previous step's moments, and write the state and G4, none of which the sweep touches.
  RRHD_CUDA(cudaEventRecord(R.ev[3], st));
  RRHD_CUDA(cudaStreamWaitEvent(R.side, R.ev[3], 0));
  const cudaStream_t ss_st = R.side;
  k_source<<<grid_for(N, 128), 128, 0, ss_st>>>(N, R.G, state, o->absorption, o->scattering, em, R.d_mE, R.d_mF,
                                                 R.d_mT, R.d_mom, R.d_G4);
  RRHD_CUDA(cudaGetLastError());
  if (o->guess) {
    if ((s = mlp_c2p(o->guess, c->eos, c->gamma, state, state + 5, 10, R.d_G4, tau, nullptr, N, 0, k_stall, ss,
                     nullptr, nullptr, ss_st)))
      return s;
  } else {
    RRHD_CUDA(cudaMemsetAsync(R.d_cnt, 0, sizeof(unsigned long long) * 8, ss_st));
    k_source_c2p<<<grid_for(N, 256), 256, 0, ss_st>>>(N, eos_of(c), state, R.d_G4, tau, R.d_cnt);
    RRHD_CUDA(cudaGetLastError());
  }
  RRHD_CUDA(cudaEventRecord(R.ev[4], ss_st));
  // 3. sweep with the previous scattering integral
  if ((s = run_sweep_coupled(c))) return s;
  RRHD_CUDA(cudaEventRecord(R.ev[2], st));
  // the scattering below overwrites the moments the source read, and the next step reads
  // the state the source wrote: join the side stream
  RRHD_CUDA(cudaStreamWaitEvent(st, R.ev[4], 0));
  RRHD_CUDA(cudaEventRecord(R.ev[5], st));
  if (!o->guess && ss) {
    unsigned long long h[8];
    RRHD_CUDA(cudaMemcpyAsync(h, R.d_cnt, sizeof h, cudaMemcpyDeviceToHost, st));
    RRHD_CUDA(cudaStreamSynchronize(st));
    ss->n_ok = (int64_t)h[0];
    ss->n_fallback = 0;
    ss->n_failed = (int64_t)h[1];
    ss->newton_iters = (int64_t)h[2];
    ss->max_iters = (int32_t)h[3];
  }
  // 5. scattering integral and moments of the new intensity, for the next step
  if (lowrank) {
    if (fp64) {
      if ((s = scatter_lowrank_fp64(R.dirs, (const double *)R.d_I, (double *)R.d_S, R.d_mE, R.d_mF, R.d_mT, N, R.G,
                                    st)))
        return s;
    } else if ((s = scatter_lowrank_fp32(R.dirs, (const float *)R.d_I, (float *)R.d_S, R.d_mom, N, R.G, st))) {
      return s;
    }
  } else if (fp64) {
    if ((s = scatter_fp64_cdg(R.dirs, (const double *)R.d_I, (double *)R.d_S, N, R.G, false, st))) return s;
    if ((s = moments_fp64_cdg(R.dirs, (const double *)R.d_I, R.d_mE, R.d_mF, R.d_mT, N, R.G, st))) return s;
  } else {
    if ((s = scatter_tc_cdg(R.tc, (const float *)R.d_I, (float *)R.d_S, R.d_mom, N, R.G, st))) return s;
  }
  RRHD_CUDA(cudaEventRecord(R.ev[6], st));
  return hstat;
}

extern "C" rrhd_status rrhd_coupled_phase_ms(rrhd_ctx *c, float *ms) {
  RRHD_CHECK_ARG(c && ms, "null argument");
  RadState &R = c->rad;
  if (!R.ev[0]) return rrhd_fail(RRHD_ERR_STATE, "no coupled step has run");
  RRHD_CUDA(cudaSetDevice(c->device));
  RRHD_CUDA(cudaEventSynchronize(R.ev[6]));
  // hydro (with the opacities), sweep, source (side stream, beside the sweep), scattering
  RRHD_CUDA(cudaEventElapsedTime(ms + 0, R.ev[0], R.ev[3]));
  RRHD_CUDA(cudaEventElapsedTime(ms + 1, R.ev[3], R.ev[2]));
  RRHD_CUDA(cudaEventElapsedTime(ms + 2, R.ev[3], R.ev[4]));
  RRHD_CUDA(cudaEventElapsedTime(ms + 3, R.ev[5], R.ev[6]));
  return RRHD_OK;
}

namespace {
// The scattering integral and moments the last coupled step left (FP32, cell-direction-group
// layout, moments [rows][16]) against their FP64 values from the same FP32 intensity, on
// every stride-th cell: one thread per (sampled cell, group) loops over the output
// directions (S relative to itself) and forms the ten moments (F and T relative to E).
// err: {max S, sum of squared S errors, count, max moments} as doubles, the maxima as the
// bit patterns of non-negative doubles.
__global__ void k_coupled_scatter_error(int64_t ncell, int64_t stride, int M, int G, const double *__restrict__ K,
                                        const double *__restrict__ w, const double *__restrict__ a, double area,
                                        const float *__restrict__ I, const float *__restrict__ S,
                                        const float *__restrict__ mom, double *err) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= ncell * G) return;
  const int64_t c = (t / G) * stride;
  const int g = (int)(t % G);
  const float *Ic = I + c * (int64_t)M * G + g;
  double emax = 0.0, esq = 0.0;
  for (int o = 0; o < M; o++) {
    double ref = 0.0;
    for (int d = 0; d < M; d++) ref += K[(int64_t)d * M + o] * (double)Ic[(int64_t)d * G];  // K[d][o] = Gamma a_d / A
    const double e = fabs((double)S[(c * M + o) * G + g] - ref) / fabs(ref);
    if (ref != 0.0) {
      emax = fmax(emax, e);
      esq += e * e;
    }
  }
  double m[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int d = 0; d < M; d++) {
    const double wi = a[d] / area * (double)Ic[(int64_t)d * G];
    const double x = w[3 * d], y = w[3 * d + 1], z = w[3 * d + 2];
    const double f[10] = {1.0, x, y, z, x * x, x * y, x * z, y * y, y * z, z * z};
    for (int k = 0; k < 10; k++) m[k] += f[k] * wi;
  }
  double mmax = 0.0;
  if (mom && m[0] != 0.0) {
    const float *mr = mom + 16 * (c * G + g);
    mmax = fabs((double)mr[0] - m[0]) / fabs(m[0]);
    for (int k = 1; k < 10; k++) mmax = fmax(mmax, fabs((double)mr[k] - m[k]) / fabs(m[0]));
  }
  atomicMax(reinterpret_cast<unsigned long long *>(err), (unsigned long long)__double_as_longlong(emax));
  atomicAdd(err + 1, esq);
  atomicAdd(err + 2, (double)M);
  atomicMax(reinterpret_cast<unsigned long long *>(err + 3), (unsigned long long)__double_as_longlong(mmax));
}
}  // namespace

extern "C" rrhd_status rrhd_coupled_scatter_error(rrhd_ctx *c, int64_t sample_cells, double *max_rel, double *rms_rel,
                                                  double *moments_max) {
  RRHD_CHECK_ARG(c && sample_cells > 0, "bad argument");
  RadState &R = c->rad;
  if (!R.ready || !R.d_I) return rrhd_fail(RRHD_ERR_STATE, "no coupled step has run");
  if (R.prec == RRHD_RAD_FP64) return rrhd_fail(RRHD_ERR_STATE, "the FP64 form has no reduced-precision scattering");
  RRHD_CUDA(cudaSetDevice(c->device));
  const int64_t N = c->N;
  const int64_t stride = std::max<int64_t>(1, N / sample_cells);
  const int64_t ncell = (N + stride - 1) / stride;
  double *d_err = nullptr;
  RRHD_CUDA(cudaMalloc(&d_err, 4 * sizeof(double)));
  double h[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemsetAsync(d_err, 0, 4 * sizeof(double), c->stream);
  if (e == cudaSuccess) {
    k_coupled_scatter_error<<<grid_for(ncell * R.G, 128), 128, 0, c->stream>>>(
        ncell, stride, R.M, R.G, R.dirs->d_K, R.dirs->d_w, R.dirs->d_a, R.dirs->full_area, (const float *)R.d_I,
        (const float *)R.d_S, R.d_mom, d_err);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d_err, sizeof h, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(d_err);
  RRHD_CUDA(e);
  if (max_rel) *max_rel = h[0];
  if (rms_rel) *rms_rel = h[2] > 0 ? std::sqrt(h[1] / h[2]) : 0.0;
  if (moments_max) *moments_max = h[3];
  return RRHD_OK;
}

// ---------------------------------------------------------------- caller-array pieces of the coupled step
// (for a step composed over ranks, where each piece runs on a rank's share of cells or rows)
namespace {
// alpha = a rho, betta = b rho, Q_g = B(T) / kRadiation / G from primitives W [n][stride]
// (the opacity and emission rule of the coupled step, as k_dyn_from_state forms them).
__global__ void k_rad_opacities(int64_t n, int64_t stride, int G, const double *W, double a_coef, double b_coef,
                                Emission em, double *alpha, double *betta, double *Q) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  const double rho = W[stride * c], prs = W[stride * c + 4];
  alpha[c] = a_coef * rho;
  betta[c] = b_coef * rho;
  const double q = planck_B(em, rho, prs) / em.rad_unit / (double)G;
  for (int g = 0; g < G; g++) Q[c * G + g] = q;
}

// 4-force per cell from the FP64 moments of its G rows (E [n G], F [n G][3], T [n G][9]),
// summed over the groups in order as k_source does.
__global__ void k_rad_source_rows(int64_t n, int64_t stride, int G, const double *W, double a_coef, double b_coef,
                                  Emission em, const double *mE, const double *mF, const double *mT, double *G4) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  double E = 0, F[3] = {0, 0, 0}, Tm[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int g = 0; g < G; g++) {
    const int64_t r = c * G + g;
    E += mE[r];
#pragma unroll
    for (int q = 0; q < 3; q++) F[q] += mF[3 * r + q];
#pragma unroll
    for (int q = 0; q < 9; q++) Tm[q] += mT[9 * r + q];
  }
  double w[5];
#pragma unroll
  for (int q = 0; q < 5; q++) w[q] = W[stride * c + q];
  double out[4];
  rad_source_cell(em, w, a_coef * w[0], b_coef * w[0], E, F, Tm, out);
#pragma unroll
  for (int q = 0; q < 4; q++) G4[4 * c + q] = out[q];
}

// U.E += tau G0, U.S += tau G (radRHD_main.cpp:117-126), then GetPhysValueStab from its own
// guess without fallback, on caller arrays; cnt as in k_source_c2p.
__global__ void k_rad_source_c2p(int64_t n, int64_t stride, Eos eos, double *U, double *W, const double *G4,
                                 double tau, unsigned long long *cnt) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  unsigned long long ok = 0, failed = 0, iters = 0;
  if (c < n) {
    double u[5], w[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      u[q] = U[stride * c + q];
      w[q] = W[stride * c + q];
    }
    u[4] += tau * G4[4 * c];
    u[1] += tau * G4[4 * c + 1];
    u[2] += tau * G4[4 * c + 2];
    u[3] += tau * G4[4 * c + 3];
    int it = 0;
    const int code = c2p_from(eos, u, w, 0.0, false, &it);
    ok = code == 0;
    failed = code != 0;
    iters = (unsigned long long)it;
#pragma unroll
    for (int q = 0; q < 5; q++) {
      U[stride * c + q] = u[q];
      W[stride * c + q] = w[q];
    }
  }
  unsigned long long mx = iters;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ok += __shfl_xor_sync(0xffffffffu, ok, o);
    failed += __shfl_xor_sync(0xffffffffu, failed, o);
    iters += __shfl_xor_sync(0xffffffffu, iters, o);
    const unsigned long long m2 = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = m2 > mx ? m2 : mx;
  }
  if ((threadIdx.x & 31) == 0 && (ok | failed)) {
    atomicAdd(cnt + 0, ok);
    atomicAdd(cnt + 1, failed);
    atomicAdd(cnt + 2, iters);
    atomicMax(cnt + 3, mx);
  }
}
}  // namespace

extern "C" rrhd_status rrhd_rad_opacities(const rrhd_emission *em, const double *W, int64_t stride, int64_t n,
                                          double absorption, double scattering, int32_t groups, double *alpha,
                                          double *betta, double *Q, void *stream) {
  RRHD_CHECK_ARG(em && W && alpha && betta && Q && n >= 0 && stride >= 5 && groups >= 1, "bad arguments");
  if (n == 0) return RRHD_OK;
  const Emission e{em->temp_coef, em->sigma_sb, em->pi, em->rad_unit};
  k_rad_opacities<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(n, stride, groups, W, absorption, scattering, e,
                                                                      alpha, betta, Q);
  RRHD_CUDA(cudaGetLastError());
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_source_rows(const rrhd_emission *em, const double *W, int64_t stride, int64_t n,
                                            double absorption, double scattering, int32_t groups, const double *E,
                                            const double *F, const double *T, double *G4, void *stream) {
  RRHD_CHECK_ARG(em && W && E && F && T && G4 && n >= 0 && stride >= 5 && groups >= 1, "bad arguments");
  if (n == 0) return RRHD_OK;
  const Emission e{em->temp_coef, em->sigma_sb, em->pi, em->rad_unit};
  k_rad_source_rows<<<grid_for(n, 128), 128, 0, (cudaStream_t)stream>>>(n, stride, groups, W, absorption, scattering,
                                                                        e, E, F, T, G4);
  RRHD_CUDA(cudaGetLastError());
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_source_con2prim(int32_t eos, double gamma, double *U, double *W, int64_t stride,
                                                const double *G4, double tau, int64_t n, rrhd_c2p_stats *stats,
                                                void *stream) {
  RRHD_CHECK_ARG(U && W && G4 && n >= 0 && stride >= 5 && (eos == 1 || eos == 2), "bad arguments");
  if (n == 0) {
    if (stats) *stats = rrhd_c2p_stats{0, 0, 0, 0, 0};
    return RRHD_OK;
  }
  cudaStream_t st = (cudaStream_t)stream;
  Eos e;
  e.eos = eos;
  e.g1 = gamma;
  e.gg = gamma / (gamma - 1.0);
  unsigned long long *cnt = nullptr;
  RRHD_CUDA(cudaMallocAsync(&cnt, 4 * sizeof(unsigned long long), st));
  cudaError_t err = cudaMemsetAsync(cnt, 0, 4 * sizeof(unsigned long long), st);
  if (err == cudaSuccess) {
    k_rad_source_c2p<<<grid_for(n, 256), 256, 0, st>>>(n, stride, e, U, W, G4, tau, cnt);
    err = cudaGetLastError();
  }
  unsigned long long h[4] = {0, 0, 0, 0};
  if (err == cudaSuccess && stats) err = cudaMemcpyAsync(h, cnt, sizeof h, cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(cnt, st);
  if (err == cudaSuccess && stats) err = cudaStreamSynchronize(st);
  RRHD_CUDA(err);
  if (stats) {
    stats->n_ok = (int64_t)h[0];
    stats->n_fallback = 0;
    stats->n_failed = (int64_t)h[1];
    stats->newton_iters = (int64_t)h[2];
    stats->max_iters = (int32_t)h[3];
  }
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_get(rrhd_ctx *c, int32_t what, double *out) {
  RRHD_CHECK_ARG(c && out, "null argument");
  RadState &R = c->rad;
  RRHD_CHECK_ARG(what == RRHD_RAD_I || what == RRHD_RAD_S || what == RRHD_RAD_G4 || what == RRHD_RAD_MOM,
                 "bad array id");
  if (!R.ready || !R.d_I) return rrhd_fail(RRHD_ERR_STATE, "no coupled step has run");
  RRHD_CUDA(cudaSetDevice(c->device));
  if (what == RRHD_RAD_I || what == RRHD_RAD_S) return move_rows(c, what == RRHD_RAD_I ? R.d_I : R.d_S, out, nullptr);
  const int64_t N = c->N;
  const int64_t width = what == RRHD_RAD_G4 ? 4 : 10 * (int64_t)R.G;
  double *tmp = nullptr;
  RRHD_CUDA(cudaMalloc(&tmp, sizeof(double) * N * width));
  if (what == RRHD_RAD_MOM)
    k_mom_to_rows<<<grid_for(N * R.G, 256), 256, 0, c->stream>>>(N, R.G, c->d_perm, R.d_mom ? nullptr : R.d_mE,
                                                                  R.d_mF, R.d_mT, R.d_mom, tmp);
  else
    k_rows_to_host_order<double><<<grid_for(N * width, 256), 256, 0, c->stream>>>(N, width, c->d_perm, R.d_G4, tmp);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, tmp, sizeof(double) * N * width, cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  cudaFree(tmp);
  RRHD_CUDA(e);
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_rad_set(rrhd_ctx *c, int32_t what, const double *in) {
  RRHD_CHECK_ARG(c && in, "null argument");
  RadState &R = c->rad;
  RRHD_CHECK_ARG(what == RRHD_RAD_I || what == RRHD_RAD_S, "bad array id");
  if (!R.ready) return rrhd_fail(RRHD_ERR_STATE, "rrhd_rad_setup has not run");
  RRHD_CUDA(cudaSetDevice(c->device));
  rrhd_status s;
  if (!R.d_I && (s = alloc_coupled(c))) return s;
  return move_rows(c, what == RRHD_RAD_I ? R.d_I : R.d_S, nullptr, in);
}
