// Image-plane ray tracing: which surface triangle (or analytic body) each ray of the
// picture plane meets first, and the image and light-curve value built from it.
//
// Reference: cuda/src/ray_tracing/cuda_ray_calc.cu (RayTracing, RayTracing_Phl1445,
// InnerRayTracing, RayTracingGrid: for each ray the nearest triangle by Moeller-Trumbore,
// RayIntersectsTriangle :10-44), cuda/src/ray_tracing/cuda_ray_geo_intersect.cu (the
// Roche-lobe root search and the accretor sphere / disk test) as launched by
// cuda/src/ray_tracing/cuda_ray_interface.cu, and the per-frame image and light curve of
// solvers/ray_tracing/src/ray_tracing_calc_illum.cpp (MakeIllumAndCurve / MakeEnergyAndCurve).
//
// Parity: this translation unit is compiled without FMA contraction and every quantity is
// formed in the reference's operation order (Eigen's cross product component by component,
// dot products as (x0 + x1) + x2, IEEE division and square root), so distances are the
// reference's bit for bit and the nearest-hit choice -- strictly closer than the best so
// far, i.e. the first triangle in input order among equal distances -- is the same.
//
// Layout: the surface lives on the device as [n][9] doubles {A, B - A, C - A} plus the
// triangles' ids; rays as the reference's Ray_t records {orig[3], direction[3]}.  A block
// of 256 rays streams the triangles through shared memory in tiles of 256 (a thread
// stages one triangle), every thread testing its ray against each staged triangle
// (broadcast reads).  Work is rays x triangles FP64 tests, most rejected by the
// barycentric u test.
// Rays of one direction (an image plane) do not do that work: see "image-plane bins" below.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "rrhd_internal.h"

struct rrhd_ray_surface {
  int device = 0;
  int64_t n = 0;
  double *tri = nullptr;  // [n][9] {A, E1 = B - A, E2 = C - A}
  int32_t *ids = nullptr;
  // image-plane bins (one trace call at a time per surface), one allocation that begins at bins
  int32_t *bins = nullptr;    // [NB + 1] counts, then offsets
  int32_t *cursor = nullptr;  // [NB]
  int32_t *entries = nullptr; // [max_bins(n) * n] triangle indices by bin
  int32_t *glist = nullptr;   // [n] triangles every ray tests
  double *pack = nullptr;     // [n][kPack] triangles as the binned pass tests them
  long long *ctrl = nullptr;  // [8]: uniform flag, global count, ray box keys (x0, x1, y0, y1), listed rays
  double *ray2d = nullptr;    // [cap][2], then the listed rays [cap]
  int64_t ray_cap = 0;
};

namespace {

namespace cg = cooperative_groups;

constexpr int kRayThreads = 256;
constexpr int kTile = 256;
// A ray's own thread tests a bin of up to kHeavy triangles, a warp a longer one.  A longer chain a thread
// is more latency, a shorter one more warps half empty: with 44,032 triangles and 180,000 rays
// a trace takes 75 us at 32, 86 at 16 and 92 at 64.
constexpr int kHeavy = 32;
constexpr double kEps = 1e-10;  // cuda_ray_calc.cu:12
constexpr int kNone = -1, kDisk = -2, kSphere = -3, kRoche = -4;  // ray_tracing_const.h e_ray_intersect_code

// what the binned pass leaves for the rays that a warp takes up
struct RayBins {
  const long long *ctrl;
  const double *ray2d, *pack;
  const int32_t *bins, *entries;
  const int64_t *listed;
};

__device__ __forceinline__ double dot3(const double *a, const double *b) {
  return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}
__device__ __forceinline__ void cross3(const double *a, const double *b, double *r) {
  r[0] = a[1] * b[2] - a[2] * b[1];
  r[1] = a[2] * b[0] - a[0] * b[2];
  r[2] = a[0] * b[1] - a[1] * b[0];
}

// FaceCell records {int32 face_id; 4 bytes padding; double A[3], B[3], C[3]} -> {A, B - A, C - A}
__global__ void k_surface_prep(const unsigned char *fc, int64_t n, double *tri, int32_t *ids) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const unsigned char *r = fc + 80 * i;
  const double *v = reinterpret_cast<const double *>(r + 8);
  ids[i] = *reinterpret_cast<const int32_t *>(r);
  double *t = tri + 9 * i;
  for (int k = 0; k < 3; k++) {
    t[k] = v[k];
    t[3 + k] = v[3 + k] - v[k];
    t[6 + k] = v[6 + k] - v[k];
  }
}

// Rosh (cuda_ray_geo_intersect.cu:22-42)
__device__ double rosh(const double *o, const double *a, double t) {
  constexpr double max_potential = -1.82547, m = 0.8795180722891566;
  const double x1 = o[0] + a[0] * t;
  const double x2 = (o[1] + a[1] * t) * (o[1] + a[1] * t);
  const double x3 = (o[2] + a[2] * t) * (o[2] + a[2] * t);
  return -max_potential - ((x1 - m) * (x1 - m) + x2 + x3) * 0.5 - m / sqrt((x1 - 1) * (x1 - 1) + x2 + x3) -
         (1 - m) / sqrt(x1 * x1 + x2 + x3);
}

// FindRoshRoots + GetIntersectionWithRosh (:44-86): sign changes of the potential at 1001
// points of t in [-3, 3]; with 4 or 6 of them the second is the entry into the donor's lobe
// if it lies at x < 0.3.  Only the first 6 roots are kept (the reference's array size); the
// roots come out ascending, so the reference's sort leaves them as they are.
__device__ int roche(const double *o, const double *dir, double *dist) {
  constexpr int n = 1001;
  constexpr double a = -3, b = 3;
  const double step = (b - a) / (n - 1);
  double r1 = 0;
  int size = 0;
  double fi_1 = rosh(o, dir, a + 0 * step);
  for (int i = 1; i < n; ++i) {
    const double fi_2 = rosh(o, dir, a + (i)*step);
    if (fi_1 * fi_2 < 0) {
      if (size == 1) r1 = ((2 * a + (2. * i - 1) * step) / 2.);
      size++;
    }
    fi_1 = fi_2;
  }
  if (size == 6 || size == 4) {
    if (o[0] + dir[0] * r1 < 0.3) {
      *dist = r1;
      return kRoche;
    }
  }
  *dist = -1;
  return kNone;
}

// IntersectionWithPlane + GetIntersectionWithSphereOfDisk (:88-169); the reference
// returns "sphere" as soon as the ray meets the accretor sphere.
__device__ int sphere_disk(const double *o, const double *n) {
  const double A[3] = {1, 0, 0}, B[3] = {0, 0.9928768384869221, 0.11914522061843064}, C[3] = {2, 0, 0};
  const double pa = A[1] * (B[2] - C[2]) + B[1] * (C[2] - A[2]) + C[1] * (A[2] - B[2]);
  const double pb = A[0] * (C[2] - B[2]) + B[0] * (A[2] - C[2]) + C[0] * (B[2] - A[2]);
  const double pc = A[0] * (B[1] - C[1]) + B[0] * (C[1] - A[1]) + C[0] * (A[1] - B[1]);
  const double pd = A[0] * (C[1] * B[2] - B[1] * C[2]) + B[0] * (A[1] * C[2] - C[1] * A[2]) +
                    C[0] * (B[1] * A[2] - A[1] * B[2]);
  const double t = -(pa * o[0] + pb * o[1] + pc * o[2] + pd) / (pa * n[0] + pb * n[1] + pc * n[2]);
  const double res[3] = {n[0] * t + o[0], n[1] * t + o[1], n[2] * t + o[2]};
  const double v1[3] = {1, 0, 0}, v2[3] = {0, -0.992877, -0.119145};
  double l0 = 0, l1 = 0;
  for (int k = 0; k < 3; k++) {
    l0 += (res[k]) * v1[k];
    l1 += (res[k]) * v2[k];
  }
  const double lx = l0 - 1, ly = l1 - 0;
  const double lsq = lx * lx + ly * ly;
  const double An = dot3(n, n);
  const double oc[3] = {o[0] - 1, o[1] - 0, o[2] - 0};
  const double proj = dot3(oc, n);
  constexpr double r_s = 0.01, r_in = 0.01, r_ex = 0.06;  // ray_tracing_const.h
  const double radical = 4. * (proj * proj - An * (1 - 2 * o[0] + dot3(o, o) - r_s * r_s));
  if (radical >= 0) return kSphere;
  if (lsq < r_ex * r_ex && (lsq > r_in * r_in)) return kDisk;
  return kNone;
}

// A triangle as the binned pass tests it for the one direction of its rays: {A, det}, {h, E2.x},
// {E1, E2.y}, {E2.z, bins, -, -}, h = dir x E2 and det = E1 . h, a 32-byte load each.  The
// lanes of a warp test different triangles, so what a test costs is its requests, one a lane
// and load: two for a triangle rejected by u (nine from the [n][9] array).
constexpr int kPack = 16;
__device__ __forceinline__ void load4(const double *p, double *x) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
               : "l"(p));
}
__device__ __forceinline__ void store4(double *p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// The reference's test of one triangle, keeping the smallest (distance, input index).  A
// triangle whose u or u + v is outside [0, 1] by more than rounding is left before the
// division: with det's sign taken off, u below -1e-14 or u + v above 1 + 2^-40 (the reference's
// own values differ from these quotients by a few 2^-53); the rest meet its comparisons.
struct Front {  // what u needs
  double A[4], h[4];
};
__device__ __forceinline__ void load_front(const double *T, Front &f) {
  load4(T, f.A);
  load4(T + 4, f.h);
}
__device__ __forceinline__ void nearest(const Front &f, const double *T, int64_t t, const double *o, const double *dir,
                                        double &best, int64_t &best_t) {
  const double det = f.A[3];
  const double s[3] = {o[0] - f.A[0], o[1] - f.A[1], o[2] - f.A[2]};
  const double un = dot3(s, f.h), lo = -1e-14 * fabs(det), hi = (1.0 + 9.094947017729282e-13) * fabs(det);
  const double us = det < 0.0 ? -un : un;
  if (us < lo || us > hi) return;
  double e1[4], q[3];
  load4(T + 8, e1);
  cross3(s, e1, q);
  const double vn = dot3(dir, q), vs = det < 0.0 ? -vn : vn;
  if (vs < lo || us + vs > hi) return;
  const double inv_det = 1.0 / det;
  const double u = inv_det * un;
  if (u < 0.0 || u > 1.0) return;
  const double v = inv_det * vn;
  if (v < 0.0 || u + v > 1.0) return;
  const double e2[3] = {f.h[3], e1[3], T[12]};
  const double d = inv_det * dot3(e2, q);
  if (d > 0.0 && (d < best || (d == best && best_t >= 0 && t < best_t))) {
    best = d;
    best_t = t;
  }
}
// the triangles entries[e0], entries[e0 + step], ...: two in flight
__device__ __forceinline__ void nearest_of(const double *pack, const int32_t *entries, int e0, int e1, int step,
                                           const double *o, const double *dir, double &best, int64_t &best_t) {
  for (int e = e0; e < e1; e += 2 * step) {
    const bool two = e + step < e1;
    const int32_t t0 = entries[e], t1 = two ? entries[e + step] : t0;
    const double *T0 = pack + kPack * (int64_t)t0, *T1 = pack + kPack * (int64_t)t1;
    Front f0, f1;
    load_front(T0, f0);
    load_front(T1, f1);
    nearest(f0, T0, t0, o, dir, best, best_t);
    if (two) nearest(f1, T1, t1, o, dir, best, best_t);
  }
}

// A warp to each ray that k_ray_trace_binned listed: the rest of its tests, a lane per triangle.
__device__ __forceinline__ void trace_listed(const double *__restrict__ rays,
                                             const int32_t *__restrict__ ids, const RayBins &w,
                                             int32_t *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t n = w.ctrl[6], warps = (int64_t)gridDim.x * (kRayThreads / 32);
  for (int64_t i = blockIdx.x * (int64_t)(kRayThreads / 32) + threadIdx.x / 32; i < n; i += warps) {
    const int64_t r = w.listed[i];
    const double o[3] = {rays[6 * r], rays[6 * r + 1], rays[6 * r + 2]};
    const double dir[3] = {rays[6 * r + 3], rays[6 * r + 4], rays[6 * r + 5]};
    double d = w.ray2d[2 * r];
    const long long kt = __double_as_longlong(w.ray2d[2 * r + 1]);
    const int k = (int)(kt >> 32), e1 = w.bins[k + 1];
    int64_t t = (int32_t)(uint32_t)kt;
    nearest_of(w.pack, w.entries, w.bins[k] + lane, e1, 32, o, dir, d, t);
    // a lane without a hit of its own holds the distance the ray came with
    for (int m = 16; m > 0; m >>= 1) {
      const double d2 = __shfl_xor_sync(0xffffffffu, d, m);
      const int64_t t2 = __shfl_xor_sync(0xffffffffu, t, m);
      if (t2 >= 0 && (d2 < d || (d2 == d && t >= 0 && t2 < t))) d = d2, t = t2;
    }
    if (lane == 0 && t >= 0) out[r] = ids[t];
  }
}

// mode 0 RayTracing / 3 RayTracingGrid: nearest triangle; 1 RayTracing_Phl1445: the
// Roche lobe first, triangles only if nearer; 2 InnerRayTracing: accretor sphere or disk,
// else the nearest triangle.
//
// Two savings that leave every decision the reference's:
//  * a block whose rays share one direction (every ray of an image plane does) stages
//    h = dir x (C - A) and det = (B - A) . h once per triangle with the tile instead of once
//    per ray and triangle (the same operations on the same operands, so the same bits);
//  * u = fl(fl(1 / det) (s . h)) is first settled without the division where it is
//    certain: u < 0 exactly when s . h is non-zero with the sign opposite to det, and
//    u > 1 certainly when |s . h| > |det| (1 + 2^-48) (two roundings move it by less than
//    2^-52); only the remaining tests divide, and then exactly as the reference does.
constexpr int kRec = 16;  // doubles per staged triangle: A, B - A, C - A, h, det, padding
__global__ void __launch_bounds__(kRayThreads)
    k_ray_trace(const double *__restrict__ rays, int64_t M, const double *__restrict__ tri,
                const int32_t *__restrict__ ids, int64_t n, int mode, int32_t *__restrict__ out,
                RayBins binned) {
  if (binned.ctrl && binned.ctrl[0] != 0) {  // every ray shares one direction: the image-plane bins answered
    trace_listed(rays, ids, binned, out);
    return;
  }
  __shared__ __align__(16) double st[kTile * kRec];
  __shared__ int32_t sid[kTile];
  __shared__ double dir0[3];
  const int64_t r0 = blockIdx.x * (int64_t)kRayThreads;
  const int64_t r = r0 + threadIdx.x;
  const bool live = r < M;
  double o[3] = {0, 0, 0}, dir[3] = {0, 0, 1};
  if (live)
    for (int k = 0; k < 3; k++) {
      o[k] = rays[6 * r + k];
      dir[k] = rays[6 * r + 3 + k];
    }
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; k++) dir0[k] = dir[k];
  __syncthreads();
  const bool uni = __syncthreads_and(!live || (__double_as_longlong(dir[0]) == __double_as_longlong(dir0[0]) &&
                                               __double_as_longlong(dir[1]) == __double_as_longlong(dir0[1]) &&
                                               __double_as_longlong(dir[2]) == __double_as_longlong(dir0[2])));
  int32_t best_id = kNone;
  double best = 1e10;
  bool done = !live;
  if (live && mode == 1) {
    double rd;
    if (roche(o, dir, &rd) != kNone) {
      best = rd;
      best_id = kRoche;
    }
  } else if (live && mode == 2) {
    const int code = sphere_disk(o, dir);
    if (code != kNone) {
      best_id = code;
      done = true;
    }
  }
  constexpr double kHi = 1.0 + 3.552713678800501e-15;  // 1 + 2^-48
  for (int64_t t0 = 0; t0 < n; t0 += kTile) {
    const int nt = n - t0 < kTile ? (int)(n - t0) : kTile;
    __syncthreads();
    if (threadIdx.x < nt) {
      const double *g = tri + 9 * (t0 + threadIdx.x);
      double *T = st + kRec * threadIdx.x;
      for (int k = 0; k < 9; k++) T[k] = g[k];
      if (uni) {
        double h[3];
        cross3(dir0, T + 6, h);
        T[9] = h[0], T[10] = h[1], T[11] = h[2];
        T[12] = dot3(T + 3, h);
      }
      sid[threadIdx.x] = ids[t0 + threadIdx.x];
    }
    __syncthreads();
    if (done) continue;
    for (int j = 0; j < nt; j++) {
      const double *A = st + kRec * j, *e1 = A + 3, *e2 = A + 6;
      double h[3], det;
      if (uni) {
        h[0] = A[9], h[1] = A[10], h[2] = A[11];
        det = A[12];
      } else {
        cross3(dir, e2, h);
        det = dot3(e1, h);
      }
      if (det > -kEps && det < kEps) continue;
      const double s[3] = {o[0] - A[0], o[1] - A[1], o[2] - A[2]};
      const double un = dot3(s, h);
      if (un != 0.0 && ((un < 0.0) != (det < 0.0))) continue;  // u < 0
      if (fabs(un) > fabs(det) * kHi) continue;                // u > 1
      const double inv_det = 1.0 / det;
      const double u = inv_det * un;
      if (u < 0.0 || u > 1.0) continue;
      double q[3];
      cross3(s, e1, q);
      const double v = inv_det * dot3(dir, q);
      if (v < 0.0 || u + v > 1.0) continue;
      const double d = inv_det * dot3(e2, q);
      if (d > 0.0 && d < best) {
        best = d;
        best_id = sid[j];
      }
    }
  }
  if (live) out[r] = best_id;
}

// ---------------------------------------------------------------- image-plane bins
// When every ray of a call has the same direction (an image plane), each ray tests only the
// triangles whose projection onto the plane normal to that direction can contain the ray's
// projected origin, instead of all of them; the test itself is unchanged, so the answer is
// the brute-force one.  Soundness: a triangle the reference accepts for a ray contains the
// ray's projected origin up to the rounding of its u, v (a few 1e-16 relative, amplified by
// at most 1e6 for triangles neither sliver-shaped nor seen edge-on), and its projected box is
// widened by 1e-7 of the scene size; slivers (sin of the corner angle < 1e-3), triangles seen
// within 1e-3 of edge-on and triangles covering more than max_bins(n) bins go to a list every ray
// tests; triangles with |det| < 1e-10 never hit (the reference rejects them as parallel).  The
// nearest hit is the smallest (distance, input index), which is what the reference's strictly-
// closer loop in input order returns, so the bins need no order.
constexpr int kGX = 256, kGY = 128, kNB = kGX * kGY;
// A triangle that covers more bins goes to the every-ray list: kMaxBins for a surface of many
// triangles, as many as kEntries entries allow for one of few, up to kMostBins.
// Every ray pays for a triangle of that list, its bins are paid for once: 1,344 triangles, of
// which 288 cover more than 128 bins, are traced in 53 us so, in 229 with 128 for every size.
constexpr int kMaxBins = 128, kMostBins = 2048;
constexpr int64_t kEntries = 4 << 20;
inline int max_bins(int64_t n) {
  return (int)std::min<int64_t>(kMostBins, std::max<int64_t>(kMaxBins, kEntries / std::max<int64_t>(n, 1)));
}
constexpr int64_t kMaxBinnedTriangles = 0x7fffffff / kMaxBins;  // bin offsets stay within int32
// warps that bin a surface of up to 32 times as many triangles: about one a scheduler slot
constexpr int64_t kSpreadWarps = 4096;
constexpr double kMargin = 1e-7;

__device__ __forceinline__ long long dkey(double x) {  // order-preserving double -> int64
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : b ^ 0x7fffffffffffffffll;
}
__device__ __forceinline__ double dval(long long k) {
  return __longlong_as_double(k >= 0 ? k : k ^ 0x7fffffffffffffffll);
}

// orthonormal u, v spanning the plane normal to d
__device__ void plane_basis(const double *d, double *u, double *v) {
  const double ax = fabs(d[0]), ay = fabs(d[1]), az = fabs(d[2]);
  const double e[3] = {(ax <= ay && ax <= az) ? 1.0 : 0.0, (!(ax <= ay && ax <= az) && ay <= az) ? 1.0 : 0.0,
                       (!(ax <= ay && ax <= az) && !(ay <= az)) ? 1.0 : 0.0};
  cross3(d, e, u);
  const double nu = sqrt(dot3(u, u));
  for (int k = 0; k < 3; k++) u[k] /= nu;
  cross3(d, u, v);
  const double nv = sqrt(dot3(v, v));
  for (int k = 0; k < 3; k++) v[k] /= nv;
}

struct Box {
  double x0, x1, y0, y1, ix, iy, margin;
};
__device__ Box ray_box(const long long *ctrl) {
  Box b;
  b.x0 = dval(ctrl[2]), b.x1 = dval(ctrl[3]), b.y0 = dval(ctrl[4]), b.y1 = dval(ctrl[5]);
  b.ix = b.x1 > b.x0 ? kGX / (b.x1 - b.x0) : 0.0;
  b.iy = b.y1 > b.y0 ? kGY / (b.y1 - b.y0) : 0.0;
  b.margin = kMargin * (1.0 + fmax(fmax(fabs(b.x0), fabs(b.x1)), fmax(fabs(b.y0), fabs(b.y1))));
  return b;
}
__device__ __forceinline__ int bin_x(const Box &b, double x) {
  const double f = floor((x - b.x0) * b.ix);
  return f < 0 ? 0 : f > kGX - 1 ? kGX - 1 : (int)f;
}
__device__ __forceinline__ int bin_y(const Box &b, double y) {
  const double f = floor((y - b.y0) * b.iy);
  return f < 0 ? 0 : f > kGY - 1 ? kGY - 1 : (int)f;
}

__global__ void k_bins_reset(int32_t *bins, long long *ctrl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= kNB) bins[i] = 0;
  if (i == 0) {
    ctrl[0] = 1;  // uniform until a ray says otherwise
    ctrl[1] = ctrl[6] = 0;
    ctrl[2] = ctrl[4] = 0x7fffffffffffffffll;
    ctrl[3] = ctrl[5] = -0x7fffffffffffffffll - 1;
  }
}

// Projected ray origins, their box, and whether all directions equal ray 0's.  Bound by the
// atomics on the four words of the box, which one address takes one at a time: a block reduces
// its rays first and sends four (180,000 rays: 6.5 us, 18.5 with four a warp).
__global__ void __launch_bounds__(256) k_rays_project(const double *__restrict__ rays, int64_t M, double *ray2d,
                                                      long long *ctrl) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const double d0[3] = {rays[3], rays[4], rays[5]};
  double u[3], v[3];
  plane_basis(d0, u, v);
  long long kx0 = 0x7fffffffffffffffll, ky0 = kx0, kx1 = -kx0 - 1, ky1 = kx1;
  bool same = true;
  if (r < M) {
    const double *ry = rays + 6 * r;
    same = __double_as_longlong(ry[3]) == __double_as_longlong(d0[0]) &&
           __double_as_longlong(ry[4]) == __double_as_longlong(d0[1]) &&
           __double_as_longlong(ry[5]) == __double_as_longlong(d0[2]);
    const double x = dot3(ry, u), y = dot3(ry, v);
    ray2d[2 * r] = x;
    ray2d[2 * r + 1] = y;
    kx0 = kx1 = dkey(x);
    ky0 = ky1 = dkey(y);
  }
  for (int o = 16; o > 0; o >>= 1) {
    kx0 = min(kx0, __shfl_xor_sync(0xffffffffu, kx0, o));
    kx1 = max(kx1, __shfl_xor_sync(0xffffffffu, kx1, o));
    ky0 = min(ky0, __shfl_xor_sync(0xffffffffu, ky0, o));
    ky1 = max(ky1, __shfl_xor_sync(0xffffffffu, ky1, o));
  }
  const bool all_same = __syncthreads_and(same);
  __shared__ long long part[4][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) part[0][warp] = kx0, part[1][warp] = kx1, part[2][warp] = ky0, part[3][warp] = ky1;
  __syncthreads();
  if (threadIdx.x < 4) {
    const long long *w = part[threadIdx.x];
    long long k = w[0];
    if (threadIdx.x & 1) {
      for (int i = 1; i < 8; i++) k = max(k, w[i]);
      atomicMax(&ctrl[2 + threadIdx.x], k);
    } else {
      for (int i = 1; i < 8; i++) k = min(k, w[i]);
      atomicMin(&ctrl[2 + threadIdx.x], k);
    }
  }
  if (threadIdx.x == 0 && !all_same) atomicExch((unsigned long long *)&ctrl[0], 0ull);
}

// classification of triangle t for direction d0: -1 skip, 0 every-ray list, 1 binned (range out)
__device__ int classify(const double *T, const double *d0, const double *u, const double *v, const Box &b,
                        int max_bins, double *h, double *det_out, int *bx0, int *bx1, int *by0, int *by1) {
  const double *e1 = T + 3, *e2 = T + 6;
  cross3(d0, e2, h);
  const double det = *det_out = dot3(e1, h);
  if (det > -kEps && det < kEps) return -1;  // rejected as parallel by the reference, whatever the ray
  double n[3];
  cross3(e1, e2, n);
  const double nn = dot3(n, n), l1 = dot3(e1, e1), l2 = dot3(e2, e2), dd = dot3(d0, d0);
  const double nd = dot3(n, d0);
  if (!(nn >= 1e-6 * l1 * l2) || !(nd * nd >= 1e-6 * nn * dd)) return 0;
  double xs[3], ys[3];
  for (int k = 0; k < 3; k++) {
    const double p[3] = {T[0] + (k == 1 ? e1[0] : k == 2 ? e2[0] : 0.0), T[1] + (k == 1 ? e1[1] : k == 2 ? e2[1] : 0.0),
                         T[2] + (k == 1 ? e1[2] : k == 2 ? e2[2] : 0.0)};
    xs[k] = dot3(p, u);
    ys[k] = dot3(p, v);
  }
  const double m = b.margin + kMargin * fmax(fmax(fabs(xs[0]), fabs(ys[0])), fmax(fabs(T[0]), fabs(T[1])));
  const double xmin = fmin(fmin(xs[0], xs[1]), xs[2]) - m, xmax = fmax(fmax(xs[0], xs[1]), xs[2]) + m;
  const double ymin = fmin(fmin(ys[0], ys[1]), ys[2]) - m, ymax = fmax(fmax(ys[0], ys[1]), ys[2]) + m;
  if (xmax < b.x0 || xmin > b.x1 || ymax < b.y0 || ymin > b.y1) return -1;  // no ray projects there
  *bx0 = bin_x(b, xmin), *bx1 = bin_x(b, xmax), *by0 = bin_y(b, ymin), *by1 = bin_y(b, ymax);
  return (*bx1 - *bx0 + 1) * (*by1 - *by0 + 1) > max_bins ? 0 : 1;
}

// Calls f(triangle, bin) for every bin of the warp's triangles, kFill at a time a lane (f gets
// the batch): lane l holds triangle t0 + l's bins as first and last column and row, 8 bits each.
// The bins of all of them form one row, dealt out evenly: surfaces have triangles of one bin and
// of hundreds.
constexpr int kFill = 8;
constexpr uint32_t kNoBins = 1;  // first column after the last
template <class F>
__device__ __forceinline__ void for_bins(uint32_t range, int64_t t0, const F &f) {
  static_assert(kGX <= 256 && kGY <= 256, "a bin's column and row fit 8 bits");
  const int lane = threadIdx.x & 31;
  const auto width = [](uint32_t q) { return (int)(q >> 8 & 255) - (int)(q & 255) + 1; };
  int incl = width(range) * ((int)(range >> 24) - (int)(range >> 16 & 255) + 1);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int all = __shfl_sync(0xffffffffu, incl, 31);
  for (int i0 = 0; i0 < all; i0 += 32 * kFill) {
    int64_t t[kFill];
    int bin[kFill];
#pragma unroll
    for (int j = 0; j < kFill; j++) {
      const int i = i0 + 32 * j + lane;
      int src = 0;  // triangles whose bins end at or before i
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, incl, src + o - 1) <= i) src += o;
      const int before = __shfl_sync(0xffffffffu, incl, max(src - 1, 0));
      const uint32_t q = __shfl_sync(0xffffffffu, range, src);
      const int at = i - (src > 0 ? before : 0), w = width(q);
      t[j] = t0 + src;
      bin[j] = i < all ? ((int)(q >> 16 & 255) + at / w) * kGX + (int)(q & 255) + at % w : -1;
    }
    f(t, bin);
  }
}

// Counts the triangles of each bin, lists those every ray tests and packs all that a ray may
// test; a triangle's bins stay in its record.  A warp takes per_warp triangles: 32 of a large
// surface, fewer of a small one, whose triangles are few and cover many bins.
__global__ void __launch_bounds__(256) k_tri_count(const double *__restrict__ rays, const double *__restrict__ tri,
                                                   int64_t n, int per_warp, int max_bins, int32_t *bins, double *pack,
                                                   int32_t *glist, long long *ctrl) {
  const int lane = threadIdx.x & 31;
  const int64_t t0 = (blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32) * per_warp;
  if (t0 >= n || ctrl[0] == 0) return;  // whole warps
  uint32_t range = kNoBins;
  if (lane < per_warp && t0 + lane < n) {
    const int64_t t = t0 + lane;
    const double d0[3] = {rays[3], rays[4], rays[5]};
    double u[3], v[3];
    plane_basis(d0, u, v);
    const Box b = ray_box(ctrl);
    int bx0, bx1, by0, by1;
    double T[9], h[3], det;
    for (int k = 0; k < 9; k++) T[k] = tri[9 * t + k];
    const int c = classify(T, d0, u, v, b, max_bins, h, &det, &bx0, &bx1, &by0, &by1);
    if (c == 1) range = (uint32_t)bx0 | (uint32_t)bx1 << 8 | (uint32_t)by0 << 16 | (uint32_t)by1 << 24;
    if (c == 0) glist[atomicAdd((unsigned long long *)&ctrl[1], 1ull)] = (int32_t)t;
    double *P = pack + kPack * t;
    if (c >= 0) {
      store4(P, T[0], T[1], T[2], det);
      store4(P + 4, h[0], h[1], h[2], T[6]);
      store4(P + 8, T[3], T[4], T[5], T[7]);
    }
    store4(P + 12, T[8], __longlong_as_double(range), 0.0, 0.0);
  }
  __syncwarp();
  for_bins(range, t0, [&](const int64_t *, const int *bin) {
#pragma unroll
    for (int j = 0; j < kFill; j++)
      if (bin[j] >= 0) atomicAdd(&bins[bin[j]], 1);
  });
}

// Each triangle into its bins.  Bound by the latency of the atomics: a lane asks for kFill
// places at once, so a store waits for its own atomic only, not for the ones before it (44,032
// triangles in 239,000 bins: 7.9 us, 15.5 a triangle a thread, its bins found again).
__global__ void __launch_bounds__(256) k_tri_fill(int64_t n, int per_warp, const double *pack, int32_t *cursor,
                                                  int32_t *entries, const long long *ctrl) {
  const int lane = threadIdx.x & 31;
  const int64_t t0 = (blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32) * per_warp;
  if (t0 >= n || ctrl[0] == 0) return;  // whole warps
  const uint32_t range = lane < per_warp && t0 + lane < n
                             ? (uint32_t)__double_as_longlong(pack[kPack * (t0 + lane) + 13])
                             : kNoBins;
  for_bins(range, t0, [&](const int64_t *t, const int *bin) {
    int at[kFill];
#pragma unroll
    for (int j = 0; j < kFill; j++) at[j] = bin[j] >= 0 ? atomicAdd(&cursor[bin[j]], 1) : 0;
#pragma unroll
    for (int j = 0; j < kFill; j++)
      if (bin[j] >= 0) entries[at[j]] = (int32_t)t[j];
  });
}

// Exclusive scan of the kNB counts into offsets (bins[kNB] = total), cursor = offsets.  One
// cluster: a thread owns four consecutive bins (one vector load, whole lines a warp), shuffles
// scan the block, the blocks' sums are read over distributed shared memory.  Bound by the
// latency of that chain: 5.4 us, 15.5 by one block with 32 bins a thread.
constexpr int kCluster = 8;
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(1024) k_bins_scan(int32_t *bins, int32_t *cursor) {
  static_assert(kNB == kCluster * 1024 * 4, "four bins a thread");
  __shared__ int32_t wsum[32];
  __shared__ int32_t block_sum;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = (int)cl.block_rank(), at = rank * 1024 + (int)threadIdx.x;
  const int4 v = reinterpret_cast<const int4 *>(bins)[at];
  const int32_t sum = v.x + v.y + v.z + v.w;
  int32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int32_t w = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    wsum[lane] = w;
    if (lane == 31) block_sum = w;
  }
  cl.sync();  // the block's own sums, and every block's total
  int32_t run = incl - sum + (warp > 0 ? wsum[warp - 1] : 0);
  for (int b = 0; b < rank; b++) run += *cl.map_shared_rank(&block_sum, b);
  int4 x;
  x.x = run, run += v.x;
  x.y = run, run += v.y;
  x.z = run, run += v.z;
  x.w = run, run += v.w;
  reinterpret_cast<int4 *>(bins)[at] = x;
  reinterpret_cast<int4 *>(cursor)[at] = x;
  if (at == kCluster * 1024 - 1) bins[kNB] = run;
  cl.sync();  // no block leaves while another reads its total
}

// One thread per ray: its bin's triangles and the every-ray list, smallest (distance, index).
// What bounds it is the longest chain of tests, not their number: a surface seen along a pole
// of its triangulation puts hundreds of triangles in a few bins (44,032 triangles, 600 x 300
// rays: 7 a ray, 301 at most), and one thread's tests follow one another at a memory latency
// each.  So a ray whose bin holds more than kHeavy is put on a list with what it has so far,
// and a warp takes it up with a lane per triangle (trace_listed): 32 us here and
// 16 there, 218 with a thread for every ray.
constexpr int kTraceThreads = 128;
constexpr int kStage = 64;  // triangles of the every-ray list in shared memory at a time
template <bool kBodies>  // the Roche lobe (mode 1) or the accretor (mode 2) stand before the surface
__global__ void __launch_bounds__(kTraceThreads)
    k_ray_trace_binned(const double *__restrict__ rays, int64_t M, double *__restrict__ ray2d,
                       const double *__restrict__ pack, const int32_t *__restrict__ ids,
                       const int32_t *__restrict__ bins, const int32_t *__restrict__ entries,
                       const int32_t *__restrict__ glist, long long *ctrl, int64_t *__restrict__ listed, int mode,
                       int32_t *__restrict__ out) {
  __shared__ __align__(16) double staged[kStage][8];
  __shared__ int32_t sid[kStage];
  if (ctrl[0] == 0) return;  // the same for every thread
  const int64_t r = blockIdx.x * (int64_t)kTraceThreads + threadIdx.x;
  const bool live = r < M;
  double o[3] = {}, dir[3] = {};
  int32_t code = kNone;
  double best = 1e10;
  int64_t best_t = -1;
  bool search = live, heavy = false;
  if (live) {
    for (int k = 0; k < 3; k++) o[k] = rays[6 * r + k], dir[k] = rays[6 * r + 3 + k];
    if (kBodies && mode == 1) {
      double rd;
      if (roche(o, dir, &rd) != kNone) {
        best = rd;
        code = kRoche;
      }
    } else if (kBodies && mode == 2) {
      code = sphere_disk(o, dir);
      search = code == kNone;
    }
  }
  int k = 0;
  if (search) {
    const Box b = ray_box(ctrl);
    k = bin_y(b, ray2d[2 * r + 1]) * kGX + bin_x(b, ray2d[2 * r]);
    const int e0 = bins[k], e1 = bins[k + 1];
    heavy = e1 - e0 > kHeavy;
    if (!heavy) nearest_of(pack, entries, e0, e1, 1, o, dir, best, best_t);
  }
  const int ng = (int)ctrl[1];
  for (int g0 = 0; g0 < ng; g0 += kStage) {
    const int m = min(kStage, ng - g0);
    __syncthreads();
    for (int i = threadIdx.x; i < m * 8; i += kTraceThreads) {
      const int32_t t = glist[g0 + i / 8];
      staged[i / 8][i % 8] = pack[kPack * (int64_t)t + i % 8];
      if (i % 8 == 0) sid[i / 8] = t;
    }
    __syncthreads();
    if (search)
      for (int g = 0; g < m; g++) {
        Front f;
#pragma unroll
        for (int c = 0; c < 4; c++) f.A[c] = staged[g][c], f.h[c] = staged[g][4 + c];
        nearest(f, pack + kPack * (int64_t)sid[g], sid[g], o, dir, best, best_t);
      }
  }
  if (!live) return;
  out[r] = best_t >= 0 ? ids[best_t] : code;
  if (heavy) {
    ray2d[2 * r] = best;
    ray2d[2 * r + 1] = __longlong_as_double((long long)k << 32 | (uint32_t)(int32_t)best_t);
    listed[atomicAdd((unsigned long long *)&ctrl[6], 1ull)] = r;
  }
}

// MakeIllumAndCurve / MakeEnergyAndCurve (ray_tracing_calc_illum.cpp): pixel value by
// intersection code, curve = sum of value * pixel_factor.  One cluster: each thread sums a
// strided slice, a fixed-order tree sums the block, block 0 the blocks in their order over
// distributed shared memory, so the curve is deterministic and needs no workspace.  Bound by
// the latency of the two dependent loads a pixel, so eight pixels are in flight and eight SMs
// share them: 180,000 pixels 11.4 us, 105 by one block a pixel at a time.
constexpr int kImgThreads = 1024;
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kImgThreads)
    k_ray_image(const int32_t *__restrict__ codes, int64_t M, const double *__restrict__ value, int cell_size,
                double pixel_factor, double *__restrict__ image, double *__restrict__ curve, int *__restrict__ bad) {
  __shared__ double part[kImgThreads];
  cg::cluster_group cl = cg::this_cluster();
  constexpr int64_t kStride = (int64_t)kCluster * kImgThreads;
  constexpr int kBatch = 8;
  double acc = 0;
  for (int64_t i0 = (int64_t)cl.block_rank() * kImgThreads + threadIdx.x; i0 < M; i0 += kBatch * kStride) {
    int c[kBatch];
    double x[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; j++) c[j] = i0 + j * kStride < M ? codes[i0 + j * kStride] : kNone;
#pragma unroll
    for (int j = 0; j < kBatch; j++) {
      switch (c[j]) {
        case kNone: x[j] = 0; break;
        case kRoche: x[j] = 0.00001; break;  // k_rosh_energy
        case kDisk: x[j] = 5; break;         // k_disk_energy
        case kSphere: x[j] = 10; break;      // k_accretion_energy
        default:
          if (c[j] < 0) {
            atomicOr(bad, 1);
            x[j] = 0;
          } else {
            x[j] = value[c[j] / cell_size];
          }
      }
    }
#pragma unroll
    for (int j = 0; j < kBatch; j++)
      if (i0 + j * kStride < M) {
        image[i0 + j * kStride] = x[j];
        acc += x[j] * pixel_factor;
      }
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kImgThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
    __syncthreads();
  }
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x == 0) {
    double sum = 0;
    for (int b = 0; b < kCluster; b++) sum += *cl.map_shared_rank(&part[0], b);
    *curve = sum;
  }
  cl.sync();  // no block leaves while block 0 reads its sum
}

}  // namespace

extern "C" rrhd_status rrhd_ray_surface_create(const void *face_cells, int64_t n, int32_t device,
                                               rrhd_ray_surface **out) {
  RRHD_CHECK_ARG(out && n >= 0 && (face_cells || n == 0), "bad arguments");
  RRHD_CUDA(cudaSetDevice(device));
  auto *s = new rrhd_ray_surface;
  s->device = device;
  s->n = n;
  if (n > 0) {
    unsigned char *d_fc = nullptr;
    cudaError_t e = cudaMalloc(&d_fc, 80 * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&s->tri, 72 * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&s->ids, 4 * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(d_fc, face_cells, 80 * (size_t)n, cudaMemcpyDefault);
    if (e == cudaSuccess) {
      k_surface_prep<<<(unsigned)((n + 255) / 256), 256>>>(d_fc, n, s->tri, s->ids);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    cudaFree(d_fc);
    if (e != cudaSuccess) {
      cudaFree(s->tri);
      cudaFree(s->ids);
      delete s;
      return rrhd_fail(e == cudaErrorMemoryAllocation ? RRHD_ERR_OOM : RRHD_ERR_CUDA, "ray surface: %s",
                       cudaGetErrorString(e));
    }
  }
  *out = s;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_ray_surface_destroy(rrhd_ray_surface *s) {
  if (!s) return RRHD_OK;
  cudaSetDevice(s->device);
  cudaFree(s->tri);
  cudaFree(s->ids);
  cudaFree(s->bins);
  cudaFree(s->ray2d);
  delete s;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_ray_trace(const rrhd_ray_surface *s, const double *rays, int64_t M, int32_t mode,
                                      int32_t *codes, void *stream) {
  RRHD_CHECK_ARG(s && M >= 0, "bad arguments");
  RRHD_CHECK_ARG(mode >= 0 && mode <= 3, "mode must be 0 (surface), 1 (Roche lobe), 2 (inner) or 3 (grid)");
  if (M == 0) return RRHD_OK;
  RRHD_CHECK_ARG(rays && codes, "null rays or codes");
  RRHD_CUDA(cudaSetDevice(s->device));
  cudaStream_t st = (cudaStream_t)stream;
  if (s->n > kMaxBinnedTriangles) {
    // bin offsets are 32-bit: a surface this large takes the every-triangle kernel
    k_ray_trace<<<(unsigned)((M + kRayThreads - 1) / kRayThreads), kRayThreads, 0, st>>>(rays, M, s->tri, s->ids,
                                                                                          s->n, mode, codes, RayBins{});
    RRHD_CUDA(cudaGetLastError());
    return RRHD_OK;
  }
  rrhd_ray_surface *sm = const_cast<rrhd_ray_surface *>(s);
  if (!sm->bins) {  // one allocation: the first call of a surface pays for it
    size_t at = 0;
    const auto place = [&at](size_t bytes) {
      const size_t here = at;
      at += (bytes + 255) & ~(size_t)255;
      return here;
    };
    const size_t n = (size_t)s->n;
    const size_t bins = place(sizeof(int32_t) * (kNB + 1)), cursor = place(sizeof(int32_t) * kNB),
                 ctrl = place(sizeof(long long) * 8), entries = place(sizeof(int32_t) * max_bins(s->n) * n),
                 glist = place(sizeof(int32_t) * n), pack = place(sizeof(double) * kPack * n);
    char *base = nullptr;
    RRHD_CUDA(cudaMalloc(&base, at));
    sm->bins = reinterpret_cast<int32_t *>(base + bins);
    sm->cursor = reinterpret_cast<int32_t *>(base + cursor);
    sm->ctrl = reinterpret_cast<long long *>(base + ctrl);
    sm->entries = reinterpret_cast<int32_t *>(base + entries);
    sm->glist = reinterpret_cast<int32_t *>(base + glist);
    sm->pack = reinterpret_cast<double *>(base + pack);
  }
  if (sm->ray_cap < M) {
    RRHD_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    cudaFree(sm->ray2d);
    sm->ray2d = nullptr;
    sm->ray_cap = 0;
    RRHD_CUDA(cudaMalloc(&sm->ray2d, sizeof(double) * 3 * (size_t)M));
    sm->ray_cap = M;
  }
  const unsigned rb = (unsigned)((M + 255) / 256);
  const int per_warp = (int)std::min<int64_t>(32, std::max<int64_t>(1, s->n / kSpreadWarps));
  const unsigned tb = (unsigned)((s->n + 8 * per_warp - 1) / (8 * per_warp));
  k_bins_reset<<<(kNB + 1 + 255) / 256, 256, 0, st>>>(sm->bins, sm->ctrl);
  k_rays_project<<<rb, 256, 0, st>>>(rays, M, sm->ray2d, sm->ctrl);
  if (s->n > 0) {
    k_tri_count<<<tb, 256, 0, st>>>(rays, s->tri, s->n, per_warp, max_bins(s->n), sm->bins, sm->pack, sm->glist, sm->ctrl);
    k_bins_scan<<<kCluster, 1024, 0, st>>>(sm->bins, sm->cursor);
    k_tri_fill<<<tb, 256, 0, st>>>(s->n, per_warp, sm->pack, sm->cursor, sm->entries, sm->ctrl);
  }
  const unsigned nb = (unsigned)((M + kTraceThreads - 1) / kTraceThreads);
  const auto trace = mode == 1 || mode == 2 ? k_ray_trace_binned<true> : k_ray_trace_binned<false>;
  int64_t *listed = reinterpret_cast<int64_t *>(sm->ray2d + 2 * sm->ray_cap);
  trace<<<nb, kTraceThreads, 0, st>>>(rays, M, sm->ray2d, sm->pack, s->ids, sm->bins, sm->entries, sm->glist, sm->ctrl,
                                      listed, mode, codes);
  // the rays left to a warp each; or, rays of several directions, every ray against every triangle
  k_ray_trace<<<(unsigned)((M + kRayThreads - 1) / kRayThreads), kRayThreads, 0, st>>>(
      rays, M, s->tri, s->ids, s->n, mode, codes, RayBins{sm->ctrl, sm->ray2d, sm->pack, sm->bins, sm->entries, listed});
  RRHD_CUDA(cudaGetLastError());
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_ray_image(const int32_t *codes, int64_t M, const double *value, int32_t cell_size,
                                      double pixel_factor, double *image, double *curve, int32_t *bad,
                                      void *stream) {
  RRHD_CHECK_ARG(M >= 0 && cell_size > 0, "bad arguments");
  RRHD_CHECK_ARG(codes && image && curve && bad && (value || M == 0), "null argument");
  k_ray_image<<<kCluster, kImgThreads, 0, (cudaStream_t)stream>>>(codes, M, value, cell_size, pixel_factor, image, curve,
                                                          bad);
  RRHD_CUDA(cudaGetLastError());
  return RRHD_OK;
}

// MakeRays(num_frame) of ray_tracing_build_plane.cpp on the host (constants of
// ray_tracing_const.h, GRB_TASK plane): [600 * 300][6] rays, ray i * 300 + j for pixel (i, j).
namespace {
void host_cross(const double *a, const double *b, double *r) {
  r[0] = a[1] * b[2] - a[2] * b[1];
  r[1] = a[2] * b[0] - a[0] * b[2];
  r[2] = a[0] * b[1] - a[1] * b[0];
}
double host_dot(const double *a, const double *b) { return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2]; }
void host_normalize(double *v) {
  const double z = host_dot(v, v);
  if (z > 0) {
    const double s = std::sqrt(z);
    for (int k = 0; k < 3; k++) v[k] = v[k] / s;
  }
}
}  // namespace

extern "C" rrhd_status rrhd_ray_make_rays(int32_t frame, double *rays) {
  RRHD_CHECK_ARG(rays, "null rays");
  const double PIv = 3.1415926535897932384626433832795, com[3] = {0.879518, 0, 0};
  constexpr int nw = 600, nh = 300, nframes = 120;
  const double width = 1.2, height = 0.6, above = 0.1;
  const double start_angle = 2 * PIv / nframes * frame;
  const double start[3] = {std::cos(start_angle) + com[0], std::sin(start_angle) + com[1], above + com[2]};
  double dir[3] = {com[0] - start[0], com[1] - start[1], com[2] - start[2]};
  host_normalize(dir);
  // intersection::SetBasis (lib/geometry/src/intersections.cpp:3-40): rows v2, v1, normal
  double v1[3], v2[3];
  if (std::fabs(dir[1]) < 1e-20) {
    v1[0] = 0, v1[1] = 1, v1[2] = 0;
  } else {
    v1[0] = 1, v1[2] = 0;
    v1[1] = -(dir[0] * v1[0] + dir[2] * v1[2]) / dir[1];
  }
  if (dir[1] < 0)
    for (int k = 0; k < 3; k++) v1[k] = -v1[k];
  host_cross(dir, v1, v2);
  host_normalize(v1);
  host_normalize(v2);
  const double ap0 = -(width / 2), ap1 = -(height / 2);
  const double step_x = width / nw, step_y = height / nh;
  for (int i = 0; i < nw; ++i)
    for (int j = 0; j < nh; ++j) {
      const double x = ap0 + i * step_x, y = ap1 + j * step_y, z = 0;
      double *r = rays + 6 * ((int64_t)i * nh + j);
      // basis.transpose() * (x, y, z): row k = (v2[k] x + v1[k] y) + dir[k] z
      const double o3[3] = {(v2[0] * x + v1[0] * y) + dir[0] * z, (v2[1] * x + v1[1] * y) + dir[1] * z,
                            (v2[2] * x + v1[2] * y) + dir[2] * z};
      for (int k = 0; k < 3; k++) {
        r[k] = o3[k] + start[k];
        r[3 + k] = dir[k];
      }
    }
  return RRHD_OK;
}
