// FP64 radiation kernels: scattering integral, direction moments, 4-force.
//
// Compiled with --fmad=false: the "exact" kernels perform the reference's
// operations in the reference's order (one rounding each) and reproduce it bit
// for bit; the FMA variant of the scattering uses explicit fma() on a
// precomputed kernel matrix K[d][k] = Gamma(d,k) a_d / full_area.
//
// Scattering is a [rows x M] x [M x M] contraction with rows = cells x groups.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "rrhd_internal.h"

#include "dirs.h"
#include "coupled.h"
#include "rad_phys.cuh"

namespace {

constexpr int kMaxGroups = 64;  // groups of the cell-direction-group layout divide this

// (3 (1 + mu^2)) / 4 with mu = (x0 + x1) + x2: cuda_integrator.cu:10-13
__global__ void k_build_gamma(int M, const double *w, const double *a, double A, double *G,
                              double *K) {
  const int d = blockIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M) return;
  const double mu = (w[3 * d] * w[3 * k] + w[3 * d + 1] * w[3 * k + 1]) + w[3 * d + 2] * w[3 * k + 2];
  const double g = (3. * (1. + mu * mu)) / 4.;
  G[(size_t)d * M + k] = g;
  K[(size_t)d * M + k] = g * a[d] / A;
}

// Element (row r, direction d) of a [rows][M] array (lg < 0) or of a
// cell-direction-group array [rows >> lg][M][1 << lg] (row r = cell * 2^lg + group).
__device__ __forceinline__ int64_t elem(int64_t r, int d, int M, int lg) {
  return lg >= 0 ? (((r >> lg) * M + d) << lg) + (r & ((1 << lg) - 1)) : r * M + d;
}

// Tile element t of a (rows) x (nd directions) tile in memory order: row r, direction d.
__device__ __forceinline__ void tile_rd(int t, int nd, int lg, int &r, int &d) {
  if (lg >= 0) {
    const int g = t & ((1 << lg) - 1), q = t >> lg;
    d = q % nd;
    r = ((q / nd) << lg) + g;
  } else {
    r = t / nd;
    d = t % nd;
  }
}

__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Brings 16-direction stages of a row tile of I to shared memory (TRX rows, pitch PI), zero
// outside the array; NTH threads, consecutive ones on consecutive addresses.  A thread's
// elements of a stage are NTH / 16 rows apart (as many times M values in either layout, while
// a cell's 16 x groups values are no more than NTH), so a stage costs it an addition and a
// comparison an element; more groups index every element.
template <int TRX, int PI, int NTH>
struct RowStager {
  static constexpr int TD = 16, RS = NTH / 16;
  const double *__restrict__ pI, *__restrict__ I;
  int64_t left;  // rows from this thread's first one on
  int64_t rows, r0;
  int M, lg, dI, oI;
  __device__ __forceinline__ RowStager(const double *I_, int64_t rows_, int M_, int lg_, int64_t r0_)
      : I(I_), rows(rows_), r0(r0_), M(M_), lg(lg_) {
    int r;
    tile_rd(threadIdx.x, TD, lg, r, dI);
    left = rows - (r0 + r);
    pI = I + elem(r0 + r, dI, M, lg);
    oI = r * PI + dI;
  }
  __device__ __forceinline__ void operator()(double *sI, int d0) const {
    if (lg < 0 || (TD << lg) <= NTH) {
      const double *p = pI + (lg >= 0 ? (int64_t)d0 << lg : d0);
      const bool ok = d0 + dI < M;
#pragma unroll
      for (int q = 0; q < TRX / RS; q++) {
        const bool in = ok && RS * q < left;
        cp_async8(sI + oI + RS * q * PI, in ? p + (int64_t)(RS * q) * M : I, in);
      }
    } else {
      for (int t = threadIdx.x; t < TRX * TD; t += NTH) {
        int r, d;
        tile_rd(t, TD, lg, r, d);
        const bool in = r0 + r < rows && d0 + d < M;
        cp_async8(sI + r * PI + d, in ? I + elem(r0 + r, d0 + d, M, lg) : I, in);
      }
    }
  }
};

// ... and the 16 x TC stages of the matrix B [M][M] beside it (pitch PB), 256 threads.
template <int TRX, int TC, int PI, int PB>
struct Stager {
  static constexpr int TD = 16;
  RowStager<TRX, PI, 256> rows_of;
  const double *__restrict__ pB;
  int dB, oB, cols;
  __device__ __forceinline__ Stager(const double *I, const double *B, int64_t rows, int M, int lg, int64_t r0, int c0)
      : rows_of(I, rows, M, lg, r0) {
    dB = threadIdx.x / TC;
    const int c = threadIdx.x % TC;
    cols = M - (c0 + c);
    pB = B + (size_t)dB * M + c0 + c;
    oB = dB * PB + c;
  }
  __device__ __forceinline__ void operator()(double *sI, double *sB, int d0) const {
    rows_of(sI, d0);
    const int M = rows_of.M;
    const double *p = pB + (size_t)d0 * M;
#pragma unroll
    for (int q = 0; q < TD * TC / 256; q++) {
      constexpr int step = 256 / TC;
      const bool in = cols > 0 && d0 + dB + step * q < M;
      cp_async8(sB + oB + step * q * PB, in ? p + (size_t)(step * q) * M : rows_of.I, in);
    }
    cp_async_commit();
  }
};

// The reference's rounding sequence (GetS_MPI_multi_device): per term Gamma I, times a_d, added
// in direction order; the sum over full_area.  A CTA of 256 threads takes 16 R rows x 16 C
// output directions, a thread R rows x C columns (16 apart); tiles of 16 directions are staged
// two deep with cp.async.  Bound: the FP64 pipe, three instructions a term.  With R = 8, C = 4
// a direction costs a thread 13 shared loads for 96 FP64 instructions (4 x 4: 9 for 48,
// and twice the staging an element).  663,552 rows x 256 directions 8.9 -> 8.1 ms (86 % of the
// pipe), 500 rows x 256 56 -> 23 us.
template <int R, int C>
__global__ void __launch_bounds__(256, R * C >= 32 ? 2 : 3)
    k_scatter_exact(int64_t rows, int M, int lg, const double *__restrict__ I, const double *__restrict__ G,
                    const double *__restrict__ a, double A, double *__restrict__ S) {
  constexpr int TRX = 16 * R, TC = 16 * C, TD = 16, PI = TD + 1, PB = TC;
  extern __shared__ __align__(16) double sm[];
  double *sI = sm, *sB = sm + 2 * TRX * PI, *sa = sB + 2 * TD * PB;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int c0 = blockIdx.x * TC;
  const int64_t r0 = (int64_t)blockIdx.y * TRX + (int64_t)blockIdx.z * 65535 * TRX;
  if (r0 >= rows) return;
  double acc[R][C];
#pragma unroll
  for (int i = 0; i < R; i++)
#pragma unroll
    for (int j = 0; j < C; j++) acc[i][j] = 0.0;
  for (int d = threadIdx.x; d < M; d += 256) sa[d] = a[d];
  const Stager<TRX, TC, PI, PB> stage(I, G, rows, M, lg, r0, c0);
  stage(sI, sB, 0);
  int buf = 0;
  for (int d0 = 0; d0 < M; d0 += TD, buf ^= 1) {
    if (d0 + TD < M) {
      stage(sI + (buf ^ 1) * TRX * PI, sB + (buf ^ 1) * TD * PB, d0 + TD);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double *xI = sI + buf * TRX * PI + ty * PI, *xB = sB + buf * TD * PB + tx;
    auto term = [&](int d) {
      double iv[R], gv[C];
#pragma unroll
      for (int i = 0; i < R; i++) iv[i] = xI[16 * i * PI + d];
#pragma unroll
      for (int j = 0; j < C; j++) gv[j] = xB[d * PB + 16 * j];
      const double ad = sa[d0 + d];
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < C; j++) {
          double t = gv[j] * iv[i];
          t = t * ad;
          acc[i][j] = acc[i][j] + t;
        }
    };
    if (d0 + TD <= M) {
#pragma unroll 4
      for (int d = 0; d < TD; d++) term(d);
    } else {
      for (int d = 0; d < M - d0; d++) term(d);
    }
    __syncthreads();
  }
  // the tile through shared memory, stored in memory order of the layout
  constexpr int PO = TC + 1;
  double *sO = sm;
#pragma unroll
  for (int i = 0; i < R; i++)
#pragma unroll
    for (int j = 0; j < C; j++) sO[(ty + 16 * i) * PO + tx + 16 * j] = acc[i][j] / A;
  __syncthreads();
#pragma unroll 4
  for (int t = threadIdx.x; t < TRX * TC; t += 256) {
    int r, k;
    tile_rd(t, TC, lg, r, k);
    if (r0 + r < rows && c0 + k < M) S[elem(r0 + r, c0 + k, M, lg)] = sO[r * PO + k];
  }
}
template <int R, int C>
constexpr size_t exact_smem(int M) {
  const size_t in = 2 * (16 * R * 17 + 16 * 16 * C) + (size_t)M, out = (size_t)16 * R * (16 * C + 1);
  return sizeof(double) * (in > out ? in : out);
}

// One FMA per term on K[d][k] = Gamma(d,k) a_d / full_area, on the FP64 matrix instruction
// (mma.sync m8n8k4: the fifth-generation tensor cores take no FP64).  A CTA of eight warps
// takes 32 WR rows x 64 output directions, a warp 8 WR x 32 (WR x 4 accumulator tiles); tiles
// of 16 directions staged two deep with cp.async, pitches of 4 modulo 16 doubles so that the
// fragment loads are free of bank conflicts.  Per k step a warp loads WR + 4 doubles a lane for
// 4 WR instructions of 256 multiply-adds; one thread per 4 x 4 block with plain FMAs needed 8
// loads for 16 x 32 and was bound by them: 663,552 rows x 256 directions 5.4 -> 2.8 ms (83 % of
// the pipe).
__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}
template <int WR>
__global__ void __launch_bounds__(256, 2)
    k_scatter_mma(int64_t rows, int M, int lg, const double *__restrict__ I, const double *__restrict__ K,
                  double *__restrict__ S) {
  constexpr int TRX = 32 * WR, TC = 64, TD = 16, PI = TD + 4, PB = TC + 4;
  extern __shared__ __align__(16) double sm[];
  double *sI = sm, *sB = sm + 2 * TRX * PI;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 1) * 8 * WR, wc = (warp & 1) * 32;
  const int c0 = blockIdx.x * TC;
  const int64_t r0 = (int64_t)blockIdx.y * TRX + (int64_t)blockIdx.z * 65535 * TRX;
  if (r0 >= rows) return;
  double acc[WR][4][2];
#pragma unroll
  for (int i = 0; i < WR; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
  const Stager<TRX, TC, PI, PB> stage(I, K, rows, M, lg, r0, c0);
  stage(sI, sB, 0);
  int buf = 0;
  for (int d0 = 0; d0 < M; d0 += TD, buf ^= 1) {
    if (d0 + TD < M) {
      stage(sI + (buf ^ 1) * TRX * PI, sB + (buf ^ 1) * TD * PB, d0 + TD);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double *xI = sI + buf * TRX * PI + (wr + g) * PI + t, *xB = sB + buf * TD * PB + t * PB + wc + g;
#pragma unroll
    for (int k = 0; k < TD; k += 4) {
      double av[WR], bv[4];
#pragma unroll
      for (int i = 0; i < WR; i++) av[i] = xI[8 * i * PI + k];
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = xB[k * PB + 8 * j];
#pragma unroll
      for (int i = 0; i < WR; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
    __syncthreads();
  }
  // lane (g, t) holds row g, columns 2t and 2t + 1 of each tile: whole sectors in either layout
  const bool pairs = lg < 0 && M % 2 == 0 && (reinterpret_cast<uintptr_t>(S) & 15) == 0;
#pragma unroll
  for (int i = 0; i < WR; i++) {
    const int64_t r = r0 + wr + 8 * i + g;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c = c0 + wc + 8 * j + 2 * t;
      if (pairs) {
        if (c < M) *reinterpret_cast<double2 *>(S + r * M + c) = make_double2(acc[i][j][0], acc[i][j][1]);
      } else {
        if (c < M) S[elem(r, c, M, lg)] = acc[i][j][0];
        if (c + 1 < M) S[elem(r, c + 1, M, lg)] = acc[i][j][1];
      }
    }
  }
}
template <int WR>
constexpr size_t mma_smem() {
  return sizeof(double) * 2 * (32 * WR * 20 + 16 * 68);
}

// Column tiles of a row tile are neighbours in the grid, so that the row tile is read from
// HBM once; rows beyond 65,535 tiles go to the grid's third dimension.
dim3 scatter_grid(int64_t rows, int M, int tr, int tc) {
  const int64_t nr = (rows + tr - 1) / tr;
  return dim3((unsigned)((M + tc - 1) / tc), (unsigned)(nr < 65535 ? nr : 65535), (unsigned)((nr + 65534) / 65535));
}

template <int R, int C>
cudaError_t run_exact(const rrhd_dirs *d, const double *I, double *S, int64_t rows, int lg, cudaStream_t st) {
  const size_t smem = exact_smem<R, C>(d->M);
  const cudaError_t e =
      cudaFuncSetAttribute(k_scatter_exact<R, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_scatter_exact<R, C><<<scatter_grid(rows, d->M, 16 * R, 16 * C), 256, smem, st>>>(rows, d->M, lg, I, d->d_G, d->d_a,
                                                                                     d->full_area, S);
  return cudaGetLastError();
}
template <int C>
cudaError_t pick_exact(const rrhd_dirs *d, const double *I, double *S, int64_t rows, int lg, cudaStream_t st) {
  const int64_t cols = (d->M + 16 * C - 1) / (16 * C);
  // the largest tile that fills the SMs (two resident CTAs of 128 rows four times over, three
  // of 64 once, one of 32), so that small calls spread out and the last wave costs little; a
  // tile holds whole cells (up to 64 groups)
  const int64_t ctas = 148;
  if (cols * ((rows + 127) / 128) >= 8 * ctas) return run_exact<8, C>(d, I, S, rows, lg, st);
  if (lg > 5 || cols * ((rows + 63) / 64) >= 3 * ctas) return run_exact<4, C>(d, I, S, rows, lg, st);
  if (lg > 4 || cols * ((rows + 31) / 32) >= ctas) return run_exact<2, C>(d, I, S, rows, lg, st);
  return run_exact<1, C>(d, I, S, rows, lg, st);
}
cudaError_t launch_exact(const rrhd_dirs *d, const double *I, double *S, int64_t rows, int lg, cudaStream_t st) {
  // 32 output directions a tile where that leaves fewer columns of padding than 64
  return (d->M + 31) / 32 * 32 < (d->M + 63) / 64 * 64 ? pick_exact<2>(d, I, S, rows, lg, st)
                                                       : pick_exact<4>(d, I, S, rows, lg, st);
}

template <int WR>
cudaError_t run_mma(const rrhd_dirs *d, const double *I, double *S, int64_t rows, int lg, cudaStream_t st) {
  const cudaError_t e =
      cudaFuncSetAttribute(k_scatter_mma<WR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mma_smem<WR>());
  if (e != cudaSuccess) return e;
  k_scatter_mma<WR><<<scatter_grid(rows, d->M, 32 * WR, 64), 256, mma_smem<WR>(), st>>>(rows, d->M, lg, I, d->d_K, S);
  return cudaGetLastError();
}
cudaError_t launch_mma(const rrhd_dirs *d, const double *I, double *S, int64_t rows, int lg, cudaStream_t st) {
  const int64_t cols = (d->M + 63) / 64, ctas = 148;
  if (cols * ((rows + 127) / 128) >= ctas) return run_mma<4>(d, I, S, rows, lg, st);
  if (lg > 5 || cols * ((rows + 63) / 64) >= ctas) return run_mma<2>(d, I, S, rows, lg, st);
  return run_mma<1>(d, I, S, rows, lg, st);
}

// cuda_sep::device::MakeEnergy / MakeStream / MakeImpuls (cuda_illum_sep_param.cu:9-69), RPT
// rows a thread, the reference's operations in its order.  Its products w_i w_j do not depend
// on the row (and T is symmetric to the bit), so they are formed once per stage of 16
// directions: 20 FP64 instructions a term instead of 41.  Bound: reading I (663,552 rows x 256
// directions 0.54 -> 0.43 ms; 500 rows x 256 43 -> 26 us, the stages' loads in flight while
// the one before is summed).
constexpr int MT = 128, MD = 16;
template <int RPT>
__global__ void __launch_bounds__(MT) k_moments(int64_t rows, int M, int lg, const double *__restrict__ I,
                                                const double *__restrict__ w, const double *__restrict__ a, double A,
                                                double *__restrict__ E, double *__restrict__ Fo,
                                                double *__restrict__ To) {
  constexpr int TRX = MT * RPT, PI = MD + 1;
  extern __shared__ __align__(16) double sm[];
  double *sI = sm;                                              // [2][TRX][PI]
  __shared__ __align__(16) double sw[2][MD][10];  // {a, w0, w1, w2, w0w0, w0w1, w0w2, w1w1, w1w2, w2w2}
  const int64_t r0 = (int64_t)blockIdx.x * TRX;
  const RowStager<TRX, PI, MT> stage(I, rows, M, lg, r0);
  auto weights = [&](int buf, int d0) {
    if (threadIdx.x < MD) {
      const int d = d0 + threadIdx.x;
      double *o = sw[buf][threadIdx.x];
      const double w0 = d < M ? w[3 * d] : 0.0, w1 = d < M ? w[3 * d + 1] : 0.0, w2 = d < M ? w[3 * d + 2] : 0.0;
      o[0] = d < M ? a[d] : 0.0;
      o[1] = w0, o[2] = w1, o[3] = w2;
      o[4] = w0 * w0, o[5] = w0 * w1, o[6] = w0 * w2, o[7] = w1 * w1, o[8] = w1 * w2, o[9] = w2 * w2;
    }
  };
  double acc[RPT][10];
#pragma unroll
  for (int i = 0; i < RPT; i++)
#pragma unroll
    for (int q = 0; q < 10; q++) acc[i][q] = 0.0;
  stage(sI, 0);
  cp_async_commit();
  weights(0, 0);
  int buf = 0;
  for (int d0 = 0; d0 < M; d0 += MD, buf ^= 1) {
    if (d0 + MD < M) {
      stage(sI + (buf ^ 1) * TRX * PI, d0 + MD);
      cp_async_commit();
      weights(buf ^ 1, d0 + MD);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const double *x = sI + buf * TRX * PI + threadIdx.x * PI;
    auto term = [&](int d) {
      double v[10];
#pragma unroll
      for (int q = 0; q < 10; q += 2) {
        const double2 t = *reinterpret_cast<const double2 *>(&sw[buf][d][q]);
        v[q] = t.x;
        v[q + 1] = t.y;
      }
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const double Ia = x[i * MT * PI + d] * v[0];
        acc[i][0] = acc[i][0] + Ia;
#pragma unroll
        for (int q = 1; q < 10; q++) acc[i][q] = acc[i][q] + v[q] * Ia;
      }
    };
    if (d0 + MD <= M) {
#pragma unroll 4
      for (int d = 0; d < MD; d++) term(d);
    } else {
      for (int d = 0; d < M - d0; d++) term(d);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RPT; i++) {
    const int64_t r = r0 + i * MT + threadIdx.x;
    if (r >= rows) continue;
    E[r] = acc[i][0] / A;
#pragma unroll
    for (int q = 0; q < 3; q++) Fo[3 * r + q] = acc[i][1 + q] / A;
    const double t00 = acc[i][4] / A, t01 = acc[i][5] / A, t02 = acc[i][6] / A;
    const double t11 = acc[i][7] / A, t12 = acc[i][8] / A, t22 = acc[i][9] / A;
    const double t[9] = {t00, t01, t02, t01, t11, t12, t02, t12, t22};
#pragma unroll
    for (int q = 0; q < 9; q++) To[9 * r + q] = t[q];
  }
}

cudaError_t launch_moments(const rrhd_dirs *d, const double *I, double *E, double *F, double *T, int64_t rows, int lg,
                           cudaStream_t st) {
  // two rows a thread share the weights' shared loads; one where that leaves SMs idle
  const bool two = rows >= 2 * MT * 4 * 148;
  const int tr = two ? 2 * MT : MT;
  const size_t smem = sizeof(double) * 2 * tr * (MD + 1);
  const unsigned nb = (unsigned)((rows + tr - 1) / tr);
  auto *k = two ? k_moments<2> : k_moments<1>;
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k<<<nb, MT, smem, st>>>(rows, d->M, lg, I, d->d_w, d->d_a, d->full_area, E, F, T);
  return cudaGetLastError();
}

// rad_rhd::GetRadSource, solvers/RadRHD/src/radRHD_utils.cpp:44-101
__global__ void k_rad_source(int64_t n, rrhd::Emission em, const double *__restrict__ W,
                             const double *__restrict__ alpha, const double *__restrict__ sigma,
                             const double *__restrict__ E, const double *__restrict__ F,
                             const double *__restrict__ T, double *__restrict__ G) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c >= n) return;
  double w[5], Fr[3], Tr[9], g[4];
#pragma unroll
  for (int i = 0; i < 5; i++) w[i] = W[5 * c + i];
#pragma unroll
  for (int i = 0; i < 3; i++) Fr[i] = F[3 * c + i];
#pragma unroll
  for (int i = 0; i < 9; i++) Tr[i] = T[9 * c + i];
  rrhd::rad_source_cell(em, w, alpha[c], sigma[c], E[c], Fr, Tr, g);
#pragma unroll
  for (int i = 0; i < 4; i++) G[4 * c + i] = g[i];
}

}  // namespace

extern "C" rrhd_status rrhd_dirs_create(int32_t M, const double *dirs, const double *areas,
                                        double full_area, int32_t device, rrhd_dirs **out) {
  RRHD_CHECK_ARG(out && dirs && areas && M > 0 && M <= 4096 && full_area > 0, "bad direction set");
  *out = nullptr;
  RRHD_CUDA(cudaSetDevice(device));
  rrhd_dirs *d = new rrhd_dirs();
  d->device = device;
  d->M = M;
  d->full_area = full_area;
  d->h_w.assign(dirs, dirs + 3 * M);
  d->h_a.assign(areas, areas + M);
  const size_t mm = sizeof(double) * (size_t)M * M;
  if (cudaMalloc(&d->d_w, sizeof(double) * 3 * M) || cudaMalloc(&d->d_a, sizeof(double) * M) ||
      cudaMalloc(&d->d_G, mm) || cudaMalloc(&d->d_K, mm)) {
    rrhd_dirs_destroy(d);
    return rrhd_fail(RRHD_ERR_OOM, "direction set allocation failed");
  }
  cudaMemcpy(d->d_w, dirs, sizeof(double) * 3 * M, cudaMemcpyHostToDevice);
  cudaMemcpy(d->d_a, areas, sizeof(double) * M, cudaMemcpyHostToDevice);
  k_build_gamma<<<dim3((M + 127) / 128, M), 128>>>(M, d->d_w, d->d_a, full_area, d->d_G, d->d_K);
  if (cudaDeviceSynchronize() != cudaSuccess) {
    rrhd_dirs_destroy(d);
    return rrhd_fail(RRHD_ERR_CUDA, "building the phase matrix failed");
  }
  *out = d;
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_dirs_destroy(rrhd_dirs *d) {
  if (!d) return RRHD_OK;
  cudaSetDevice(d->device);
  cudaFree(d->d_w);
  cudaFree(d->d_a);
  cudaFree(d->d_G);
  cudaFree(d->d_K);
  delete d;
  return RRHD_OK;
}

extern "C" int32_t rrhd_dirs_count(const rrhd_dirs *d) { return d ? d->M : 0; }
extern "C" const double *rrhd_dirs_device_kernel(const rrhd_dirs *d) { return d ? d->d_K : nullptr; }

extern "C" rrhd_status rrhd_scatter_fp64(const rrhd_dirs *d, const double *I, double *S, int64_t rows,
                                         void *stream) {
  RRHD_CHECK_ARG(d && I && S && rows >= 0, "bad arguments");
  if (rows == 0) return RRHD_OK;
  RRHD_CUDA(launch_exact(d, I, S, rows, -1, (cudaStream_t)stream));
  return RRHD_OK;
}

// Same contraction with one FMA per term on K = Gamma a / full_area (rounding
// differs from the reference's three roundings by a few ulp per term).
extern "C" rrhd_status rrhd_scatter_fp64_fma(const rrhd_dirs *d, const double *I, double *S, int64_t rows,
                                             void *stream) {
  RRHD_CHECK_ARG(d && I && S && rows >= 0, "bad arguments");
  if (rows == 0) return RRHD_OK;
  RRHD_CUDA(launch_mma(d, I, S, rows, -1, (cudaStream_t)stream));
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_moments_fp64(const rrhd_dirs *d, const double *I, double *E, double *F,
                                         double *T, int64_t rows, void *stream) {
  RRHD_CHECK_ARG(d && I && E && F && T && rows >= 0, "bad arguments");
  if (rows == 0) return RRHD_OK;
  RRHD_CUDA(launch_moments(d, I, E, F, T, rows, -1, (cudaStream_t)stream));
  return RRHD_OK;
}

rrhd_status rrhd::scatter_fp64_cdg(const rrhd_dirs *d, const double *I, double *S, int64_t cells, int ng, bool exact,
                                   cudaStream_t st) {
  RRHD_CHECK_ARG(d && I && S && cells >= 0 && ng > 0 && kMaxGroups % ng == 0, "bad arguments");
  const int64_t rows = cells * ng;
  if (rows == 0) return RRHD_OK;
  int lg = 0;
  while ((1 << lg) < ng) lg++;
  RRHD_CUDA(exact ? launch_exact(d, I, S, rows, lg, st) : launch_mma(d, I, S, rows, lg, st));
  return RRHD_OK;
}

rrhd_status rrhd::moments_fp64_cdg(const rrhd_dirs *d, const double *I, double *E, double *F, double *T,
                                   int64_t cells, int ng, cudaStream_t st) {
  RRHD_CHECK_ARG(d && I && E && F && T && cells >= 0 && ng > 0 && MT % ng == 0, "bad arguments");
  const int64_t rows = cells * ng;
  if (rows == 0) return RRHD_OK;
  int lg = 0;
  while ((1 << lg) < ng) lg++;
  RRHD_CUDA(launch_moments(d, I, E, F, T, rows, lg, st));
  return RRHD_OK;
}

extern "C" rrhd_emission rrhd_emission_reference(void) {
  // CGS constants of lib/global_consts.h and the unit system it defines
  const double kC_Light = 3 * 1e10, k_boltzmann = 1.3807 * 1e-16, kM_hydrogen = 1.6735575 * 1e-24;
  const double kStefanBoltzmann = 5.670374419 * 1e-5, kGravity = 6.6726 * 1e-8;
  const double PI = 3.1415926535897932384626433832795;
  const double kDist = 1e13, kVelocity = kC_Light;
  const double kMass = (kVelocity * kVelocity * kDist) / kGravity;
  const double kTime = (kDist / kVelocity);
  const double kDensity = (kMass / (kDist * kDist * kDist));
  const double kPressure = kMass / (kDist * kTime * kTime);
  const double kRadiation = (kMass / (kTime * kTime * kTime));
  rrhd_emission e;
  e.temp_coef = (kM_hydrogen / k_boltzmann) * kPressure / kDensity;
  e.sigma_sb = kStefanBoltzmann;
  e.pi = PI;
  e.rad_unit = kRadiation;
  return e;
}

extern "C" rrhd_status rrhd_rad_source(const rrhd_emission *em, const double *W, const double *alpha,
                                       const double *sigma, const double *E, const double *F, const double *T,
                                       double *G, int64_t n, void *stream) {
  RRHD_CHECK_ARG(em && W && alpha && sigma && E && F && T && G && n >= 0, "bad arguments");
  if (n == 0) return RRHD_OK;
  rrhd::Emission e{em->temp_coef, em->sigma_sb, em->pi, em->rad_unit};
  k_rad_source<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)stream>>>(n, e, W, alpha, sigma, E, F, T, G);
  RRHD_CUDA(cudaGetLastError());
  return RRHD_OK;
}

extern "C" rrhd_status rrhd_scatter_fp64_cdg(const rrhd_dirs *d, const double *I, double *S, int64_t cells,
                                             int32_t groups, int32_t exact, void *stream) {
  return rrhd::scatter_fp64_cdg(d, I, S, cells, groups, exact != 0, (cudaStream_t)stream);
}

extern "C" rrhd_status rrhd_moments_fp64_cdg(const rrhd_dirs *d, const double *I, double *E, double *F, double *T,
                                             int64_t cells, int32_t groups, void *stream) {
  return rrhd::moments_fp64_cdg(d, I, E, F, T, cells, groups, (cudaStream_t)stream);
}
