// Jacobi-preconditioned CG of a small grid as ONE launch: a thread-block cluster
// holds the whole solve on chip.
//
// Each CTA owns a band of grid rows.  The direction p (with one halo row on each
// side) and the inverse diagonal sit in shared memory, x, r and q in registers, so
// a pass touches no global memory.  The recurrence is k_cg_pq / k_cg_xr's (SciPy's,
// pycfd/core/pressure.py:388-391) with two cluster barriers per pass: one behind the
// p.q partials, one behind the r.r and r.z partials.  Every CTA writes its partials
// into every other CTA's shared memory (distributed shared memory) before the barrier
// and adds all of them in CTA order behind it, so the scalars are formed redundantly,
// deterministically and without a second round trip.  The band's first and last rows
// of z travel with the second set: a CTA forms its halo rows of p itself.
//
// What bounds a pass is the latency of its two reductions and barriers, and from about
// 30,000 cells the shared-memory traffic of a band; one launch per phase cost two
// launches and a WHILE iteration, or a host read, instead.  Measured on B200, us per
// pass: 64x64 (recorded steps) 16 -> 2.4, 200x150 (host loop) 28 -> 3.5; 256x256 now
// 5.0, 512x256 9.2, and 520x300, the first that no cluster holds, 29 by the phases.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "poisson.cuh"

namespace pcfd {

constexpr int kClThreads = 512;
constexpr int kClMaxCtas = 16;       // the largest cluster (opt-in size)
constexpr int kClMaxCells = 16;      // cells per thread at most
constexpr int kClRegCells = 8;       // up to here x stays in registers, above in shared memory

struct ClSolve {
  const uint8_t* flags;
  Geo g;
  SolveCfg cfg;
  double* x;
  const double* r;    // initial residual (k_rhs_init)
  double* S;
  int* I;
  int rmax;           // rows of the largest band
};

// Dynamic shared memory of one CTA: p with its halo rows, the inverse diagonal, the
// neighbours' rows of z, x above kClRegCells, a flag byte per cell.
inline size_t cl_smem(int rmax, int ny, bool xs) {
  const size_t n = (size_t)rmax * ny;
  return (n + 2 * (size_t)ny + n + 2 * (size_t)ny + (xs ? n : 0)) * sizeof(double) + n;
}

// Sum of the cluster's partials part[0..15] (rows past the cluster size are zero), in
// every thread: lanes 0-15 take row 0, lanes 16-31 row 1.
__device__ __forceinline__ void cl_total2(const double (*part)[kClMaxCtas], double* a, double* b) {
  const int lane = threadIdx.x & 31;
  double v = part[lane >> 4][lane & 15];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  *a = __shfl_sync(0xffffffffu, v, 0);
  *b = __shfl_sync(0xffffffffu, v, 16);
}

template <int CPT>
__global__ void __launch_bounds__(kClThreads, 1) k_cg_cluster(ClSolve t) {
  pdl_begin();
  if (t.I[I_DONE]) return;   // the same word for every CTA
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr bool XS = CPT > kClRegCells;
  constexpr int kWarps = kClThreads / 32;
  extern __shared__ double cl_sm[];
  __shared__ double part1[2][kClMaxCtas];   // p.q (row 1 stays zero)
  __shared__ double part2[2][kClMaxCtas];   // r.r, r.z
  __shared__ double wsum[2][kWarps];
  const Geo& g = t.g;
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int nx = g.nx, ny = g.ny;
  const int r0 = (int)((long)rank * nx / C), r1 = (int)((long)(rank + 1) * nx / C);
  const int cells = (r1 - r0) * ny;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* p = cl_sm;                                   // halo row, band, halo row
  double* dinv = p + (size_t)(t.rmax + 2) * ny;
  double* zh = dinv + (size_t)t.rmax * ny;             // west neighbour's last row, east neighbour's first
  double* xs = zh + 2 * (size_t)ny;
  uint8_t* fl = (uint8_t*)(xs + (XS ? (size_t)t.rmax * ny : 0));
  const int west = rank > 0 ? rank - 1 : (g.periodic_x ? C - 1 : -1);
  const int east = rank < C - 1 ? rank + 1 : (g.periodic_x ? 0 : -1);
  // where this CTA's first and last rows of z go
  double* zw = west >= 0 ? cl.map_shared_rank(zh, west) + ny : nullptr;
  double* ze = east >= 0 ? cl.map_shared_rank(zh, east) : nullptr;
  const long base = (long)r0 * ny;

  if (tid < 2 * kClMaxCtas) {
    (&part1[0][0])[tid] = 0.0;
    (&part2[0][0])[tid] = 0.0;
  }
  double rv[CPT], qz[CPT], xv[XS ? 1 : CPT];
#pragma unroll
  for (int m = 0; m < CPT; ++m) {
    const int k = tid + m * kClThreads;
    rv[m] = qz[m] = 0.0;
    if (!XS) xv[m] = 0.0;
    if (k < cells) {
      const int il = k / ny, j = k - il * ny;
      const uint8_t f = t.flags[base + k];
      const double di = 1.0 / fine_diag(f, r0 + il, j, g);
      dinv[k] = di;
      // bits 5, 6: the first and last column of a row (the wrap of a periodic y axis)
      fl[k] = (uint8_t)((f & 31) | (j == 0 ? 32 : 0) | (j == ny - 1 ? 64 : 0));
      rv[m] = t.r[base + k];
      qz[m] = rv[m] * di;
      if (XS) xs[k] = t.x[base + k];
      else xv[m] = t.x[base + k];
    }
  }
  for (int k = tid; k < 2 * ny; k += kClThreads) {   // the neighbours' rows of z at the start
    const bool e = k >= ny;
    const int j = e ? k - ny : k;
    double z = 0.0;
    if (e ? east >= 0 : west >= 0) {
      const int i = e ? (r1 < nx ? r1 : 0) : (r0 > 0 ? r0 - 1 : nx - 1);
      const long c = (long)i * ny + j;
      z = t.r[c] * (1.0 / fine_diag(t.flags[c], i, j, g));
    }
    zh[k] = z;
    p[e ? (size_t)(r1 - r0 + 1) * ny + j : j] = 0.0;
  }
  double rho = t.S[S_RHO], rho_prev = 1.0, rr = t.S[S_RNORM2];
  const double atol = t.S[S_ATOL];
  int it = 0;
  bool conv = false;
  cl.sync();   // every CTA runs and has set its words before any remote write

  for (;;) {
    // ---- p = z + beta p on the band and its halo rows
    const double beta = it ? rho / rho_prev : 0.0;
#pragma unroll
    for (int m = 0; m < CPT; ++m) {
      const int k = tid + m * kClThreads;
      if (k < cells) p[ny + k] = it ? p[ny + k] * beta + qz[m] : qz[m];
    }
    for (int k = tid; k < 2 * ny; k += kClThreads) {
      double* h = p + (k < ny ? k : (size_t)(r1 - r0 + 1) * ny + (k - ny));
      *h = it ? *h * beta + zh[k] : zh[k];
    }
    __syncthreads();
    // ---- q = A p, p.q
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < CPT; ++m) {
      const int k = tid + m * kClThreads;
      if (k < cells) {
        const uint8_t f = fl[k];
        const double* pc = p + ny + k;
        const double c = pc[0];
        const double w = (f & F_W) ? pc[-ny] : 0.0, e = (f & F_E) ? pc[ny] : 0.0;
        const double s = (f & F_S) ? pc[(f & 32) ? ny - 1 : -1] : 0.0;
        const double n = (f & F_N) ? pc[(f & 64) ? 1 - ny : 1] : 0.0;
        int jj = 1, ii = 1;
        double d;
        if (g.dir_w | g.dir_e | g.dir_s | g.dir_n) {   // Dirichlet edges add to the diagonal
          const int il = k / ny;
          ii = r0 + il;
          jj = k - il * ny;
          d = fine_diag(f, ii, jj, g);
        } else {
          d = 0.0;
          if (f & F_W) d -= g.cx;
          if (f & F_E) d -= g.cx;
          if (f & F_S) d -= g.cy;
          if (f & F_N) d -= g.cy;
          if (!(f & F_SOLV)) d = 1.0;
        }
        double q = d * c;
        q += g.cx * w;
        q += g.cx * e;
        q += g.cy * s;
        q += g.cy * n;
        qz[m] = q;
        acc += c * q;
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) wsum[0][warp] = acc;
    __syncthreads();
    if (warp == 0) {
      double v = wsum[0][lane & (kWarps - 1)];
#pragma unroll
      for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < C) cl.map_shared_rank(&part1[0][0], lane)[rank] = v;
    }
    cl.sync();
    double pq, unused;
    cl_total2(part1, &pq, &unused);
    const double alpha = rho / pq;
    // ---- x += alpha p, r -= alpha q, z = r / d; r.r and r.z; the edge rows of z
    double a0 = 0.0, a1 = 0.0;
#pragma unroll
    for (int m = 0; m < CPT; ++m) {
      const int k = tid + m * kClThreads;
      if (k < cells) {
        const double pc = p[ny + k];
        if (XS) xs[k] += alpha * pc;
        else xv[m] += alpha * pc;
        const double r = rv[m] - alpha * qz[m];
        rv[m] = r;
        const double z = r * dinv[k];
        qz[m] = z;
        a0 += r * r;
        a1 += r * z;
        if (k < ny && zw) zw[k] = z;
        if (k >= cells - ny && ze) ze[k - (cells - ny)] = z;
      }
    }
    a0 = warp_sum(a0);
    a1 = warp_sum(a1);
    if (lane == 0) {
      wsum[0][warp] = a0;
      wsum[1][warp] = a1;
    }
    __syncthreads();
    if (warp < 2) {
      double v = wsum[warp][lane & (kWarps - 1)];
#pragma unroll
      for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < C) cl.map_shared_rank(&part2[warp][0], lane)[rank] = v;
    }
    cl.sync();
    rho_prev = rho;
    cl_total2(part2, &rr, &rho);
    ++it;
    conv = sqrt(rr) < atol;
    if (conv || it >= t.cfg.maxiter) break;
  }
#pragma unroll
  for (int m = 0; m < CPT; ++m) {
    const int k = tid + m * kClThreads;
    if (k < cells) t.x[base + k] = XS ? xs[k] : xv[m];
  }
  if (rank == 0 && tid == 0) {
    t.S[S_RNORM2] = rr;
    t.S[S_RHO] = rho;
    t.S[S_RHO_PREV] = rho_prev;
    t.I[I_IT] = it;
    t.I[I_TOTAL_IT] += it;
    t.I[I_CONVERGED] = conv;
    t.I[I_DONE] = 1;
  }
}

}  // namespace pcfd
