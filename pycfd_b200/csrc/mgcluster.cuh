// Multigrid-preconditioned CG of a small grid as ONE launch: a thread-block cluster
// runs the whole solve.
//
// Each CTA owns a band of grid rows whose CG vectors -- r (with the halo rows that the
// products read), p (one halo row each side), q or z, and x -- stay in shared memory for
// the solve.  The V-cycle is the pattern products of pattern.cuh: level 0 reads r from
// shared memory, the vectors of the coarser levels (a few kilobytes) go through L2, and
// from the first level of at most kMcDenseRows rows on one dense operator
// D_t = T_t M_t, x_t = D_t b_{t-1}, closes the cycle (T_t the cycle at and below level t).
// A pass is 2 t + 2 phases between cluster barriers, three of which also carry sums
// (sum z and r.z; p.q; r.r and sum r) that every CTA writes into every other CTA's shared
// memory and adds in CTA order.  Rows of r and z that a neighbour reads are written into
// its halo by the phase that forms them.
//
// The recurrence and the arithmetic are those of the one-kernel-per-phase forms
// (poisson.cuh, batch.cuh; pycfd/core/pressure.py:619-623): vectors stored in T, products
// and stencils accumulated in A, sums and scalars in double.  A problem's result depends
// on nothing but its own record, so a batch of such solves -- one cluster per problem --
// gives the bits of each solved alone with the same cluster size.
//
// What bounds a pass is the chain of barriers (about 0.4 us each) up to about 1,000 cells
// per CTA, and the gathers of the level-0 and level-1 products above; the forms with one
// launch per phase paid 9 to 15 launches per pass, or re-read every CG vector from L2 or
// DRAM in each.
#pragma once
#include <cooperative_groups.h>

#include "cluster.cuh"
#include "common.cuh"
#include "pattern.cuh"
#include "poisson.cuh"

namespace pcfd {

constexpr int kMcThreads = 512;
constexpr int kMcMaxLevels = 10;
constexpr int kMcDenseRows = 512;          // level closed by the dense operator: at most this many rows,
constexpr size_t kMcDenseBytes = 4 << 20;  // ... and this many bytes of operator
constexpr int kMcHalo = 2;                 // halo rows of r (the products reach no further)

// What an inner pass needs of one problem (device record).
template <class T>
struct McProb {
  Geo g;
  const uint8_t* flags;
  const uint8_t* solving;     // batch: the problem takes part (null: always)
  const T* r;                 // initial residual
  T* x;                       // iterate (in and out)
  double* S;
  int* I;
  int singular;
  int maxiter;
  int unit;                   // rows of x a band is made of: the first coarsening factor along x
  int rmax;                   // rows of the largest band
  int t;                      // level the dense operator gives
  int nt, ns;                 // its rows, and the rows of level t - 1
  const T* D;                 // nt x ns, row-major
  Pat<T> dn[kMcMaxLevels];    // 1 .. t - 1
  Pat<T> up[kMcMaxLevels];    // 0 .. t - 1
  T* b[kMcMaxLevels];         // 1 .. t - 1
  T* xl[kMcMaxLevels];        // 1 .. t
  unsigned* cap_set;          // batch: pass cap set by the host (0: none), and where a cap that
  int* capped;                // ended a solve is noted
  uint8_t* solving_out;       // batch: cleared when the solve ends
};

// Dynamic shared memory of a CTA: r, p, q, x, the neighbours' rows of z, the dense
// operator's source, partial sums and a flag byte per cell.
template <class T, class A>
inline size_t mc_smem(int rmax, int ny, int ns) {
  const size_t n = (size_t)rmax * ny;
  return (4 * n + (size_t)(2 * kMcHalo + 2 + 2) * ny + ns) * sizeof(T) + kMcThreads * sizeof(A) + n + 2 * (size_t)ny + 16;
}

// Rows [lo, hi) of operator E in one CTA: a row's entries split over L parts of the block
// where the rows are few.
template <class A, class T, class X1, class X2, class Put>
__device__ __forceinline__ void mc_rows(const Pat<T>& E, int lo, int hi, A* red, X1 x1, X2 x2, Put put) {
  const int n = hi - lo;
  const int K1 = E.K, K = E.K + E.K2;
  int L = 1;
  while (L < 32 && n * 2 * L <= kMcThreads && K >= 4 * L) L *= 2;
  const int rpb = kMcThreads / L, part = (int)threadIdx.x / rpb, rl = (int)threadIdx.x - part * rpb;
  const int per = (K + L - 1) / L, k0 = part * per, k1 = min(K, k0 + per);
  constexpr int U = 8;
  for (int base = lo; base < hi; base += rpb) {
    const int row = base + rl;
    A acc = (A)0;
    if (row < hi) {
      const PatEntry<T>* tb = E.tab + (long)__ldg(E.pid + row) * K;
      const int c0 = pat_base(E, row);
      for (int k = k0; k < k1; k += U) {
        int at[U];
        T val[U];
        A x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          at[u] = 0;
          val[u] = (T)0;
          if (k + u < k1) pat_load(tb + k + u, &at[u], &val[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          x[u] = (A)0;
          if (k + u < k1) x[u] = k + u < K1 ? x1(c0 + at[u]) : x2(row + at[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) acc += (A)val[u] * x[u];
      }
    }
    if (L == 1) {
      if (row < hi) put(row, acc);
      continue;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    if (part == 0 && row < hi) {
      for (int q = 1; q < L; ++q) acc += red[q * rpb + rl];
      put(row, acc);
    }
    __syncthreads();
  }
}

// The block's two sums into every CTA's part[.][rank]; totals after the barrier.
__device__ __forceinline__ void mc_reduce(cooperative_groups::cluster_group& cl, double a0, double a1,
                                          double (*wsum)[kMcThreads / 32], double (*part)[kClMaxCtas], double* t0,
                                          double* t1) {
  constexpr int kWarps = kMcThreads / 32;
  const int lane = (int)threadIdx.x & 31, warp = (int)threadIdx.x >> 5;
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
    if (lane < (int)cl.num_blocks()) cl.map_shared_rank(&part[warp][0], lane)[cl.block_rank()] = v;
  }
  cl.sync();
  cl_total2(part, t0, t1);
}

// One cluster per entry of `order` (null: problem 0).
template <class T, class A>
__global__ void __launch_bounds__(kMcThreads, sizeof(A) == 4 ? 2 : 1)
    k_mg_cluster(const McProb<T>* __restrict__ probs, const int* __restrict__ order) {
  pdl_begin();
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const McProb<T>& P = probs[order ? order[blockIdx.x / C] : 0];
  if (P.solving && !*P.solving) return;   // the same words for every CTA of the cluster
  if (P.I[I_DONE]) return;
  extern __shared__ __align__(16) unsigned char mc_sm[];
  __shared__ double partz[2][kClMaxCtas], partq[2][kClMaxCtas], partr[2][kClMaxCtas];
  __shared__ double wsum[2][kMcThreads / 32];
  __shared__ A dtab[32];
  const Geo g = P.g;
  const int nx = g.nx, ny = g.ny, n = nx * ny;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int H = kMcHalo;
  const int units = (nx + P.unit - 1) / P.unit;
  auto band0 = [&](int k) { return min(nx, (int)((long)k * units / C) * P.unit); };
  const int r0 = band0(rank), r1 = band0(rank + 1), rows = r1 - r0, cells = rows * ny;
  // the layout follows rmax, so that every CTA's arrays lie at the same offsets
  const size_t nmax = (size_t)P.rmax * ny;
  T* rs = reinterpret_cast<T*>(mc_sm);                 // halo, band, halo
  T* ps = rs + nmax + 2 * (size_t)H * ny;              // row, band, row
  T* qs = ps + nmax + 2 * (size_t)ny;                  // q, and z between the cycle and p's update
  T* xs = qs + nmax;
  T* zh = xs + nmax;                                   // west neighbour's last row of z, east neighbour's first
  T* sb = zh + 2 * (size_t)ny;
  A* red = reinterpret_cast<A*>((reinterpret_cast<uintptr_t>(sb + P.ns) + 7) & ~(uintptr_t)7);
  uint8_t* fl = reinterpret_cast<uint8_t*>(red + kMcThreads);   // row, band, row
  T* rb = rs + (size_t)H * ny;
  T* pb = ps + ny;
  const int west = rank > 0 ? rank - 1 : (g.periodic_x ? C - 1 : -1);
  const int east = rank < C - 1 ? rank + 1 : (g.periodic_x ? 0 : -1);
  T *rw = nullptr, *re = nullptr, *zw = nullptr, *ze = nullptr;   // where the neighbours keep our rows
  if (west >= 0) {
    rw = cl.map_shared_rank(rs, west) + (size_t)(H + band0(west + 1) - band0(west)) * ny;
    zw = cl.map_shared_rank(zh, west) + ny;
  }
  if (east >= 0) {
    re = cl.map_shared_rank(rs, east);
    ze = cl.map_shared_rank(zh, east);
  }
  const long c0 = (long)r0 * ny;
  const bool any_dir = g.dir_w | g.dir_e | g.dir_s | g.dir_n;
  const A cx = (A)g.cx, cy = (A)g.cy;

  // ---- load: r with its halo, x, flags with one halo row, the diagonal by face flags
  if (tid < 32) {
    double d = 0.0;   // fine_diag's subtractions in its order
    if (tid & F_W) d -= g.cx;
    if (tid & F_E) d -= g.cx;
    if (tid & F_S) d -= g.cy;
    if (tid & F_N) d -= g.cy;
    dtab[tid] = (A)((tid & F_SOLV) ? d : 1.0);
  }
  if (tid < 2 * kClMaxCtas) {
    (&partz[0][0])[tid] = 0.0;
    (&partq[0][0])[tid] = 0.0;
    (&partr[0][0])[tid] = 0.0;
  }
  for (int il = -H + warp; il < rows + H; il += kMcThreads / 32) {   // a warp per row
    int i = r0 + il;
    if (i < 0) i = g.periodic_x ? i + nx : -1;
    else if (i >= nx) i = g.periodic_x ? i - nx : -1;
    const bool own = il >= 0 && il < rows;
    for (int j = lane; j < ny; j += 32) {
      const long c = (long)i * ny + j;
      rb[(long)il * ny + j] = i >= 0 ? P.r[c] : (T)0;
      if (il >= -1 && il <= rows) {
        const uint8_t f = i >= 0 ? P.flags[c] : 0;
        // bits 5, 6: the first and last column of a row (the wrap of a periodic y axis)
        fl[(il + 1) * ny + j] = (uint8_t)((f & 31) | (j == 0 ? 32 : 0) | (j == ny - 1 ? 64 : 0));
        pb[(long)il * ny + j] = (T)0;
      }
      if (own) xs[il * ny + j] = P.x[c];
    }
  }
  const double n_fluid = (double)g.n_fluid;
  double sum_r = P.S[S_SUM_R], rr = P.S[S_RNORM2], rho = P.S[S_RHO], rho_prev = 1.0, mean_z = 0.0;
  const double atol = P.S[S_ATOL];
  const unsigned cap = P.cap_set ? *P.cap_set : 0u;
  // local index of cell c of the grid in rb (halo rows wrap on a periodic axis)
  const int wrap_lo = -H * ny, wrap_hi = (rows + H) * ny, cbase = (int)c0;
  auto rloc = [&](int c) {
    int k = c - cbase;
    if (g.periodic_x) {
      if (k < wrap_lo) k += n;
      else if (k >= wrap_hi) k -= n;
    }
    return k;
  };
  const int t = P.t;
  int it = 0;
  bool conv = false, was_capped = false;
  cl.sync();

  for (;;) {
    const T mr = (T)(P.singular && g.n_fluid ? sum_r / n_fluid : 0.0);
    const A mra = sizeof(A) == sizeof(T) ? (A)mr : (A)(P.singular && g.n_fluid ? sum_r / n_fluid : 0.0);
    // ---- down: b_1 from r in shared memory, b_2 .. b_{t-1} through L2
    if (t > 1) {
      const Pat<T>& E = P.dn[1];
      const int cyl = E.ny_r;
      mc_rows<A>(E, (r0 / P.unit) * cyl, ((r1 + P.unit - 1) / P.unit) * cyl, red,
                 [&](int c) { return (A)rb[rloc(c)] - mra; }, [&](int) { return (A)0; },
                 [&](int row, A v) { P.b[1][row] = (T)v; });
      cl.sync();
      for (int l = 2; l < t; ++l) {
        const Pat<T>& F = P.dn[l];
        const T* src = P.b[l - 1];
        mc_rows<A>(F, (int)((long)rank * F.n / C), (int)((long)(rank + 1) * F.n / C), red,
                   [&](int c) { return (A)__ldcg(src + c); }, [&](int) { return (A)0; },
                   [&](int row, A v) { P.b[l][row] = (T)v; });
        cl.sync();
      }
    }
    // ---- x_t = D b_{t-1}, a warp per row
    for (int k = tid; k < P.ns; k += kMcThreads)
      sb[k] = t > 1 ? __ldcg(P.b[t - 1] + k) : (T)((A)rb[k] - mra);   // t = 1: one CTA holds the grid
    __syncthreads();
    for (int row = (int)((long)rank * P.nt / C) + warp; row < (int)((long)(rank + 1) * P.nt / C);
         row += kMcThreads / 32) {
      const T* d = P.D + (long)row * P.ns;
      A acc = (A)0;
      for (int k0 = lane; k0 < P.ns; k0 += 8 * 32) {
        T dv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) dv[u] = k0 + 32 * u < P.ns ? __ldg(d + k0 + 32 * u) : (T)0;
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (k0 + 32 * u < P.ns) acc += (A)dv[u] * (A)sb[k0 + 32 * u];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) P.xl[t][row] = (T)acc;
    }
    cl.sync();
    // ---- up: x_{t-1} .. x_1 through L2
    for (int l = t - 1; l >= 1; --l) {
      const Pat<T>& E = P.up[l];
      const T *xc = P.xl[l + 1], *bl = P.b[l];
      mc_rows<A>(E, (int)((long)rank * E.n / C), (int)((long)(rank + 1) * E.n / C), red,
                 [&](int c) { return (A)__ldcg(xc + c); }, [&](int c) { return (A)__ldcg(bl + c); },
                 [&](int row, A v) { P.xl[l][row] = (T)v; });
      cl.sync();
    }
    // ---- z on the band, its edge rows into the neighbours, sum z and r.z
    double a0 = 0.0, a1 = 0.0;
    {
      const Pat<T>& E = P.up[0];
      const T* xc = P.xl[1];
      mc_rows<A>(E, cbase, cbase + cells, red, [&](int c) { return (A)__ldcg(xc + c); },
                 [&](int c) { return (A)rb[rloc(c)] - mra; },
                 [&](int row, A v) {
                   const int k = row - cbase;
                   const T z = (T)v;
                   qs[k] = z;
                   if (k < ny && zw) zw[k] = z;
                   if (k >= cells - ny && ze) ze[k - (cells - ny)] = z;
                   if (fl[ny + k] & F_SOLV) {
                     a0 += (double)z;
                     a1 += (double)rb[k] * (double)z;
                   }
                 });
    }
    double sz, rz;
    mc_reduce(cl, a0, a1, wsum, partz, &sz, &rz);
    mean_z = P.singular && g.n_fluid ? sz / n_fluid : 0.0;
    rho_prev = rho;
    rho = rz - mean_z * sum_r;
    const double beta = it ? rho / rho_prev : 0.0;
    // ---- p = (z - mean z) + beta p on the band and one row each side
    {
      const T tm = (T)mean_z, tb = (T)beta;
      auto pnew = [&](uint8_t f, T z, T po) -> T {
        if constexpr (sizeof(A) == sizeof(T)) {
          const T zz = (f & F_SOLV) ? z - tm : (T)0;
          return it ? po * tb + zz : zz;
        } else {
          const double zz = (f & F_SOLV) ? (double)z - mean_z : 0.0;
          return (T)(it ? (double)po * beta + zz : zz);
        }
      };
#pragma unroll 4
      for (int k = tid; k < cells; k += kMcThreads) pb[k] = pnew(fl[ny + k], qs[k], pb[k]);
      for (int k = tid; k < 2 * ny; k += kMcThreads) {
        const int at = k < ny ? k : (rows + 1) * ny + (k - ny);
        ps[at] = pnew(fl[at], zh[k], ps[at]);
      }
    }
    __syncthreads();
    // ---- q = A p, p.q
    a0 = 0.0;
#pragma unroll 4
    for (int k = tid; k < cells; k += kMcThreads) {
      const uint8_t f = fl[ny + k];
      const T* pc = pb + k;
      A d = dtab[f & 31];
      if (any_dir && (f & F_SOLV)) {   // Dirichlet edges add to the diagonal
        const int il = k / ny;
        d = (A)fine_diag((uint8_t)(f & 31), r0 + il, k - il * ny, g);
      }
      A q = d * (A)pc[0];
      if (f & F_W) q += cx * (A)pc[-ny];
      if (f & F_E) q += cx * (A)pc[ny];
      if (f & F_S) q += cy * (A)pc[(f & 32) ? ny - 1 : -1];
      if (f & F_N) q += cy * (A)pc[(f & 64) ? 1 - ny : 1];
      qs[k] = (T)q;
      a0 += sizeof(A) == sizeof(T) ? (double)pc[0] * (double)(T)q : (double)pc[0] * (double)q;
    }
    double pq, unused;
    mc_reduce(cl, a0, 0.0, wsum, partq, &pq, &unused);
    const double alpha = rho / pq;
    // ---- x += alpha p, r -= alpha q; the edge rows of r into the neighbours; r.r, sum r
    a0 = a1 = 0.0;
#pragma unroll 4
    for (int k = tid; k < cells; k += kMcThreads) {
      xs[k] = (T)((double)xs[k] + alpha * (double)pb[k]);
      const T rn = (T)((double)rb[k] - alpha * (double)qs[k]);
      rb[k] = rn;
      if (k < H * ny && rw) rw[k] = rn;
      if (k >= cells - H * ny && re) re[k - (cells - H * ny)] = rn;
      a0 += (double)rn * (double)rn;
      if (fl[ny + k] & F_SOLV) a1 += (double)rn;
    }
    mc_reduce(cl, a0, a1, wsum, partr, &rr, &sum_r);
    ++it;
    conv = sqrt(rr) < atol;
    if (conv || it >= P.maxiter) break;
    if (cap && it >= (int)cap) {
      was_capped = true;
      break;
    }
  }
  for (int k = tid; k < cells; k += kMcThreads) P.x[c0 + k] = xs[k];
  if (rank == 0 && tid == 0) {
    double* S = P.S;
    int* I = P.I;
    S[S_RNORM2] = rr;
    S[S_RHO] = rho;
    S[S_RHO_PREV] = rho_prev;
    S[S_MEAN_Z] = mean_z;
    S[S_SUM_R] = sum_r;
    S[S_MEAN_R] = g.n_fluid ? sum_r / n_fluid : 0.0;
    I[I_IT] = it;
    I[I_TOTAL_IT] += it;
    I[I_CONVERGED] = conv;
    if (was_capped) {
      *P.capped = 1;
    } else {
      I[I_DONE] = 1;
      if (P.solving_out) *P.solving_out = 0;
    }
  }
}

}  // namespace pcfd
