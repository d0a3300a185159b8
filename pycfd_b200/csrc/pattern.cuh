// Sparse operators as tables of row patterns.
//
// On a regular grid almost every row of a multigrid operator is the same stencil with
// the same coefficients; only rows near walls, seams and bodies differ.  A row is then
// a base index (the row's own cell, or the cell of the other grid it belongs to) plus
// one of a few patterns of (offset, value) entries -- 9 to 40 patterns for the levels
// of a closed or periodic box, about 200 around a cylinder -- so the operator is read
// from a table of some kilobytes that stays in L1 instead of 8 or 12 bytes per entry
// and row from L2 or DRAM, a thread keeps a whole row (or a contiguous part of one),
// and the rows of a warp, adjacent along y, gather adjacent values.  Rows share a
// pattern only where offsets and values (in the storage type) are equal bit for bit.
//
// The V-cycle with one sweep per level runs in three kinds of product, all the same
// linear map as the sweeps, restrictions and prolongations it stands for
// (pycfd/core/multigrid.py:430-474):
//   down  b_l = M_l b_{l-1},            M_l = R_l (I - A_{l-1} W_{l-1})
//   up    x_l = Q_l x_{l+1} + G_l b_l,  Q_l = (I - W_l A_l) P_{l+1}, G_l = W_l (2 I - A_l W_l)
// (the prolongation onto the first sweep W b and the sweep that follows it, as one
// product of the coarse iterate and one of the right-hand side), so a cycle takes one
// launch per level and direction and stores one vector per level and direction.
// Measured on B200 against the stored operators (ms per step): 512x512 vortex 2.67 ->
// 1.91, 2048x1024 cylinder 15.9 -> 10.2, 512x256 cylinder in the mixed form 2.39 -> 2.06;
// batches: 64 cavities in FP64 7.48 -> 4.16, 256 mixed 13.0 -> 10.4, 24 odd 5.4 -> 3.5
// (with entries in units of four, tiles and groups 2.8).
#pragma once
#include "common.cuh"

namespace pcfd {

template <class T> struct PatEntry;
template <> struct alignas(8) PatEntry<float> { int off; float val; };
template <> struct alignas(16) PatEntry<double> { double val; int off; int pad; };

// The walks over a row's entries below compile for the host too, where the tables are
// checked against the products they hold.
__host__ __device__ __forceinline__ void pat_load(const PatEntry<float>* e, int* off, float* val) {
#ifdef __CUDA_ARCH__
  const int2 w = __ldg(reinterpret_cast<const int2*>(e));
  *off = w.x;
  *val = __int_as_float(w.y);
#else
  *off = e->off;
  *val = e->val;
#endif
}
__host__ __device__ __forceinline__ void pat_load(const PatEntry<double>* e, int* off, double* val) {
#ifdef __CUDA_ARCH__
  const int4 w = __ldg(reinterpret_cast<const int4*>(e));
  *val = __hiloint2double(w.y, w.x);
  *off = w.z;
#else
  *off = e->off;
  *val = e->val;
#endif
}

// How a row's base index follows from the row: its own index, the cell of the coarser
// grid it lies in, or the first cell of the finer grid inside it.
enum PatBase { PB_SAME = 0, PB_COARSER = 1, PB_FINER = 2 };

// An operator of one source (K2 = 0), or of two: K entries on the first from its base
// index, then K2 on the second, a vector on the rows' own grid.  Both counts are padded to
// units of four entries (kPatUnit), so that no entry needs a test of its own -- except the
// level-0 up product of 2 x 2 aggregates, whose 6 + 5 entries have code of their own in the
// level-0 kernels (pat_is_65).  A coarse level can have rows of 6 and 5 entries too (level 1 of
// a one-cell channel with a bend): its tables are in units, as its kernels read them.
template <class T>
struct Pat {
  const uint16_t* pid;        // pattern of each row
  const PatEntry<T>* tab;     // K + K2 entries per pattern, each part padded with (0, 0)
  int n, K, K2;               // rows, entries per pattern
  int base, ny_r, ny_c;       // PatBase; columns (y cells) of the row and the source grid
  int fx, fy;                 // coarsening factors between them (1 or 2)
  unsigned inv;               // ceil(2^32 / ny_r): rows are divided by a multiplication
};
constexpr int kPatUnit = 4;
// The layout follows from the counts, since every padded one is a multiple of four.  (As a
// member of its own, loaded with the operator, it cost the batch of 256 cavities 0.6 %.)
template <class T>
__host__ __device__ __forceinline__ bool pat_is_65(const Pat<T>& E) { return E.K == 6; }

template <class T>
__host__ __device__ __forceinline__ int pat_base(const Pat<T>& E, int row) {
  if (E.base == PB_SAME) return row;
#ifdef __CUDA_ARCH__
  int i = (int)__umulhi((unsigned)row, E.inv);   // the quotient, or one off
#else
  int i = (int)(((unsigned long long)(unsigned)row * E.inv) >> 32);
#endif
  int j = row - i * E.ny_r;
  if (j < 0) {
    --i;
    j += E.ny_r;
  } else if (j >= E.ny_r) {   // ny_r = 1, whose inverse does not fit
    ++i;
    j -= E.ny_r;
  }
  return E.base == PB_COARSER ? (i >> (E.fx - 1)) * E.ny_c + (j >> (E.fy - 1))
                              : (i << (E.fx - 1)) * E.ny_c + (j << (E.fy - 1));
}
template <class T>
__device__ __forceinline__ const PatEntry<T>* pat_tab(const Pat<T>& E, int row) {
  return E.tab + (long)__ldg(E.pid + row) * (E.K + E.K2);
}

// acc[g] += N entries of tb applied to x(g, index), all gathers issued before the sums.
#pragma nv_exec_check_disable
template <int N, int GS, class T, class A, class X>
__host__ __device__ __forceinline__ void pat_batch(const PatEntry<T>* tb, int base, X x, A (&acc)[GS]) {
  int at[N];
  T val[N];
  A xv[N][GS];
#pragma unroll
  for (int u = 0; u < N; ++u) pat_load(tb + u, &at[u], &val[u]);
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int g = 0; g < GS; ++g) xv[u][g] = x(g, base + at[u]);
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int g = 0; g < GS; ++g) acc[g] += (A)val[u] * xv[u][g];
}

// Units [q0, q1) of a row (its table at tb): xa(g, index) gathers the first source, xb the
// second, for GS members.  Up to 16 gathers are in flight together.
#pragma nv_exec_check_disable
template <int GS, class T, class A, class XA, class XB>
__host__ __device__ __forceinline__ void pat_units(const Pat<T>& E, const PatEntry<T>* tb, int base, int row, int q0, int q1,
                                          XA xa, XB xb, A (&acc)[GS]) {
  const int ka = E.K / kPatUnit, qa = q1 < ka ? q1 : ka;
  int q = q0;
  if constexpr (GS <= 2) {
    for (; q + 2 <= qa; q += 2) pat_batch<2 * kPatUnit, GS>(tb + q * kPatUnit, base, xa, acc);
    if (q < qa) pat_batch<kPatUnit, GS>(tb + q++ * kPatUnit, base, xa, acc);
    for (; q + 2 <= q1; q += 2) pat_batch<2 * kPatUnit, GS>(tb + q * kPatUnit, row, xb, acc);
    if (q < q1) pat_batch<kPatUnit, GS>(tb + q * kPatUnit, row, xb, acc);
  } else if constexpr (GS <= 4) {
    for (; q < qa; ++q) pat_batch<kPatUnit, GS>(tb + q * kPatUnit, base, xa, acc);
    for (; q < q1; ++q) pat_batch<kPatUnit, GS>(tb + q * kPatUnit, row, xb, acc);
  } else {
    for (; q < qa; ++q) {
      pat_batch<kPatUnit / 2, GS>(tb + q * kPatUnit, base, xa, acc);
      pat_batch<kPatUnit / 2, GS>(tb + q * kPatUnit + kPatUnit / 2, base, xa, acc);
    }
    for (; q < q1; ++q) {
      pat_batch<kPatUnit / 2, GS>(tb + q * kPatUnit, row, xb, acc);
      pat_batch<kPatUnit / 2, GS>(tb + q * kPatUnit + kPatUnit / 2, row, xb, acc);
    }
  }
}

// The whole row: the level-0 up product of 2 x 2 aggregates (6 + 5 entries) by code of its
// own, any other by units.
#pragma nv_exec_check_disable
template <bool F65, int GS, class T, class A, class XA, class XB>
__host__ __device__ __forceinline__ void pat_whole(const Pat<T>& E, const PatEntry<T>* tb, int row, XA xa, XB xb, A (&acc)[GS]) {
  const int base = pat_base(E, row);
  if constexpr (F65) {
    pat_batch<6, GS>(tb, base, xa, acc);
    pat_batch<5, GS>(tb + 6, row, xb, acc);
  } else {
    pat_units<GS>(E, tb, base, row, 0, (E.K + E.K2) / kPatUnit, xa, xb, acc);
  }
}

}  // namespace pcfd
