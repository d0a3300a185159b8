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
// batches: 64 cavities in FP64 7.48 -> 4.16, 256 mixed 13.0 -> 10.4, 24 odd 5.4 -> 3.5.
#pragma once
#include "common.cuh"

namespace pcfd {

template <class T> struct PatEntry;
template <> struct alignas(8) PatEntry<float> { int off; float val; };
template <> struct alignas(16) PatEntry<double> { double val; int off; int pad; };

__device__ __forceinline__ void pat_load(const PatEntry<float>* e, int* off, float* val) {
  const int2 w = __ldg(reinterpret_cast<const int2*>(e));
  *off = w.x;
  *val = __int_as_float(w.y);
}
__device__ __forceinline__ void pat_load(const PatEntry<double>* e, int* off, double* val) {
  const int4 w = __ldg(reinterpret_cast<const int4*>(e));
  *val = __hiloint2double(w.y, w.x);
  *off = w.z;
}

// How a row's base index follows from the row: its own index, the cell of the coarser
// grid it lies in, or the first cell of the finer grid inside it.
enum PatBase { PB_SAME = 0, PB_COARSER = 1, PB_FINER = 2 };

// An operator of one source (K2 = 0), or of two: K entries on the first from its base
// index, then K2 on the second, a vector on the rows' own grid.
template <class T>
struct Pat {
  const uint16_t* pid;        // pattern of each row
  const PatEntry<T>* tab;     // K + K2 entries per pattern, each part padded with (0, 0)
  int n, K, K2;               // rows, entries per pattern
  int base, ny_r, ny_c;       // PatBase; columns (y cells) of the row and the source grid
  int fx, fy;                 // coarsening factors between them (1 or 2)
};

template <class T>
__host__ __device__ __forceinline__ int pat_base(const Pat<T>& E, int row) {
  if (E.base == PB_SAME) return row;
  const int i = row / E.ny_r, j = row - i * E.ny_r;
  return E.base == PB_COARSER ? (i >> (E.fx - 1)) * E.ny_c + (j >> (E.fy - 1))
                              : (i << (E.fx - 1)) * E.ny_c + (j << (E.fy - 1));
}

// Entries whose gathers are in flight together: 16 values over the GS members.
template <class T, int GS>
__host__ __device__ constexpr int pat_unroll() {
  constexpr int u = 16 / GS;
  return u < 2 ? 2 : u > 8 ? 8 : u;
}

// acc[g] += sum over `count` entries tb[0 ..] applied to the GS vectors src from index
// base.  Every member's pointer is valid (an absent one repeats another's), so that no
// branch separates the members' gathers.  shift: subtracted from every gathered value
// (the mean of a projected residual).  KC > 0: the count, known when compiling.
template <int GS, int KC, bool SHIFT, class T>
__device__ __forceinline__ void pat_entries(const PatEntry<T>* tb, int count, int base, const T* const (&src)[GS],
                                            const T (&shift)[GS], T (&acc)[GS]) {
  constexpr int U = KC > 0 ? KC : pat_unroll<T, GS>();
  if (KC > 0) count = KC;
  for (int k = 0; k < count; k += U) {
    int at[U];
    T val[U], x[U][GS];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      at[u] = 0;
      val[u] = (T)0;
      if (KC > 0 || k + u < count) pat_load(tb + k + u, &at[u], &val[u]);
      at[u] += base;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int g = 0; g < GS; ++g) x[u][g] = src[g][at[u]];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int g = 0; g < GS; ++g) acc[g] += val[u] * (SHIFT ? x[u][g] - shift[g] : x[u][g]);
  }
}

}  // namespace pcfd
