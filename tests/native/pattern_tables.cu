// Host harness of the row-pattern tables (tests/test_pattern_tables.py): builds the
// products of a hierarchy with the library's own code and applies a table entry by entry
// as the kernels walk it.  No kernel and no CUDA call.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <functional>
#include <memory>
#include <thread>
#include <unordered_map>
#include <vector>

#include "../../include/pycfd_b200.h"
#include "../../pycfd_b200/csrc/common.cuh"
#include "../../pycfd_b200/csrc/multigrid.cuh"
#include "../../pycfd_b200/csrc/pattern.cuh"

using namespace pcfd;
#define TRY(x) do { if (int rc_ = (x)) return rc_; } while (0)

namespace {
// what solver.cu declares ahead of the header under test
void csr_transpose(int nrows, int ncols, const int64_t* indptr, const int32_t* idx, const double* data,
                   std::vector<int64_t>& tp, std::vector<int32_t>& ti, std::vector<double>& td) {
  tp.assign(ncols + 1, 0);
  for (int64_t e = 0; e < indptr[nrows]; ++e) tp[idx[e] + 1]++;
  for (int c = 0; c < ncols; ++c) tp[c + 1] += tp[c];
  ti.resize(indptr[nrows]);
  td.resize(indptr[nrows]);
  std::vector<int64_t> pos(tp.begin(), tp.end() - 1);
  for (int r = 0; r < nrows; ++r)
    for (int64_t e = indptr[r]; e < indptr[r + 1]; ++e) {
      ti[pos[idx[e]]] = r;
      td[pos[idx[e]]++] = data[e];
    }
}
template <class T>
int upload(pycfd_solver*, T**, const T*, size_t) { return 1; }
}  // namespace
#include "../../pycfd_b200/csrc/pattern_host.cuh"

namespace {

struct Cycle {
  PatCycle<double> d;
  PatCycle<float> f;
  bool ok_d = false, ok_f = false;
};

template <class T>
bool build(const pycfd_mg_level* lv, int t, PatRule rule, const uint8_t* flags, PatCycle<T>* c) {
  std::vector<std::function<bool()>> tasks;
  return pat_tasks<T>(lv, t, rule, flags, c, &tasks) && run_tasks(tasks);
}

// y = E s1 (+ E2 s2) as the kernels walk a row: level 0's up product whole, any other by
// its units, in `parts` parts added in order.
template <class T>
void apply(const Pat<T>& E0, const PatHost<T>& h, bool level0_up, int parts, const double* s1, const double* s2,
           double* y) {
  Pat<T> E = E0;
  E.pid = h.pid.data();
  E.tab = h.tab.data();
  auto xa = [&](int, int c) { return s1[c]; };
  auto xb = [&](int, int c) { return s2[c]; };
  const int units = (E.K + E.K2) / kPatUnit;
  for (int row = 0; row < E.n; ++row) {
    const PatEntry<T>* tb = E.tab + (long)E.pid[row] * (E.K + E.K2);
    double sum = 0.0;
    if (level0_up) {
      double acc[1] = {0.0};
      if (pat_is_65(E)) pat_whole<true, 1>(E, tb, row, xa, xb, acc);
      else pat_whole<false, 1>(E, tb, row, xa, xb, acc);
      sum = acc[0];
    } else {
      for (int q = 0; q < parts; ++q) {
        double acc[1] = {0.0};
        pat_units<1>(E, tb, pat_base(E, row), row, q * units / parts, (q + 1) * units / parts, xa, xb, acc);
        sum += acc[0];
      }
    }
    y[row] = sum;
  }
}

template <class T>
const PatHost<T>& pick(const PatCycle<T>& c, int l, int up) { return up ? c.up[l] : c.dn[l]; }

}  // namespace

extern "C" {

// The products of levels 0 .. t by the rule of a batch or of a problem alone; solvable: one
// byte per fine cell.
void* pt_build(const pycfd_mg_level* lv, int t, int batch, const uint8_t* solvable) {
  std::unique_ptr<Cycle> c(new Cycle());
  std::vector<uint8_t> flags(lv[0].n);
  for (int k = 0; k < lv[0].n; ++k) flags[k] = solvable[k] ? F_SOLV : 0;
  c->ok_d = build<double>(lv, t, batch ? kPatBatch : kPatAlone, flags.data(), &c->d);
  c->ok_f = build<float>(lv, t, batch ? kPatBatch : kPatAlone, flags.data(), &c->f);
  return c.release();
}
void pt_free(void* h) { delete (Cycle*)h; }
int pt_ok(void* h, int single) { return single ? ((Cycle*)h)->ok_f : ((Cycle*)h)->ok_d; }

// out: K, K2, rows, patterns, 6 + 5 layout.
void pt_info(void* h, int single, int l, int up, int* out) {
  auto fill = [&](const auto& p) {
    out[0] = p.v.K;
    out[1] = p.v.K2;
    out[2] = p.v.n;
    out[3] = (int)(p.tab.size() / (p.v.K + p.v.K2));
    out[4] = pat_is_65(p.v);
  };
  if (single) fill(pick(((Cycle*)h)->f, l, up));
  else fill(pick(((Cycle*)h)->d, l, up));
}

void pt_apply(void* h, int single, int l, int up, int parts, const double* s1, const double* s2, double* y) {
  const Cycle& c = *(Cycle*)h;
  if (single) apply<float>(pick(c.f, l, up).v, pick(c.f, l, up), up && l == 0, parts, s1, s2, y);
  else apply<double>(pick(c.d, l, up).v, pick(c.d, l, up), up && l == 0, parts, s1, s2, y);
}

// Whether the launch of a product over nx x ny rows of K entries fits the GPU's grid.
int pt_fits(int nx, int ny, int K) {
  Pat<double> E{};
  E.n = nx * ny;
  E.ny_r = ny;
  E.K = K;
  return pat_fits(pat_launch(E, 592 * 256, true));
}

// Counts in hits[nx * ny] the threads of that launch per row, by the kernel's own index
// arithmetic (k_pat); returns the parts of a row.
int pt_cover(int nx, int ny, int K, int* hits) {
  Pat<double> E{};
  E.n = nx * ny;
  E.ny_r = ny;
  E.K = K;
  const PatLaunch p = pat_launch(E, 592 * 256, true);
  for (int by = 0; by < (int)p.grid.y; ++by)
    for (int bx = 0; bx < (int)p.grid.x; ++bx)
      for (int t = 0; t < 256; ++t) {
        int part, i, j;
        pat_thread(t, bx, by, p.L, p.sh, &part, &i, &j);
        if (j < ny && i * ny + j < E.n) ++hits[i * ny + j];
      }
  return p.L;
}

}  // extern "C"
