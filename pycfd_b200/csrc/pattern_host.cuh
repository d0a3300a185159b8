// Host side of the row patterns: the down and up products of a hierarchy formed from
// its A, P and W in double precision, and their rows sorted into patterns.  Included in
// solver.cu after its upload helpers.
#pragma once

namespace {

// A CSR matrix owned elsewhere, and one of our own.
struct CsrV {
  int n, m;
  const int64_t* ptr;
  const int32_t* idx;
  const double* val;
};
struct Csr {
  int n = 0, m = 0;
  std::vector<int64_t> ptr;
  std::vector<int32_t> idx;
  std::vector<double> val;
  operator CsrV() const { return CsrV{n, m, ptr.data(), idx.data(), val.data()}; }
};

// A B; a row's columns come out sorted.
Csr csr_mul(const CsrV& A, const CsrV& B) {
  Csr c;
  c.n = A.n;
  c.m = B.m;
  c.ptr.assign(A.n + 1, 0);
  c.idx.reserve((size_t)A.ptr[A.n] * 3);
  c.val.reserve((size_t)A.ptr[A.n] * 3);
  std::vector<int> mark(B.m, -1), cols;
  std::vector<double> acc(B.m, 0.0);
  for (int r = 0; r < A.n; ++r) {
    cols.clear();
    for (int64_t e = A.ptr[r]; e < A.ptr[r + 1]; ++e) {
      const int k = A.idx[e];
      const double a = A.val[e];
      for (int64_t f = B.ptr[k]; f < B.ptr[k + 1]; ++f) {
        const int j = B.idx[f];
        if (mark[j] != r) {
          mark[j] = r;
          acc[j] = 0.0;
          cols.push_back(j);
        }
        acc[j] += a * B.val[f];
      }
    }
    std::sort(cols.begin(), cols.end());
    for (int j : cols) {
      c.idx.push_back(j);
      c.val.push_back(acc[j]);
    }
    c.ptr[r + 1] = (int64_t)c.idx.size();
  }
  return c;
}

// A^T (its rows' columns ascend).
Csr csr_t(const CsrV& A) {
  Csr t;
  t.n = A.m;
  t.m = A.n;
  csr_transpose(A.n, A.m, A.ptr, A.idx, A.val, t.ptr, t.idx, t.val);
  return t;
}

// X - Y, both with sorted rows; exact zeros are dropped.
Csr csr_sub(const CsrV& X, const CsrV& Y) {
  Csr c;
  c.n = X.n;
  c.m = X.m;
  c.ptr.assign(X.n + 1, 0);
  c.idx.reserve((size_t)std::max(X.ptr[X.n], Y.ptr[Y.n]));
  c.val.reserve((size_t)std::max(X.ptr[X.n], Y.ptr[Y.n]));
  auto put = [&](int j, double v) {
    if (v == 0.0) return;
    c.idx.push_back(j);
    c.val.push_back(v);
  };
  for (int r = 0; r < X.n; ++r) {
    int64_t e = X.ptr[r], f = Y.ptr[r];
    const int64_t e1 = X.ptr[r + 1], f1 = Y.ptr[r + 1];
    while (e < e1 || f < f1) {
      if (f == f1 || (e < e1 && X.idx[e] < Y.idx[f])) {
        put(X.idx[e], X.val[e]);
        ++e;
      } else if (e == e1 || Y.idx[f] < X.idx[e]) {
        put(Y.idx[f], -Y.val[f]);
        ++f;
      } else {
        put(X.idx[e], X.val[e] - Y.val[f]);
        ++e;
        ++f;
      }
    }
    c.ptr[r + 1] = (int64_t)c.idx.size();
  }
  return c;
}

void csr_scale_rows(Csr* A, const double* w) {
  for (int r = 0; r < A->n; ++r)
    for (int64_t e = A->ptr[r]; e < A->ptr[r + 1]; ++e) A->val[e] *= w[r];
}
void csr_scale_cols(Csr* A, const double* w) {
  for (size_t e = 0; e < A->val.size(); ++e) A->val[e] *= w[A->idx[e]];
}

// A copy with every row's columns ascending (duplicates, which a sum over the row would
// add, stay side by side: the caller's matrices have none).
Csr csr_sorted(const CsrV& A) {
  Csr c;
  c.n = A.n;
  c.m = A.m;
  c.ptr.assign(A.ptr, A.ptr + A.n + 1);
  c.idx.assign(A.idx, A.idx + A.ptr[A.n]);
  c.val.assign(A.val, A.val + A.ptr[A.n]);
  std::vector<std::pair<int32_t, double>> row;
  for (int r = 0; r < A.n; ++r) {
    if (std::is_sorted(c.idx.begin() + c.ptr[r], c.idx.begin() + c.ptr[r + 1])) continue;
    row.clear();
    for (int64_t e = c.ptr[r]; e < c.ptr[r + 1]; ++e) row.push_back({c.idx[e], c.val[e]});
    std::stable_sort(row.begin(), row.end(), [](const std::pair<int32_t, double>& a,
                                                const std::pair<int32_t, double>& b) { return a.first < b.first; });
    for (size_t k = 0; k < row.size(); ++k) {
      c.idx[c.ptr[r] + k] = row[k].first;
      c.val[c.ptr[r] + k] = row[k].second;
    }
  }
  return c;
}

CsrV level_A(const pycfd_mg_level& f) { return CsrV{f.n, f.n, f.a_indptr, f.a_indices, f.a_data}; }
CsrV level_P(const pycfd_mg_level& f, const pycfd_mg_level& c) {
  return CsrV{f.n, c.n, c.p_indptr, c.p_indices, c.p_data};
}

// M = R (I - A W), the restriction from level f onto level c.
Csr down_product(const pycfd_mg_level& f, const pycfd_mg_level& c) {
  const Csr R = csr_t(level_P(f, c));
  Csr RA = csr_mul(R, level_A(f));
  csr_scale_cols(&RA, f.weighted_dinv);
  return csr_sub(R, RA);
}
// Q = (I - W A) P and G = W (2 I - A W), which close level f above level c.
void up_products(const pycfd_mg_level& f, const pycfd_mg_level& c, Csr* Q, Csr* G) {
  Csr AP = csr_mul(level_A(f), level_P(f, c));
  csr_scale_rows(&AP, f.weighted_dinv);
  *Q = csr_sub(csr_sorted(level_P(f, c)), AP);
  Csr D;
  D.n = D.m = f.n;
  D.ptr.resize(f.n + 1);
  D.idx.resize(f.n);
  D.val.resize(f.n);
  for (int r = 0; r < f.n; ++r) {
    D.ptr[r + 1] = r + 1;
    D.idx[r] = r;
    D.val[r] = 2.0 * f.weighted_dinv[r];
  }
  Csr WAW = csr_sorted(level_A(f));
  csr_scale_cols(&WAW, f.weighted_dinv);
  csr_scale_rows(&WAW, f.weighted_dinv);
  *G = csr_sub(D, WAW);
}

// Runs the tasks on a few host threads; false if any of them answers false or throws.
bool run_tasks(const std::vector<std::function<bool()>>& tasks) {
  std::atomic<size_t> next{0};
  std::atomic<bool> ok{true};
  auto work = [&]() {
    for (size_t k; (k = next.fetch_add(1)) < tasks.size();) {
      try {
        if (!tasks[k]()) ok = false;
      } catch (...) {
        ok = false;
      }
    }
  };
  std::vector<std::thread> pool;
  const size_t want = std::min<size_t>({tasks.size(), 8, std::max(1u, std::thread::hardware_concurrency())});
  try {
    for (size_t k = 1; k < want; ++k) pool.emplace_back(work);
  } catch (...) {   // fewer threads: the rest of the tasks run here
  }
  work();
  for (auto& t : pool) t.join();
  return ok;
}

// The geometry of a product between a grid of sr (rows) and sc (columns): the base
// rule, or false where the shapes are not grids coarsened by 1 or 2 along each axis.
template <class T>
bool pat_shape(Pat<T>* E, int nr, int rx, int ry, int nc, int cx, int cy) {
  if ((long)rx * ry != nr || (long)cx * cy != nc) return false;
  E->n = nr;
  E->ny_r = ry;
  E->inv = (unsigned)std::min<unsigned long long>(0xffffffffull, ((1ull << 32) + ry - 1) / (unsigned)ry);
  E->ny_c = cy;
  E->fx = E->fy = 1;
  E->base = PB_SAME;
  if (nr == nc && rx == cx && ry == cy) return true;
  const int fx = nr > nc ? rx : cx, fy = nr > nc ? ry : cy, sx = nr > nc ? cx : rx, sy = nr > nc ? cy : ry;
  E->fx = sx == fx ? 1 : 2;
  E->fy = sy == fy ? 1 : 2;
  E->base = nr > nc ? PB_COARSER : PB_FINER;
  return (fx + E->fx - 1) / E->fx == sx && (fy + E->fy - 1) / E->fy == sy;
}

// Host copy of a pattern operator.
template <class T>
struct PatHost {
  Pat<T> v{};
  std::vector<uint16_t> pid;
  std::vector<PatEntry<T>> tab;
};

// How many patterns pay, measured on masks with nearly as many patterns as rows (one solid
// cell at a random place of every 4 x 4 block), ms per step.
// One problem alone: at most one per 4 rows on levels over 16384 rows, where a row with a
// pattern of its own reads its table uncoalesced (FP64 400x400: 2.3 with the stored
// operators, 2.6 on patterns; 500x500 2.8 and 2.9); smaller levels stay in L1 and L2 whatever
// their patterns (256x256 1.63 stored, 1.56 on patterns, 64x64 1.06 and 0.87).
// dense (a batch): no limit but the 65,535 a row can name.  Against the default level-by-level
// cycle the patterns are always faster (FP64 / mixed, each problem its own mask: 8 of 256x256
// 8.4 / 8.7 -> 7.3 / 6.6, 24 of 256x256 17.3 / 15.9 -> 15.7 / 14.1, 8 of 400x400 13.6 / 13.6
// -> 12.8 / 12.4, 64 of 128x128 11.6 / 10.2 -> 11.2 / 9.3).  Against the fused down sweep on
// stored operators they gain less (one mask 400x400 6.1 / 6.0 -> 4.7 / 5.0, 8 of 256x256 7.6 /
// 7.5 -> 7.3 / 6.6) and lose up to 6 % where the tables of many such masks outgrow L2 (64 of
// 128x128 10.6 / 9.0 -> 11.2 / 9.3, 8 of 400x400 12.4 / 11.8 -> 12.8 / 12.4); a limit per
// structure would not see that, and one per engine would tie a problem's route to its
// neighbours.
//
// How wide rows may be: a level above the closing one whose widest row of A has more than
// `widest` entries keeps its structure on stored operators.  Uniform cells of aspect 1.5 and
// more coarsen along one axis at a time, and their rows grow to hundreds and thousands of
// entries (square cells stay near 100): the products grow with the square of the width, hardly
// two rows are equal, and a row's table is read by one lane at a stride of the whole row.
// ms, stored -> patterns.  Solves of one problem, FP64 / mixed: width 225 (256x256) 0.53 / 0.61
// -> 0.51 / 0.52; 349 (192x192) 0.69 / 0.66 -> 0.68 / 0.59, (256x256) 0.98 / 1.01 -> 0.91 /
// 0.72, (256x128) 0.78 / 0.76 -> 0.84 / 0.72; 425 (160x160) 0.85 / 0.77 -> 1.01 / 0.80; 1155
// (400x100) 0.92 / 1.09 -> 1.48 / 1.29; 1577 (512x256) 2.48 -> 3.12.  Steps of 64 problems,
// default down sweep (and the fused one on stored operators): width 225 (160x160) 7.5 / 7.9
// (6.3 / 6.8) -> 6.4 / 6.1; 349 (96x96) 5.7 / 5.0 (4.7 / 4.2) -> 5.9 / 4.7, and 256 of them
// 13.4 / 10.9 (11.7 / 9.2) -> 16.9 / 11.9; 1361 (160x160) 16.8 / 13.8 (14.1 / 11.6) -> 22.8 /
// 18.8.
struct PatRule {
  bool dense;
  int widest;
};
constexpr PatRule kPatAlone{false, 400}, kPatBatch{true, 256};

// The rows of A (and of B, the second source) as patterns, or false where there are
// more than the rule allows.  liveA, liveB: entries at columns whose source value is
// zero by definition are dropped.
// up0: the level-0 up product, whose kernels read 6 + 5 entries without padding.
template <class T>
bool pat_build(const CsrV& A, const uint8_t* liveA, const CsrV* B, const uint8_t* liveB, bool up0, bool dense,
               PatHost<T>* out) {
  Pat<T>& E = out->v;
  const int n = A.n;
  int K = 1, K2 = 0;
  for (int r = 0; r < n; ++r) {
    K = std::max<int>(K, (int)(A.ptr[r + 1] - A.ptr[r]));
    if (B) K2 = std::max<int>(K2, (int)(B->ptr[r + 1] - B->ptr[r]));
  }
  if (!(up0 && K == 6 && K2 == 5)) {   // units of four entries (pattern.cuh)
    K = (K + kPatUnit - 1) / kPatUnit * kPatUnit;
    K2 = (K2 + kPatUnit - 1) / kPatUnit * kPatUnit;
  }
  const int KT = K + K2;
  const size_t most = std::min<size_t>(65535, n > 16384 && !dense ? (size_t)n / 4 : (size_t)n);
  E.K = K;
  E.K2 = K2;
  out->pid.resize(n);
  out->tab.clear();
  std::vector<PatEntry<T>> row(KT);
  std::unordered_multimap<uint64_t, int> seen;
  int recent[2] = {-1, -1};   // rows along y alternate between two patterns of a coarsened grid
  auto same = [&](int p) {
    const PatEntry<T>* t = &out->tab[(size_t)p * KT];
    for (int k = 0; k < KT; ++k)
      if (t[k].off != row[k].off || memcmp(&t[k].val, &row[k].val, sizeof(T))) return false;
    return true;
  };
  for (int r = 0; r < n; ++r) {
    uint64_t h = 1469598103934665603ull;
    auto part = [&](const CsrV& M, const uint8_t* live, int base, int k0, int kn) {
      int k = k0;
      for (int64_t e = M.ptr[r]; e < M.ptr[r + 1]; ++e) {
        const T v = (T)M.val[e];
        if (v == (T)0 || (live && !live[M.idx[e]])) continue;
        row[k].off = M.idx[e] - base;
        row[k].val = v;
        uint64_t bits = 0;
        memcpy(&bits, &v, sizeof(T));
        h = (h ^ (uint32_t)row[k].off) * 1099511628211ull;
        h = (h ^ bits) * 1099511628211ull;
        h ^= h >> 29;
        ++k;
      }
      for (; k < k0 + kn; ++k) row[k] = PatEntry<T>{};
    };
    part(A, liveA, pat_base(E, r), 0, K);
    if (B) part(*B, liveB, r, K, K2);
    int id = -1;
    for (int q : recent)
      if (id < 0 && q >= 0 && same(q)) id = q;
    if (id < 0) {
      auto range = seen.equal_range(h);
      for (auto it = range.first; it != range.second && id < 0; ++it)
        if (same(it->second)) id = it->second;
    }
    if (id < 0) {
      id = (int)(out->tab.size() / KT);
      if ((size_t)id >= most) return false;
      seen.emplace(h, id);
      out->tab.insert(out->tab.end(), row.begin(), row.end());
    }
    out->pid[r] = (uint16_t)id;
    if (id != recent[0]) {
      recent[1] = recent[0];
      recent[0] = id;
    }
  }
  return true;
}

// The products of levels 0 .. t of a hierarchy closed by a dense operator at level t:
// dn[l] restricts onto level l (1 .. t), up[l] closes level l (0 .. t - 1) from level
// l + 1 and its own right-hand side.  False where a level has no patterns (the caller
// keeps its general operators).
template <class T>
struct PatCycle {
  std::vector<PatHost<T>> dn, up;
  std::vector<uint8_t> live;   // solvable cells
};
// Appends the cycle's work to `tasks` (largest level first); false where its shapes
// rule patterns out.  out and lv stay as they are until the tasks have run.
template <class T>
bool pat_tasks(const pycfd_mg_level* lv, int t, PatRule rule, const uint8_t* flags, PatCycle<T>* out,
               std::vector<std::function<bool()>>* tasks) {
  out->dn.resize(t + 1);
  out->up.resize(t + 1);
  out->live.resize(lv[0].n);
  for (int c = 0; c < lv[0].n; ++c) out->live[c] = (flags[c] & F_SOLV) ? 1 : 0;
  for (int l = 0; l < t; ++l) {
    const pycfd_mg_level *f = lv + l, *c = lv + l + 1;
    if (!f->a_indptr || !f->weighted_dinv || !c->p_indptr) return false;
    for (int r = 0; r < f->n; ++r)
      if (f->a_indptr[r + 1] - f->a_indptr[r] > rule.widest) return false;
    PatHost<T>*m = &out->dn[l + 1], *q = &out->up[l];
    if (!pat_shape(&m->v, c->n, c->shape_x, c->shape_y, f->n, f->shape_x, f->shape_y) ||
        !pat_shape(&q->v, f->n, f->shape_x, f->shape_y, c->n, c->shape_x, c->shape_y))
      return false;
    const uint8_t* live = l == 0 ? out->live.data() : nullptr;   // the projected residual is zero off the solvable rows
    tasks->push_back([=]() {
      Csr Q, G;
      up_products(*f, *c, &Q, &G);
      const CsrV g = G;
      return pat_build<T>(Q, nullptr, &g, live, l == 0, rule.dense, q);
    });
    tasks->push_back([=]() { return pat_build<T>(down_product(*f, *c), live, nullptr, nullptr, false, rule.dense, m); });
  }
  return true;
}

template <class T>
int pat_upload(pycfd_solver* s, const PatHost<T>& h, Pat<T>* d) {
  *d = h.v;
  uint16_t* pid = nullptr;
  PatEntry<T>* tab = nullptr;
  TRY(upload(s, &pid, h.pid.data(), h.pid.size()));
  TRY(upload(s, &tab, h.tab.data(), h.tab.size()));
  d->pid = pid;
  d->tab = tab;
  return 0;
}

}  // namespace
