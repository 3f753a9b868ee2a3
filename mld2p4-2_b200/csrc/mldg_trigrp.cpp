// mldg_trigrp.cpp -- see mldg_trigrp.h.  The rows of one level depend only on
// earlier levels, so a level's rows may be formed in parallel; each row is formed
// by one thread in stored order, so the plan does not depend on the number of
// threads.
#include "mldg_trigrp.h"

#include <omp.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>

namespace mldg {

namespace {

typedef GroupEntry Entry;

// Sums entries by column in an open-addressing table that grows with the row.
class RowSum {
 public:
  RowSum() : key_(256, -1), val_(256), mask_(255) {}
  void add(int col, double v) {
    if (used_.size() * 2 > (size_t)mask_) grow();
    unsigned h = slot(col);
    while (key_[h] != -1 && key_[h] != col) h = (h + 1) & mask_;
    if (key_[h] == -1) {
      key_[h] = col;
      val_[h] = v;
      used_.push_back(h);
    } else {
      val_[h] += v;
    }
  }
  size_t size() const { return used_.size(); }
  // the entries in column order; leaves the table empty
  void take(Entry *out) {
    size_t k = 0;
    for (unsigned h : used_) {
      out[k++] = {key_[h], val_[h]};
      key_[h] = -1;
    }
    used_.clear();
    std::sort(out, out + k, [](const Entry &a, const Entry &b) { return a.col < b.col; });
  }

 private:
  unsigned slot(int col) const { return ((unsigned)col * 2654435761u >> 9) & mask_; }
  void grow() {
    std::vector<Entry> e(used_.size());
    const size_t k = e.size();
    take(e.data());
    mask_ = mask_ * 2 + 1;
    key_.assign((size_t)mask_ + 1, -1);
    val_.resize((size_t)mask_ + 1);
    for (size_t i = 0; i < k; ++i) add(e[i].col, e[i].val);
  }
  std::vector<int> key_;
  std::vector<double> val_;
  std::vector<unsigned> used_;
  unsigned mask_;
};

// A thread's work space: row sums, and a bump allocator whose rows keep their
// address until the plan is done.
struct Worker {
  RowSum v, w;
  Entry *at = nullptr;
  size_t left = 0;
  std::vector<std::unique_ptr<Entry[]>> *blocks = nullptr;
  Entry *alloc(size_t n) {
    if (n > left) {
      const size_t c = std::max<size_t>(n, 1 << 15);
      blocks->emplace_back(new Entry[c]);
      at = blocks->back().get();
      left = c;
    }
    Entry *p = at;
    at += n;
    left -= n;
    return p;
  }
};

}  // namespace

void build_tri_groups(const std::vector<int> &lvl_ptr, const std::vector<int> &irp, const std::vector<int> &dep,
                      const std::vector<double> &val, int64_t budget, int row, double growth, bool par,
                      TriGroups *out) {
  const int nl = (int)lvl_ptr.size() - 1, n = nl > 0 ? lvl_ptr[nl] : 0;
  out->gptr.assign(1, 0);
  out->row.resize((size_t)n);
  std::vector<GroupRow> &rows = out->row;
  std::vector<Worker> workers(par ? (size_t)omp_get_max_threads() : 1);
  out->store.resize(workers.size());
  for (size_t t = 0; t < workers.size(); ++t) workers[t].blocks = &out->store[t];
  // the rows of level L in a group that starts at position g0: entries, or -1
  // where a row grows beyond its bounds
  auto level = [&](int L, int g0) -> int64_t {
    int64_t tot = 0;
    int wild = 0, failed = 0;
    const int p0 = lvl_ptr[L], p1 = lvl_ptr[L + 1];
#pragma omp parallel for schedule(dynamic, 4) reduction(+ : tot, wild, failed) if (par && p1 - p0 > 64)
    for (int p = p0; p < p1; ++p) try {
      Worker &k = workers[par ? (size_t)omp_get_thread_num() : 0];
      k.w.add(p, 1.0);
      for (int e = irp[p]; e < irp[p + 1]; ++e) {
        const int q = dep[e];
        const double a = val[e];
        if (q < g0) {
          k.v.add(q, a);
          continue;
        }
        const GroupRow &r = rows[q];
        for (int i = 0; i < r.nv; ++i) k.v.add(r.v[i].col, -(a * r.v[i].val));
        for (int i = 0; i < r.nw; ++i) k.w.add(r.w[i].col, -(a * r.w[i].val));
      }
      GroupRow &r = rows[p];
      r.nv = (int)k.v.size();
      r.nw = (int)k.w.size();
      Entry *at = k.alloc((size_t)r.nv + r.nw);
      k.v.take(at);
      k.w.take(at + r.nv);
      r.v = at;
      r.w = at + r.nv;
      double s = 0.0;
      for (int i = 0; i < r.nw; ++i) s += std::fabs(r.w[i].val);
      if (r.nw > 1 && (!(s <= growth) || std::max(r.nv, r.nw) > row)) ++wild;
      tot += r.nv + r.nw;
    } catch (const std::bad_alloc &) {  // no exception may leave the parallel loop
      ++failed;
    }
    if (failed) throw std::bad_alloc();
    return wild ? -1 : tot;
  };
  int64_t held = 0;
  for (int L = 0; L < nl; ++L) {
    int64_t t = level(L, out->gptr.back());
    if (lvl_ptr[L] > out->gptr.back() && (t < 0 || held + t > budget)) {
      out->gptr.push_back(lvl_ptr[L]);
      held = 0;
      t = level(L, lvl_ptr[L]);
    }
    held += t;
    out->entries += t;
  }
  out->gptr.push_back(n);
}

}  // namespace mldg
