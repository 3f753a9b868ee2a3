// mldg_trigrp.cpp -- see mldg_trigrp.h.  The rows of one level depend only on
// earlier levels, so a level's rows may be formed in parallel; each row is formed
// by one thread in stored order, so the plan does not depend on the number of
// threads.
#include "mldg_trigrp.h"

#include <omp.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <new>

namespace mldg {

namespace {

typedef GroupEntry Entry;

// Sums entries by column: a value per column and a bit where there is one, so
// that the columns come out in order without a sort (a second bit says where a
// word has any, as a row's columns lie far apart).  V's columns lie before the
// group and W's in it, so one sum holds a row of both.
class RowSum {
 public:
  explicit RowSum(int n)
      : val_(new double[(size_t)n]), bit_((size_t)n / 64 + 1, 0), any_(bit_.size() / 64 + 1, 0), lo_(any_.size()) {}
  void add(int col, double v) {
    uint64_t &w = bit_[(size_t)col >> 6];
    const uint64_t m = (uint64_t)1 << (col & 63);
    if (w & m) {
      val_[col] += v;
      return;
    }
    if (!w) {
      const size_t a = (size_t)col >> 12;
      any_[a] |= (uint64_t)1 << (col >> 6 & 63);
      lo_ = std::min(lo_, a);
      hi_ = std::max(hi_, a);
    }
    w |= m;
    val_[col] = v;
    ++size_;
  }
  size_t size() const { return size_; }
  // the entries in column order; leaves no entry
  void take(Entry *out) {
    for (size_t a = lo_; a <= hi_ && size_; ++a) {
      for (uint64_t u = any_[a]; u; u &= u - 1) {
        const size_t w = a << 6 | (size_t)__builtin_ctzll(u);
        for (uint64_t b = bit_[w]; b; b &= b - 1) {
          const int col = (int)(w << 6) + __builtin_ctzll(b);
          *out++ = {col, val_[col]};
        }
        bit_[w] = 0;
      }
      any_[a] = 0;
    }
    lo_ = any_.size();
    hi_ = 0;
    size_ = 0;
  }

 private:
  std::unique_ptr<double[]> val_;
  std::vector<uint64_t> bit_, any_;
  size_t lo_, hi_ = 0, size_ = 0;
};

// A thread's work space: a row's sum, and a bump allocator whose rows keep their
// address until the plan is done.
struct Worker {
  std::unique_ptr<RowSum> sum;
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
                      const std::vector<double> &val, int64_t budget, int row, double growth,
                      TriGroups *out) {
  const int nl = (int)lvl_ptr.size() - 1, n = nl > 0 ? lvl_ptr[nl] : 0;
  out->gptr.assign(1, 0);
  out->row.resize((size_t)n);
  std::vector<GroupRow> &rows = out->row;
  std::vector<Worker> workers((size_t)omp_get_max_threads());
  out->store.resize(workers.size());
  for (size_t t = 0; t < workers.size(); ++t) workers[t].blocks = &out->store[t];
  // row p of V and W, in a group that starts at position g0
  auto row_of = [&](Worker &k, int p, int g0) -> const GroupRow & {
    RowSum &s = *k.sum;
    s.add(p, 1.0);
    for (int e = irp[p]; e < irp[p + 1]; ++e) {
      const int q = dep[e];
      const double a = val[e];
      if (q < g0) {
        s.add(q, a);
        continue;
      }
      const GroupRow &r = rows[q];
      for (int i = 0; i < r.nv; ++i) s.add(r.v[i].col, -(a * r.v[i].val));
      for (int i = 0; i < r.nw; ++i) s.add(r.w[i].col, -(a * r.w[i].val));
    }
    GroupRow &r = rows[p];
    const int size = (int)s.size();
    Entry *at = k.alloc((size_t)size);
    s.take(at);
    r.nv = 0;
    while (at[r.nv].col < g0) ++r.nv;
    r.nw = size - r.nv;
    r.v = at;
    r.w = at + r.nv;
    return r;
  };
  // the rows of level L in a group that starts at position g0: entries, or -1
  // where they are more than `most` or a row grows beyond its bounds (given up
  // as soon as one thread sees it).  A level is shared by the threads where its
  // sums are worth it, a few microseconds each: the entries that its rows add
  // up, taking the rows that they depend on to be as long as the last level's.
  int64_t len = 1;
  auto level = [&](int L, int g0, int64_t most) -> int64_t {
    std::atomic<int64_t> tot{0};
    std::atomic<bool> wild{false}, failed{false};
    const int p0 = lvl_ptr[L], p1 = lvl_ptr[L + 1];
    const bool share = (irp[p1] - irp[p0] + p1 - p0) * len > 8192;
    const int chunk = share ? std::max(1, std::min(64, (p1 - p0) / (4 * (int)workers.size()))) : 64;
#pragma omp parallel for schedule(dynamic, 1) if (share)
    for (int c = p0; c < p1; c += chunk) {
      if (wild.load(std::memory_order_relaxed) || failed.load(std::memory_order_relaxed)) continue;
      try {
        Worker &k = workers[share ? (size_t)omp_get_thread_num() : 0];
        if (!k.sum) k.sum.reset(new RowSum(n));
        int64_t got = 0;
        for (int p = c; p < std::min(c + chunk, p1); ++p) {
          const GroupRow &r = row_of(k, p, g0);
          double sum = 0.0;
          for (int i = 0; i < r.nw; ++i) sum += std::fabs(r.w[i].val);
          if (r.nw > 1 && (!(sum <= growth) || std::max(r.nv, r.nw) > row)) wild = true;
          got += r.nv + r.nw;
        }
        if (tot.fetch_add(got, std::memory_order_relaxed) + got > most) wild = true;
      } catch (const std::bad_alloc &) {  // no exception may leave the parallel loop
        failed = true;
      }
    }
    if (failed) throw std::bad_alloc();
    if (wild) return -1;
    len = 1 + tot / std::max(1, p1 - p0);
    return tot;
  };
  int64_t held = 0;
  for (int L = 0; L < nl; ++L) {
    const bool joins = lvl_ptr[L] > out->gptr.back();
    int64_t t = joins ? level(L, out->gptr.back(), budget - held) : -1;
    if (t < 0) {  // the first level of a group, whatever its size
      if (joins) out->gptr.push_back(lvl_ptr[L]);
      held = 0;
      t = level(L, lvl_ptr[L], INT64_MAX);
    }
    held += t;
    out->entries += t;
  }
  out->gptr.push_back(n);
}

}  // namespace mldg
