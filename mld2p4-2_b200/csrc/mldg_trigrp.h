// mldg_trigrp.h -- host-side plan of the grouped triangular solve
// (mldg_trsv_grp.cuh): consecutive dependency levels of a unit-triangular
// factor joined into groups, each group's diagonal block inverted explicitly.
#pragma once
#include <cstdint>
#include <memory>
#include <vector>

namespace mldg {

struct GroupEntry {
  int col;
  double val;
};
struct GroupRow {  // entries of V and W, columns ascending
  const GroupEntry *v = nullptr, *w = nullptr;
  int nv = 0, nw = 0;
};

// Rows are positions (dependency-level order).  With L_gg the unit-triangular
// diagonal block of a group g and L_g< its part left of the block, the plan
// holds
//   W = diag_g(L_gg^{-1})         (its rows include the unit diagonal)
//   V = diag_g(L_gg^{-1}) L_g<    (columns: positions of earlier groups)
// so that L x = b is x_g = (W b)_g - (V x)_g, group after group.
struct TriGroups {
  std::vector<int> gptr;  // groups + 1 first positions
  std::vector<GroupRow> row;
  int64_t entries = 0;    // of V and W together
  std::vector<std::vector<std::unique_ptr<GroupEntry[]>>> store;  // the rows' memory
};

// lvl_ptr: levels + 1 first positions; (irp, dep, val): the factor's strict
// part by position, dep the positions of the dependencies.  A group grows by
// whole levels while it holds at most `budget` entries of V and W together,
// no row of either has more than `row`, and every row of W has an absolute sum
// of at most `growth` (a bound on ||L_gg^{-1}||, by which the errors of the
// explicit inverse can exceed those of a substitution); a single level is always a
// group (W = I, V = L).  The rows of a level are shared by the OpenMP threads;
// idim=45's factors (91,125 rows of 3 entries; 10,978 of 14), N and T, take 35
// ms on 16 cores.
void build_tri_groups(const std::vector<int> &lvl_ptr, const std::vector<int> &irp, const std::vector<int> &dep,
                      const std::vector<double> &val, int64_t budget, int row, double growth,
                      TriGroups *out);

}  // namespace mldg
