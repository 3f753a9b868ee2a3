"""CPU: the groups of a grouped triangular plan against a direct restatement of
their rule (whole levels joined while the entries of V and W, a row's length
and the absolute row sums of W stay within bounds), and the plan's independence
of the number of threads."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp


def _lower(n, per_row, size, near, seed):
    rng = np.random.default_rng(seed)
    i, j = [], []
    for r in range(1, n):
        lo = max(0, r - near)
        k = min(r - lo, int(rng.integers(0, per_row + 1)))
        for c in rng.choice(np.arange(lo, r), k, replace=False):
            i.append(r)
            j.append(c)
    T = sp.csr_matrix((size * rng.uniform(0.1, 1, len(i)), (i, j)), shape=(n, n))
    T.sort_indices()
    return T


def _plan(mld, T, budget, row, growth, ncols=1):
    f = mld.lib().mldg_grp_plan_check
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_longlong, C.c_int,
                  C.c_double, C.c_int, C.c_void_p]
    n = T.shape[0]
    c = mld.CSR(T.indptr, T.indices, T.data, ncols=n).c()
    rhs = np.random.default_rng(1).uniform(-1, 1, n)
    t = np.zeros(n)
    st = np.zeros(4, np.int64)
    assert f(C.byref(c), 0, None, rhs.ctypes.data, t.ctypes.data, ncols, budget, row, growth, 0, st.ctypes.data) == 0
    return t, st


def _rule(T, budget, row, growth):
    """(groups, entries) by the rule, rows as dictionaries."""
    n = T.shape[0]
    level = np.zeros(n, int)
    for r in range(n):
        c = T.indices[T.indptr[r]:T.indptr[r + 1]]
        level[r] = 1 + level[c].max() if len(c) else 0
    rows = {}

    def entries(rs, start):
        made = {}
        for r in rs:
            v, w = {}, {r: 1.0}
            for k in range(T.indptr[r], T.indptr[r + 1]):
                q, a = T.indices[k], T.data[k]
                if level[q] < start:
                    v[q] = v.get(q, 0.0) + a
                    continue
                for d, s in ((v, rows[q][0]), (w, rows[q][1])):
                    for c, x in s.items():
                        d[c] = d.get(c, 0.0) - a * x
            made[r] = (v, w)
        return made

    groups, held, total, start = 0, 0, 0, None
    for L in range(level.max() + 1):
        rs = np.flatnonzero(level == L)
        ok = False
        if start is not None:
            made = entries(rs, start)
            size = sum(len(v) + len(w) for v, w in made.values())
            ok = held + size <= budget and all(
                len(w) == 1 or (max(len(v), len(w)) <= row and sum(abs(x) for x in w.values()) <= growth)
                for v, w in made.values())
        if not ok:
            start, held, groups = L, 0, groups + 1
            made = entries(rs, start)
            size = sum(len(v) + len(w) for v, w in made.values())
        rows.update(made)
        held += size
        total += size
    return groups, total


@pytest.mark.parametrize("budget,row,growth", [(10 ** 6, 10 ** 6, 1e30), (400, 10 ** 6, 1e30), (10 ** 6, 7, 1e30),
                                               (10 ** 6, 10 ** 6, 2.5), (900, 40, 5.0), (1, 1, 1.0)])
@pytest.mark.parametrize("n,per_row,near", [(1, 1, 1), (70, 3, 9), (400, 4, 400), (640, 8, 40)])
def test_rule(mld, n, per_row, near, budget, row, growth):
    T = _lower(n, per_row, 0.4, near, n + per_row)
    _, st = _plan(mld, T, budget, row, growth)
    assert st[0] == 0
    assert (st[2], st[3]) == _rule(T, budget, row, growth)


_CHILD = """
import sys
sys.path[:0] = {path!r}
import hashlib
from conftest import load_package
from test_grp_groups import _lower, _plan
mld = load_package()
for n, per_row, near, budget in ((3000, 6, 500, 60000), (20000, 3, 20000, 0)):
    t, st = _plan(mld, _lower(n, per_row, 0.3, near, n), budget, 0, 0.0, 4)
    print(st.tolist(), hashlib.sha256(t.tobytes()).hexdigest())
"""


def test_threads_do_not_change_the_plan():
    here = os.path.dirname(os.path.abspath(__file__))
    out = [subprocess.run([sys.executable, "-c", _CHILD.format(path=[here, os.path.join(here, "..", "oracle")])],
                          env=dict(os.environ, OMP_NUM_THREADS=k), capture_output=True, text=True, check=True).stdout
           for k in ("1", "2", "7")]
    assert out[0].count("[0,") == 2 and out[0] == out[1] == out[2]
