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


def _plan(mld, T, budget, row, growth, ncols=1, fp32=0, rhs=None):
    f = mld.lib().mldg_grp_plan_check
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_longlong, C.c_int,
                  C.c_double, C.c_int, C.c_void_p]
    n = T.shape[0]
    c = mld.CSR(T.indptr, T.indices, T.data, ncols=n).c()
    if rhs is None:
        rhs = np.random.default_rng(1).uniform(-1, 1, n)
    t = np.zeros(n)
    st = np.zeros(4, np.int64)
    assert f(C.byref(c), 0, None, rhs.ctypes.data, t.ctypes.data, ncols, budget, row, growth, fp32,
             st.ctypes.data) == 0
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


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("a", [0.99, -0.99])
def test_row_sums_near_the_bound(mld, a, fp32):
    """A chain with ||L^{-1}|| = 100 and a smooth solution.  W's rows sum 1 + .99 +
    .99^2 + ..., 63.8 after 101 terms, 64.1 after 102: 101 levels a
    group.  A group's x_g = W b - V x errs by at most 105 u (|W||b| + |V||x|) (101
    terms of W, one of V, their roundings and the storage of b and x), which later
    groups pass on as G^{-1}, G = diag(W) L."""
    n, k = 404, 101
    L = np.eye(n) + np.diag(np.full(n - 1, a), -1)
    D = np.zeros((n, n))
    for g in range(0, n, k):
        D[g:g + k, g:g + k] = L[g:g + k, g:g + k]
    W = np.linalg.inv(D)
    assert 63 < np.abs(W).sum(1).max() <= 64
    V = W @ (L - D)
    b = L @ (np.sin(np.arange(n) / 50.0) + 1.5)
    x = np.zeros(n, np.longdouble)
    for i in range(n):
        x[i] = b[i] - (np.longdouble(a) * x[i - 1] if i else 0)
    t, st = _plan(mld, sp.diags([np.full(n - 1, a)], [-1]).tocsr(), 0, 0, 0.0, fp32=fp32, rhs=b)
    assert st[0] == 0 and st[2] == n // k
    u = 2.0 ** (-24 if fp32 else -53)
    local = 105 * u * (np.abs(W) @ np.abs(b) + np.abs(V) @ np.abs(x).astype(float))
    assert np.all(np.abs(t - x) <= np.abs(np.linalg.inv(W @ L)) @ local)


def test_growing_chain(mld):
    """1 + 3 + 9 + 27 = 40 <= 64 < 121: four levels a group, exactly."""
    _, st = _plan(mld, sp.diags([np.full(59, 3.0)], [-1]).tocsr(), 10 ** 9, 10 ** 6, 0.0)
    assert st[0] == 0 and st[2] == 15
