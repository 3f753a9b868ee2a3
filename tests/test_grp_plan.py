"""CPU: plans of the grouped triangular solve (k_trsv_grp), replayed
task by task through mldg_grp_plan_check, against a direct sparse triangular
solve: both triangles, one to 32 columns, both precisions, group budgets from
one level per group to one group, factors whose inverse grows (the growth
bound), empty rows, and the smallest sizes.

Tolerances: a grouped solve sums each row's terms of the exact solution
operator; with m terms of a factor whose inverse has norm c the error is at
most about m c eps of the data, below 1e-13 (FP64) and 1e-5 (FP32) for the
factors here (m <= 2,000 terms, c <= 64)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sla

from conftest import ANISO, ISO, oracle_params

TOL = {0: 1e-13, 1: 1e-5}


def _check(mld, T, upper, scale, ncols=1, budget=0, row=0, growth=0.0, fp32=0):
    f = mld.lib().mldg_grp_plan_check
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_longlong, C.c_int,
                  C.c_double, C.c_int, C.c_void_p]
    n = T.shape[0]
    m = mld.CSR(T.indptr, T.indices, T.data, ncols=n)
    c = m.c()
    rhs = np.random.default_rng(n).uniform(-1, 1, n)
    t = np.zeros(n)
    st = np.zeros(4, np.int64)
    assert f(C.byref(c), upper, None if scale is None else scale.ctypes.data, rhs.ctypes.data, t.ctypes.data, ncols,
             budget, row, growth, fp32, st.ctypes.data) == 0
    b = rhs if scale is None else scale * rhs
    ref = sla.spsolve_triangular((T + sp.identity(n)).tocsr(), b, lower=not upper)
    assert st[0] == 0
    assert np.linalg.norm(t - ref) <= TOL[fp32] * np.linalg.norm(ref)
    return st


def _random_lower(n, per_row, size, seed):
    rng = np.random.default_rng(seed)
    T = sp.lil_matrix((n, n))
    for i in range(1, n):
        k = rng.integers(0, min(i, per_row) + 1)
        for j in rng.choice(i, k, replace=False):
            T[i, j] = size * rng.uniform(-1, 1)
    T = T.tocsr()
    T.sort_indices()
    return T


@pytest.mark.parametrize("idim,coef,lev", [(16, ISO, 0), (20, ANISO, 0), (28, ISO, 1)])
@pytest.mark.parametrize("ncols,fp32", [(1, 0), (1, 1), (2, 0), (8, 1), (32, 0)])
def test_ilu_factors(mld, orc, idim, coef, lev, ncols, fp32):
    op = orc.Prec(oracle_params(orc, "BJAC", mcs=50))
    op.build(orc.gen_pde3d(idim, 1, coef))
    d = op.level_vec(lev, "d")
    for which, upper in (("L", 0), ("U", 1)):
        m = op.level_csr(lev, which)
        T = sp.csr_matrix((m.val, m.ja, m.irp), shape=(m.nrows, m.nrows))
        for Tm, up in ((T, upper), (sp.csr_matrix(T.T), 1 - upper)):
            Tm.sort_indices()
            st = _check(mld, Tm, up, d, ncols, 20000, 0, 0.0, fp32)
            assert 1 <= st[2] < st[1]  # levels were joined


@pytest.mark.parametrize("budget", [1, 300, 10 ** 9])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257])
def test_sizes_and_budgets(mld, n, budget):
    T = _random_lower(n, 4, 0.3, n)
    st = _check(mld, T, 0, None, budget=budget)
    _check(mld, sp.csr_matrix(T.T), 1, None, budget=budget)
    assert budget != 1 or st[2] == st[1]
    _check(mld, T, 0, None, budget=budget, row=3)


def test_chain_and_growth(mld):
    """A bidiagonal factor: one row per level.  With entries of size 3 the
    inverse grows as 3^k, so groups stay a few levels deep; with 0.5 one group
    holds the whole chain."""
    n = 60
    small = sp.diags([np.full(n - 1, 0.5)], [-1]).tocsr()
    assert _check(mld, small, 0, None, budget=10 ** 9, row=10 ** 6)[2] == 1
    big = sp.diags([np.full(n - 1, 3.0)], [-1]).tocsr()
    st = _check(mld, big, 0, None, budget=10 ** 9, row=10 ** 6)
    assert n / 4 <= st[2] < n  # 1 + 3 + 9 + 27 = 40 <= 64 < 121: four levels a group


def test_no_entries(mld):
    st = _check(mld, sp.csr_matrix((70, 70)), 0, np.linspace(1, 2, 70))
    assert st[1] == 1 and st[2] == 1
