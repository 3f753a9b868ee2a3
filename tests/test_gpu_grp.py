"""GPU: the grouped triangular solves (k_trsv_grp) and the dense K-column
products (k_gemm_m_rows, k_gemm_m_cols) against the oracle, at the edges of
their ranges: levels of a few rows up to several groups, the transposed pair,
Gauss-Seidel's single solves, the column widths 1, 2, 4, 8 of one task, the
wider ones of the dense products, and repeated applications (a solve resets
what the next ones need).  Tolerances: the repository's parity bars, 1e-12 in
FP64 and 2e-5 with an FP32 V-cycle."""
import numpy as np
import pytest

from conftest import ANISO, ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu

TOL = {"PREC_FP64": 1e-12, "PREC_FP32": 2e-5}


def _rel(y, ref):
    return np.linalg.norm(y - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("idim,coef,mcs", [(3, ISO, 5), (13, ISO, 40), (21, ANISO, 30), (33, ISO, 60)])
def test_ilu_pairs(mld, orc, idim, coef, mcs, prec):
    a = orc.gen_pde3d(idim, 1, coef)
    op = orc.Prec(oracle_params(orc, "BJAC", mcs=mcs))
    op.build(a)
    h = upload_oracle_hierarchy(mld, orc, op, precision=getattr(mld, prec))
    rng = np.random.default_rng(idim)
    for k in range(3):
        x = rng.uniform(-1, 1, a.nrows)
        for trans in ("N", "T"):
            assert _rel(h.apply(x, trans=trans), op.apply(x, trans)) <= TOL[prec], (k, trans)


@pytest.mark.parametrize("nrhs", [2, 3, 7, 9, 31])
@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
def test_column_widths(mld, orc, smoother, nrhs):
    """K = 2, 4, 8, 16, 32: a wide block and a narrow one on the same handle."""
    a = orc.gen_pde3d(18, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=150))
    op.build(a)
    h = upload_oracle_hierarchy(mld, orc, op)
    X = np.random.default_rng(nrhs).uniform(-1, 1, (nrhs, a.nrows))
    ref = [op.apply(x) for x in X]
    for w in (nrhs, 2, nrhs):
        Y = h.apply_block(X[:w].copy())
        assert max(_rel(y, r) for y, r in zip(Y, ref)) <= TOL["PREC_FP64"], w
