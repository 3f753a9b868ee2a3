"""GPU: the dense inverses of small levels (ILU(0) and Gauss-Seidel) and the
solves that they are timed against."""
import numpy as np
import pytest

from conftest import ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu

TOL = {"PREC_FP64": 1e-12, "PREC_FP32": 2e-5}  # the repository's parity bars


@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
def test_not_formed_without_ell_plans(mld, orc, monkeypatch, capfd, smoother):
    """An inverse is formed with the 32-column ELL solves: where these are
    missing it is neither timed nor said to be kept."""
    a = orc.gen_pde3d(14, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=20))
    op.build(a)
    assert op.nlev >= 3  # a level between the finest and the coarsest
    x = np.random.default_rng(1).uniform(-1, 1, a.nrows)
    ref = op.apply(x)
    monkeypatch.setenv("MLDG_VERBOSE", "1")
    monkeypatch.setenv("MLDG_DENSE_INV", "1")
    for env in (None, "MLDG_NO_ELL"):
        if env:
            monkeypatch.setenv(env, "1")
        capfd.readouterr()
        h = upload_oracle_hierarchy(mld, orc, op)
        said = "inverse n=" in capfd.readouterr().err
        assert said == (env is None)
        y = h.apply(x)
        assert np.linalg.norm(y - ref) <= TOL["PREC_FP64"] * np.linalg.norm(ref)
