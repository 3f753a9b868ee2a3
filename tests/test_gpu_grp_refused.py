"""GPU: grouped plans that are refused (MLDG_GRP_MB bounds a level's plans): the
level takes its other solves, at finalize and for a block's width later on."""
import numpy as np
import pytest

from conftest import ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu

TOL = {"PREC_FP64": 1e-12, "PREC_FP32": 2e-5}  # the repository's parity bars


def _rel(y, ref):
    return np.linalg.norm(y - ref) / np.linalg.norm(ref)


def _problem(orc, smoother, trans="N"):
    a = orc.gen_pde3d(16, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=100))
    op.build(a)
    X = np.random.default_rng(4).uniform(-1, 1, (5, a.nrows))
    return op, X, {t: [op.apply(x, t) for x in X] for t in ("N", trans)}


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
def test_at_finalize(mld, orc, monkeypatch, capfd, smoother, prec):
    op, X, ref = _problem(orc, smoother, "T" if smoother == "BJAC" else "N")
    monkeypatch.setenv("MLDG_VERBOSE", "1")
    monkeypatch.setenv("MLDG_GRP_MB", "0")
    h = upload_oracle_hierarchy(mld, orc, op, precision=getattr(mld, prec))
    said = capfd.readouterr().err
    assert "mldg: grp K=" not in said
    # an ILU(0) level of this size has its window plans again
    assert ("level 0 win0" in said) == (smoother == "BJAC")
    for trans, r in ref.items():
        assert max(_rel(h.apply(x, trans=trans), y) for x, y in zip(X, r)) <= TOL[prec]
    assert max(_rel(y, r) for y, r in zip(h.apply_block(X.copy()), ref["N"])) <= TOL[prec]


@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
def test_for_a_width(mld, orc, monkeypatch, smoother):
    """One column and two are grouped and their graphs captured; then the plans
    of a wider block, and of the transposed block, are refused."""
    trans = "T" if smoother == "BJAC" else "N"
    op, X, ref = _problem(orc, smoother, trans)
    h = upload_oracle_hierarchy(mld, orc, op)
    tol = TOL["PREC_FP64"]

    def check(t, w):
        assert max(_rel(y, r) for y, r in zip(h.apply_block(X[:w].copy(), trans=t), ref[t])) <= tol, (t, w)

    check("N", 5)
    check("N", 2)
    monkeypatch.setenv("MLDG_GRP_MB", "0")
    check(trans, 2)  # transposed: refused with the other direction's graph captured
    check("N", 2)
    check("N", 3)
    check("N", 5)  # planned before
    check(trans, 5)
    X[:] = X[::-1].copy()
    for t in ref:
        ref[t].reverse()
    check("N", 5)
    assert _rel(h.apply(X[0]), ref["N"][0]) <= tol
