"""GPU: the grouped solves of blocks of 16 and 32 columns on a level of wide
rows, the dense K-column products in their place, the level-by-level solves with
the grouped ones turned off, and the recovery of a block's and of Gauss-Seidel's
grouped solves after a wait that ran out."""
import ctypes as C

import numpy as np
import pytest

from conftest import ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu

TOL = {"PREC_FP64": 1e-12, "PREC_FP32": 2e-5}  # the repository's parity bars


def _problem(orc, smoother, idim, mcs, count):
    a = orc.gen_pde3d(idim, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=mcs))
    op.build(a)
    assert op.nlev >= 3
    X = np.random.default_rng(idim).uniform(-1, 1, (count, a.nrows))
    trans = ("N", "T") if smoother == "BJAC" else ("N",)
    return op, X, {t: [op.apply(x, t) for x in X] for t in trans}


def _err(Y, ref):
    return max(np.linalg.norm(y - r) / np.linalg.norm(r) for y, r in zip(Y, ref))


@pytest.mark.parametrize("prec", ["PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
@pytest.mark.parametrize("env", ["MLDG_NO_DENSE_INV", "MLDG_DENSE_INV", "MLDG_NO_GRP"])
def test_widths(mld, orc, monkeypatch, capfd, env, smoother, prec):
    op, X, ref = _problem(orc, smoother, 19, 60, 31)
    monkeypatch.setenv(env, "1")
    if env == "MLDG_NO_GRP":
        monkeypatch.setenv("MLDG_NO_DENSE_INV", "1")
    monkeypatch.setenv("MLDG_VERBOSE", "1")
    h = upload_oracle_hierarchy(mld, orc, op, precision=getattr(mld, prec))
    for w in (31, 9, 3):
        for t, r in ref.items():
            assert _err(h.apply_block(X[:w].copy(), trans=t), r[:w]) <= TOL[prec], (w, t)
            assert _err([h.apply(X[0], trans=t)], r) <= TOL[prec], t
    said = capfd.readouterr().err
    grouped = {K: f"grp K={K} " in said for K in (1, 4, 16, 32)}
    if env == "MLDG_NO_DENSE_INV":
        assert all(grouped.values()), grouped
    elif env == "MLDG_NO_GRP":
        assert not any(grouped.values()), grouped
    else:
        assert "-> dense" in said and "-> solves" not in said


@pytest.mark.parametrize("idim,mcs", [(7, 12), (10, 20), (16, 30)])
def test_dense_products(mld, orc, monkeypatch, idim, mcs):
    """The dense inverses of small and odd sizes, every width."""
    monkeypatch.setenv("MLDG_DENSE_INV", "1")
    op, X, ref = _problem(orc, "BJAC", idim, mcs, 17)
    for prec in TOL:
        h = upload_oracle_hierarchy(mld, orc, op, precision=getattr(mld, prec))
        for w in (2, 3, 8, 13, 17):
            for t, r in ref.items():
                assert _err(h.apply_block(X[:w].copy(), trans=t), r[:w]) <= TOL[prec], (prec, w, t)


@pytest.mark.parametrize("smoother,width", [("BJAC", 1), ("BJAC", 5), ("BJAC", 31), ("FBGS", 1), ("FBGS", 5)])
def test_recovery_after_a_wait_ran_out(mld, orc, monkeypatch, smoother, width):
    """With no polls a wait gives up at once, the kernel ends and the call returns
    an error; with the limit back the same handle is right at every width."""
    monkeypatch.setenv("MLDG_NO_DENSE_INV", "1")
    op, X, ref = _problem(orc, smoother, 30, 200, 5)
    X = np.resize(X, (width, X.shape[1])) if width > 5 else X[:width]
    ref = {t: (r * 7)[:width] for t, r in ref.items()}
    h = upload_oracle_hierarchy(mld, orc, op)

    def call(t):
        return h.apply_block(X.copy(), trans=t) if width > 1 else [h.apply(X[0], trans=t)]

    def check():
        for t, r in ref.items():
            assert _err(call(t), r) <= TOL["PREC_FP64"], t
            assert _err([h.apply(X[0], trans=t)], r) <= TOL["PREC_FP64"], t

    check()
    f = mld.lib().mldg_test_set_spin_limit
    f.argtypes = [C.c_int, C.c_int]
    codes = []
    for t in ref:
        assert f(0, 0) == 0
        try:
            for _ in range(3):
                try:
                    call(t)
                    codes.append(0)
                except mld.MldError as e:
                    codes.append(e.code)
        finally:
            assert f(0, -1) == 0
        check()
    assert mld.ERR_TIMEOUT in codes and set(codes) <= {0, mld.ERR_TIMEOUT}, codes
