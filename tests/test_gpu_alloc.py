"""GPU: a device allocation that fails leaves nothing half made.

mldg_test_set_alloc_failure makes one allocation of the library fail on the
host, each in turn; the call returns MLDG_ERR_ALLOC, and the same call repeated
on the same handle is right (a plan or a buffer that only counted as made would
be a null pointer in its kernel)."""
import ctypes as C

import numpy as np
import pytest

from conftest import ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu

ERR_ALLOC = 4010
TOL = 1e-12  # the repository's parity bar in FP64


def _fail_after(mld, n):
    f = mld.lib().mldg_test_set_alloc_failure
    f.argtypes = [C.c_int]
    assert f(n) == 0


@pytest.fixture(autouse=True)
def _none_fails(mld):
    yield
    _fail_after(mld, -1)


def _each_allocation(mld, call, check, prepare=lambda: None):
    """Runs `call` with its first, second, ... allocation failing until none is
    left to fail; after each failure the call is repeated."""
    n = 0
    while True:
        prepare()
        _fail_after(mld, n)
        try:
            call()
            failed = False
        except mld.MldError as e:
            assert e.code == ERR_ALLOC, e.code
            failed = True
        finally:
            _fail_after(mld, -1)
        if not failed:
            return n
        check(call())
        n += 1
        assert n < 500


def _close(y, ref):
    assert max(np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in zip(y, ref)) <= TOL


@pytest.mark.parametrize("smoother,trans,width", [("BJAC", "N", 8), ("BJAC", "T", 3), ("BJAC", "N", 31),
                                                  ("FBGS", "N", 8), ("JACOBI", "N", 5)])
def test_block(mld, orc, smoother, trans, width):
    """The plans and buffers of a block's width, made at its first use: on a new
    handle, and on one whose graph of a narrower block is captured."""
    a = orc.gen_pde3d(9, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=100))
    op.build(a)
    X = np.random.default_rng(width).uniform(-1, 1, (width, a.nrows))
    ref = [op.apply(x, trans) for x in X]
    state = {}

    def new(narrow):
        state["h"] = upload_oracle_hierarchy(mld, orc, op, autotune=False)
        if narrow:
            _close(state["h"].apply_block(X[:2].copy(), trans=trans), ref[:2])

    for narrow in (False, True):
        n = _each_allocation(mld, lambda: state["h"].apply_block(X.copy(), trans=trans), lambda y: _close(y, ref),
                             lambda: new(narrow))
        assert n >= 4
        # a failure, then the narrower block whose graph was captured before it
        new(True)
        _fail_after(mld, n // 2)
        with pytest.raises(mld.MldError):
            state["h"].apply_block(X.copy(), trans=trans)
        _fail_after(mld, -1)
        _close(state["h"].apply_block(X[:2].copy(), trans=trans), ref[:2])


def test_krylov_vectors(mld, orc):
    """The vectors of a block solve: grown for a wider block, the allocation
    fails, and a narrower solve follows on the same handle; and the vectors of
    the K-cycle."""
    a = orc.gen_pde3d(9, 1, ISO)
    op = orc.Prec(oracle_params(orc, "BJAC", mcs=100))
    op.build(a)
    B = np.array([orc.spmv(a, np.full(a.nrows, 1.0 + k)) for k in range(9)])
    ones = np.array([np.full(a.nrows, 1.0 + k) for k in range(9)])
    state = {}

    def solve(k):
        return state["h"].krylov_multi("FCG", B[:k].copy(), eps=1e-12)[0]

    def new():
        state["h"] = upload_oracle_hierarchy(mld, orc, op, autotune=False)
        state["h"].apply_block(np.zeros((16, a.nrows)))  # the block's own buffers are there
        assert np.max(np.abs(solve(2) / ones[:2] - 1)) < 1e-9

    n = 0
    while True:
        new()
        _fail_after(mld, n)
        try:
            solve(9)
            break
        except mld.MldError as e:
            assert e.code == ERR_ALLOC
        finally:
            _fail_after(mld, -1)
        assert np.max(np.abs(solve(2) / ones[:2] - 1)) < 1e-9  # the narrower solve first
        assert np.max(np.abs(solve(9) / ones - 1)) < 1e-9
        n += 1
    assert n >= 4
    x = np.random.default_rng(3).uniform(-1, 1, a.nrows)
    h = upload_oracle_hierarchy(mld, orc, op, autotune=False)
    h.set_cycle(2)
    ref = h.apply(x)

    def kcycle():
        state["h"] = upload_oracle_hierarchy(mld, orc, op, autotune=False)
        state["h"].set_cycle(2)

    n = _each_allocation(mld, lambda: [state["h"].apply(x)], lambda y: _close(y, [ref]), kcycle)
    assert n >= 4


@pytest.mark.parametrize("smoother", ["BJAC", "FBGS"])
def test_finalize(mld, orc, smoother):
    """A hierarchy finalized again whose device data do not fit: the handle is
    not built (it answers with an error, as before its first finalize), and
    finalizing it once more mends it."""
    a = orc.gen_pde3d(9, 1, ISO)
    op = orc.Prec(oracle_params(orc, smoother, mcs=100))
    op.build(a)
    h = upload_oracle_hierarchy(mld, orc, op, autotune=False)
    x = np.random.default_rng(5).uniform(-1, 1, a.nrows)
    ref = op.apply(x)
    for n in (0, 1, 7, 20, 33, 40):
        _fail_after(mld, n)
        with pytest.raises(mld.MldError) as e:
            h.finalize(op.nlev)
        assert e.value.code == ERR_ALLOC
        _fail_after(mld, -1)
        with pytest.raises(mld.MldError):
            h.apply(x)
        h.finalize(op.nlev)
        _close([h.apply(x)], [ref])
