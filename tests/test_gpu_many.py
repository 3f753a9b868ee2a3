"""GPU: many systems at once, in a batch of more systems than the SMs have room
for, and on threads of their own: however many blocks a grouped solve is left
with, the results equal those of the systems one by one bit for bit."""
import threading

import numpy as np
import pytest

from conftest import ANISO, ISO, oracle_params, upload_oracle_hierarchy

pytestmark = pytest.mark.gpu


def _systems(mld, orc, dims, precision):
    made = {}
    out = []
    for k, idim in enumerate(dims):
        key = (idim, k % 2)
        if key not in made:
            a = orc.gen_pde3d(idim, 1, ANISO if k % 2 else ISO)
            op = orc.Prec(oracle_params(orc, "BJAC", mcs=100))
            op.build(a)
            made[key] = a, op
        a, op = made[key]
        out.append((a, upload_oracle_hierarchy(mld, orc, op, precision=precision, autotune=False),
                    np.random.default_rng(k).uniform(-1, 1, a.nrows)))
    return out


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_of_many(mld, orc, precision):
    sy = _systems(mld, orc, [6 + k % 7 for k in range(59)] + [30], precision)
    hs, bs = [h for _, h, _ in sy], [b for _, _, b in sy]
    xs, its, rel, _ = mld.krylov_batch("FCG", hs, bs, eps=1e-10, itmax=300)
    for (a, h, b), x, it, r in zip(sy, xs, its, rel):
        x1, it1, r1 = h.krylov("FCG", b.copy(), eps=1e-10, itmax=300)
        assert it == it1 and r == r1 and r <= 1e-10
        assert np.array_equal(x, x1)
        assert np.linalg.norm(b - orc.spmv(a, x)) <= 2e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("precision", [0, 1])
def test_handles_on_threads(mld, orc, precision):
    """Applications, transposed ones and blocks, on ten handles at once."""
    sy = _systems(mld, orc, [30, 8, 24, 12, 31, 17, 28, 9, 33, 21], precision)
    X = [np.random.default_rng(k).uniform(-1, 1, (3, a.nrows)) for k, (a, _, _) in enumerate(sy)]

    def calls(h, x):
        return [h.apply(x[0]), h.apply(x[1], trans="T"), h.apply_block(x.copy()), h.krylov("FCG", x[2].copy(), eps=1e-8)[0]]

    ref = [calls(h, x) for (_, h, _), x in zip(sy, X)]
    bad = []

    def work(h, x, r):
        try:
            for _ in range(15):
                if not all(np.array_equal(y, z) for y, z in zip(calls(h, x), r)):
                    bad.append("differs")
        except Exception as e:  # noqa: BLE001 (a thread's failure is reported below)
            bad.append(repr(e))

    th = [threading.Thread(target=work, args=(h, x, r)) for (_, h, _), x, r in zip(sy, X, ref)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
    assert all(np.array_equal(y, z) for (_, h, _), x, r in zip(sy, X, ref) for y, z in zip(calls(h, x), r))
