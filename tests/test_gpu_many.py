"""GPU: many systems at once: a batch of more systems than the SMs have room
for, each with a few blocks of its grouped solves, equals the systems one by
one bit for bit."""
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
