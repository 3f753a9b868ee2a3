"""The work that this framework's users have it do, as cases that can be timed.

A case is one call through the Python view of the library (``MldPrec``,
``krylov``, ``krylov_batch``): one multilevel preconditioner application, a
block of them, a whole Krylov solve, or the adjoint gradient.  ``prepare``
builds the matrix and the preconditioner (hierarchy, smoother data, upload) as
a user's program does once per matrix, and draws from the seed the residual to
apply it to, or the right-hand side of a smooth known solution; ``run`` is the
call.

The problems are the repository's own: the 7-point convection-diffusion
problem (isotropic, or with 0.01 u_zz) on idim^3 cells and
-div(kappa grad u) with a log-normal kappa, with the settings of the tests and
of the benchmark (decoupled smoothed aggregation, theta 0.01, coarsening to
2,000 rows, coarsest level 4 sweeps of block-Jacobi ILU(0)).

The solves with an FP32 V-cycle run to 1e-12: the V-cycle's own rounding then
no longer shows in the FP64 solution.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = "cuda:0"
S3 = 1.0 / math.sqrt(3.0)
COEF = {"iso": (1.0, 1.0, 1.0, S3, S3, S3, 0.0), "aniso": (1.0, 1.0, 0.01, S3, S3, S3, 0.0)}


def _package():
    name = "mld2p4_2_b200"
    if name not in sys.modules:
        d = os.path.join(ROOT, "mld2p4-2_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def listed():
    return [
        # the smallest hierarchy (two levels, the 4,096 rows of the recorded
        # fixture): an inner preconditioner of small blocks; latency and
        # launches are all it costs
        {"name": "apply_bjac_16", "kind": "apply", "smoother": "BJAC", "coef": "iso", "idim": 16, "trans": "N"},
        # the transposed application of an adjoint code, an odd size, the
        # anisotropic problem's wide coarse rows
        {"name": "apply_jacobi_t_61", "kind": "apply", "smoother": "JACOBI", "coef": "aniso", "idim": 61, "trans": "T"},
        # an ordinary drop-in call of prec%apply with the ILU(0) smoother
        {"name": "apply_bjac_101", "kind": "apply", "smoother": "BJAC", "coef": "iso", "idim": 101, "trans": "N"},
        # a large application: more than a million rows streamed from memory
        {"name": "apply_jacobi_104", "kind": "apply", "smoother": "JACOBI", "coef": "iso", "idim": 104, "trans": "N"},
        # a few right-hand sides at once (a multivector of odd width)
        {"name": "block_bjac_5x45", "kind": "block", "smoother": "BJAC", "coef": "iso", "idim": 45, "nrhs": 5},
        # the first benchmark configuration: CG to 1e-9
        {"name": "cg_bjac_40", "kind": "solve", "smoother": "BJAC", "coef": "iso", "idim": 40, "precision": "FP64",
         "method": "CG", "eps": 1e-9},
        # the reference's default preconditioner (hybrid Gauss-Seidel V-cycle)
        {"name": "fcg_fbgs_50", "kind": "solve", "smoother": "FBGS", "coef": "iso", "idim": 50, "precision": "FP64",
         "method": "FCG", "eps": 1e-10},
        # the plain FP64 solve of the anisotropic problem
        {"name": "fcg_jacobi_80", "kind": "solve", "smoother": "JACOBI", "coef": "aniso", "idim": 80,
         "precision": "FP64", "method": "FCG", "eps": 1e-10},
        # the benchmark's headline form, at 1.4 million rows: FP16 operator
        # values, FP32 V-cycle
        {"name": "fcg_jacobi_h16_112", "kind": "solve", "smoother": "JACOBI", "coef": "aniso", "idim": 112,
         "precision": "FP32_H16", "method": "FCG", "eps": 1e-12},
        # differentiation: forward solve, adjoint solve, gradient scatter
        {"name": "gradient_kappa_64", "kind": "gradient", "idim": 64},
        # 32 right-hand sides advanced together
        {"name": "multi_bjac_32x64", "kind": "multi", "smoother": "BJAC", "coef": "iso", "idim": 64, "nrhs": 32},
        # independent systems of mixed sizes in one call
        {"name": "batch_8x24_44", "kind": "batch", "smoother": "BJAC", "coef": "iso", "nsys": 8, "lo": 24, "hi": 44},
    ]


def _size(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "block", "solve", "solve", "solve", "gradient", "multi", "batch"))
    coef = rng.choice(("iso", "aniso"))
    if kind == "apply":
        return {"kind": kind, "smoother": rng.choice(("BJAC", "JACOBI")), "coef": coef, "idim": _size(rng, 16, 96),
                "trans": rng.choice("NNT")}
    if kind == "block":
        return {"kind": kind, "smoother": rng.choice(("BJAC", "JACOBI")), "coef": coef, "idim": _size(rng, 16, 64),
                "nrhs": _size(rng, 2, 32)}
    if kind == "solve":
        smoother = rng.choice(("BJAC", "JACOBI", "JACOBI", "FBGS"))
        # the ILU(0) V-cycle is used on the isotropic problem (it is not
        # symmetric, and CG needs it nearly so)
        prec = rng.choice(("FP64", "FP32", "FP32_P16", "FP32_H16"))
        return {"kind": kind, "smoother": smoother, "coef": coef if smoother == "JACOBI" else "iso",
                "idim": _size(rng, 20, 80 if smoother == "JACOBI" else 64), "precision": prec,
                "method": "FCG" if prec != "FP64" else rng.choice(("CG", "FCG")),
                "eps": 1e-10 if prec == "FP64" else 1e-12}
    if kind == "gradient":
        return {"kind": kind, "idim": _size(rng, 16, 72)}
    if kind == "multi":
        return {"kind": kind, "smoother": rng.choice(("BJAC", "JACOBI")), "coef": "iso", "idim": _size(rng, 20, 64),
                "nrhs": _size(rng, 2, 32)}
    lo = _size(rng, 20, 32)
    return {"kind": kind, "smoother": rng.choice(("BJAC", "JACOBI")), "coef": "iso", "nsys": rng.randint(3, 8),
            "lo": lo, "hi": lo + rng.randint(4, 12)}


def _configured(smoother, precision):
    p = _package().MldPrec(device=0)
    p.init("ML")
    p.set("SMOOTHER_TYPE", smoother)
    if smoother == "JACOBI":
        p.set("SMOOTHER_SWEEPS", 2)
        p.set("SMOOTHER_DAMPING", 0.8)
    else:
        p.set("SMOOTHER_SWEEPS", 1)
        if smoother == "BJAC":
            p.set("SUB_SOLVE", "ILU")
    p.set("COARSE_SOLVE", "BJAC")
    p.set("COARSE_SUBSOLVE", "ILU")
    p.set("COARSE_SWEEPS", 4)
    p.set("MIN_COARSE_SIZE", 2000)
    p.set("AGGR_THRESH", 0.01)
    p.set("PRECISION", precision)
    return p


def _built(a, smoother, precision="FP64"):
    p = _configured(smoother, precision)
    p.build(a)
    return p


def _uniform(seed, *shape):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g) * 2.0 - 1.0


def _smooth(seed, idim, *count):
    # solutions of a few low modes, zero on the boundary
    rng = np.random.default_rng(seed)
    t = torch.arange(1, idim + 1, dtype=torch.float64, device=DEV) * (math.pi / (idim + 1))
    out = []
    for _ in range(math.prod(count)):
        x = 0.0
        for c, (i, j, k) in zip(rng.standard_normal(4), rng.integers(1, 6, (4, 3))):
            x = x + c * torch.sin(i * t)[:, None, None] * torch.sin(j * t)[:, None] * torch.sin(k * t)
        out.append(x.reshape(-1))
    return torch.stack(out).reshape(*count, -1)


def _sparse(m):
    return torch.sparse_csr_tensor(torch.from_numpy(m.irp), torch.from_numpy(m.ja), torch.from_numpy(m.val),
                                   size=(m.nrows, m.ncols), device=DEV)


def _matrix(case, seed):
    mld = _package()
    if case["kind"] == "gradient":
        return mld.gen_kappa3d(case["idim"], _kappa(case, seed))
    return mld.gen_pde3d(case["idim"], 1, COEF[case["coef"]])


def _kappa(case, seed):
    # log-normal with a correlation length of some cells: white noise smoothed
    # by neighbour averages (periodic), standardised
    d = case["idim"]
    w = np.random.default_rng(seed).standard_normal((d, d, d))
    for _ in range(4):
        for ax in range(3):
            w = 0.5 * w + 0.25 * (np.roll(w, 1, ax) + np.roll(w, -1, ax))
    return np.exp((w - w.mean()) / w.std()).ravel()


def _dims(case):
    # the sizes of a batch: spread over the range, the same for every seed
    # (one program's systems), so that the work of a case is one number
    return [int(v) for v in np.random.default_rng(1).integers(case["lo"], case["hi"] + 1, case["nsys"])]


def prepare(case, seed):
    kind = case["kind"]
    mld = _package()
    if kind == "batch":
        precs, bs = [], []
        for i, d in enumerate(_dims(case)):
            a = mld.gen_pde3d(d, 1, COEF[case["coef"]])
            precs.append(_built(a, case["smoother"], "FP32"))
            bs.append(_sparse(a) @ _smooth(seed * 64 + i, d))
        return {"case": case, "precs": precs, "bs": bs}
    a = _matrix(case, seed)
    n = a.nrows
    s = {"case": case, "a": a, "n": n}
    if kind == "apply":
        s |= {"p": _built(a, case["smoother"]), "x": _uniform(seed, n), "y": torch.zeros(n, dtype=torch.float64, device=DEV)}
    elif kind == "block":
        s |= {"p": _built(a, case["smoother"]), "x": _uniform(seed, case["nrhs"], n)}
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "solve":
        s |= {"p": _built(a, case["smoother"], case["precision"]), "b": _sparse(a) @ _smooth(seed, case["idim"])}
    elif kind == "multi":
        s["p"] = _built(a, case["smoother"], "FP32")
        s["b"] = (_sparse(a) @ _smooth(seed, case["idim"], case["nrhs"]).T).T.contiguous()
    else:
        m = _sparse(a)  # symmetric
        s |= {"p": _built(a, "JACOBI"), "b": m @ _smooth(seed, case["idim"]),
              "g": m @ _smooth(seed + 1, case["idim"]),
              "kappa": torch.from_numpy(_kappa(case, seed)).to(DEV)}
    return s


def _zeros(like):
    # the library runs on streams of its own: a zero guess has to be there
    x = torch.zeros_like(like)
    torch.cuda.current_stream().synchronize()
    return x


def run(s):
    c = s["case"]
    kind = c["kind"]
    mld = _package()
    if kind == "apply":
        return s["p"].apply(s["x"], s["y"], trans=c["trans"])
    if kind == "block":
        return s["p"].apply_block(s["x"], s["y"])
    if kind == "solve":
        x, _, _ = mld.krylov(c["method"], s["a"], s["p"], s["b"], _zeros(s["b"]), eps=c["eps"], itmax=1000,
                             use_prec_matrix=True)
        return x
    if kind == "multi":
        x, _, _ = s["p"].krylov_multi("FCG", s["b"], _zeros(s["b"]), eps=1e-12, itmax=500)
        return x
    if kind == "batch":
        xs = [torch.zeros_like(b) for b in s["bs"]]
        torch.cuda.current_stream().synchronize()
        return mld.krylov_batch("FCG", s["precs"], s["bs"], xs, eps=1e-12, itmax=500)[0]
    x, _, _ = mld.krylov("FCG", s["a"], s["p"], s["b"], _zeros(s["b"]), eps=1e-12, itmax=500, use_prec_matrix=True)
    lam, _, _ = s["p"].adjoint(s["g"], _zeros(s["g"]), eps=1e-12, itmax=500)
    grad = torch.empty_like(x)
    s["p"].kappa_grad(c["idim"], s["kappa"], x, lam, grad)
    return x, lam, grad


# entries of the hierarchy per entry of the finest matrix, all levels together
# (A; P), and rows per finest row, as the aggregation leaves them
_GROWTH = {"iso": (1.56, 0.62, 1.13), "aniso": (2.4, 1.06, 1.19)}


def work(case):
    """Each operator of the hierarchy and of its smoother read once per V-cycle
    (CSR: a value and a 4-byte column per entry, no more for R = P^T), each
    finest-level vector once; a solve does that in every iteration, with the
    iteration counts that these problems take."""
    kind = case["kind"]
    if kind == "batch":
        each = [work({"kind": "solve", "smoother": case["smoother"], "coef": case["coef"], "idim": d,
                      "precision": "FP32", "method": "FCG", "eps": 1e-12}) for d in _dims(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    d = case["idim"]
    n = d ** 3
    nnz = 7 * n - 6 * d * d
    ca, cp, cr = _GROWTH[case.get("coef", "iso")]
    smoother = case.get("smoother", "JACOBI")
    precision = {"solve": case.get("precision"), "multi": "FP32"}.get(kind, "FP64")
    size = {"FP64": 12, "FP32_H16": 6}.get(precision, 8)
    entries = nnz * (ca * (2 if smoother == "BJAC" else 1) + cp)  # the ILU(0) factors beside A
    vec = 8 if precision == "FP64" else 4
    cycle_bytes = entries * size + vec * n * cr
    # multiply-adds: 2 smoothings and 2 residuals a level, P and R
    cycle_flops = 2.0 * nnz * (4 * ca + 2 * cp)
    nrhs = case.get("nrhs", 1)
    if kind in ("apply", "block"):
        return {"bytes": cycle_bytes + 16.0 * n * nrhs, "flops": cycle_flops * nrhs}
    digits = -math.log10(case.get("eps", 1e-12))
    if case.get("coef") == "aniso":
        its = digits * 2.0
    else:
        its = digits * (1.5 if smoother == "JACOBI" else 1.1) * (d / 50.0) ** 0.3
    # q = A d, and x, r, d, q of the iteration read and written
    its *= 2 if kind == "gradient" else 1
    return {"bytes": its * (cycle_bytes + 12.0 * nnz + 64.0 * n * nrhs),
            "flops": its * nrhs * (cycle_flops + 2.0 * nnz + 10.0 * n)}


class _Cycle:
    """The V-cycle in plain 64-bit torch on the hierarchy as it is uploaded
    (the levels' A, P, L, U, d: the input of an application)."""

    def __init__(self, p, smoother):
        self.smoother = smoother
        get = lambda l, w: p.level_csr(l, w)  # noqa: E731
        self.levels = []
        for l in range(p.nlev):
            ilu = smoother == "BJAC" or l == p.nlev - 1
            lev = {"A": _sparse(get(l, "A")), "ilu": ilu, "d": torch.from_numpy(p.level_vec(l, "d")).to(DEV)[:, None]}
            if l:
                lev["P"], lev["R"] = _sparse(get(l, "P")), _sparse(get(l, "R"))
            lev |= {k: get(l, k) for k in (("L", "U") if ilu else ())}
            if not ilu:
                lev["ND"] = _sparse(get(l, "ND"))
            self.levels.append(lev)

    @staticmethod
    def _unit(m, upper, trans, b):
        one = np.arange(m.nrows + 1, dtype=np.int32)
        rows = np.repeat(one[:-1], np.diff(m.irp))
        i, j = (m.ja, rows) if trans else (rows, m.ja)
        i, j = np.concatenate((i, one[:-1])), np.concatenate((j, one[:-1]))
        v = np.concatenate((m.val, np.ones(m.nrows)))
        t = torch.sparse_coo_tensor(torch.from_numpy(np.stack((i, j)).astype(np.int64)), torch.from_numpy(v),
                                    (m.nrows, m.nrows), device=DEV).coalesce().to_sparse_csr()
        return torch.triangular_solve(b, t, upper=upper != trans)[0]

    def _smooth(self, lev, x, trans):
        if lev["ilu"]:
            first, last = ("U", "L") if trans else ("L", "U")
            t = self._unit(lev[first], first == "U", trans, x)
            return self._unit(lev[last], last == "U", trans, lev["d"] * t)
        nd = lev["ND"].t() if trans else lev["ND"]
        y = 0.8 * lev["d"] * x
        return 0.2 * y + 0.8 * lev["d"] * (x - nd @ y)

    def __call__(self, x, trans, l=0):
        lev = self.levels[l]
        if l == len(self.levels) - 1:
            return self._smooth(lev, x, trans)
        nxt = self.levels[l + 1]
        a = lev["A"].t() if trans else lev["A"]
        y = self._smooth(lev, x, trans)
        y = y + nxt["P"] @ self(nxt["R"] @ (x - a @ y), trans, l + 1)
        return y + self._smooth(lev, x - a @ y, trans)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_smooth(seed * 64 + i, d) for i, d in enumerate(_dims(case))]
    n = case["idim"] ** 3
    if kind == "solve":
        return _smooth(seed, case["idim"])
    if kind == "multi":
        return _smooth(seed, case["idim"], case["nrhs"])
    if kind == "gradient":
        x, lam = _smooth(seed, case["idim"]), _smooth(seed + 1, case["idim"])
        return x, lam, _gradient(case["idim"], torch.from_numpy(_kappa(case, seed)).to(DEV), x, lam)
    p = _configured(case["smoother"], "FP64")
    p.hierarchy_build(_matrix(case, seed))
    p.smoothers_build_host()
    x = _uniform(seed, case["nrhs"], n).T if kind == "block" else _uniform(seed, n)[:, None]
    y = _Cycle(p, case["smoother"])(x.contiguous(), case.get("trans") == "T")
    return y.T.contiguous() if kind == "block" else y[:, 0].contiguous()


def _gradient(d, kappa, x, lam):
    """d(lam . A(kappa) x)/d kappa, negated, for harmonic-mean faces; a boundary
    face takes its own cell's kappa."""
    k, x, lam = (t.reshape(d, d, d) for t in (kappa, x, lam))
    g = torch.zeros_like(k)
    for ax in range(3):
        for step in (1, -1):
            ks, xs, ls = (torch.roll(t, step, ax) for t in (k, x, lam))
            face = 2 * ks ** 2 / (k + ks) ** 2 * (lam - ls) * (x - xs)
            edge = [slice(None)] * 3
            edge[ax] = 0 if step == 1 else d - 1
            face[tuple(edge)] = (lam * x)[tuple(edge)]
            g += face
    return (-(d + 1) ** 2 * g).reshape(-1)
