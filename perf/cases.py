"""Performance cases of the UA-AMG preconditioned Krylov library.

A case is one call sequence of a user's program, by ``kind``:

* ``assemble``  the P1 stiffness matrix on the Kuhn mesh from a device field;
* ``precond``   one preconditioner application z = B r on a kept hierarchy, for
  a program with a Krylov loop of its own;
* ``resolve``   a solve with a new right-hand side on a kept hierarchy (time
  steps with a fixed operator);
* ``step``      hierarchy setup and solve of a new matrix, on device arrays
  (a coefficient that changes from step to step);
* ``dropin``    linear_solver_dcsr_krylov_amg on host arrays, as a HAZmath
  program calls it;
* ``batch``     setup and solve of many independent systems in one call;
* ``bsr``       setup and solve of a block (BSR) system;
* ``learn``     one training gradient of the learned l1-Jacobi weights
  (inference, contraction loss by adjoint cycles, network backward).

``dim`` 3 is the P1 matrix on N^3 Kuhn cubes with a log-normal coefficient
((N - 1)^3 rows, 15-point pattern), ``dim`` 2 the P1 matrix of anisotropic
diffusion on m x m interior vertices (7-point pattern).  ``precision`` is the
drop-in's fp64 (exact heavy edge matching) or mixed (FP32 cycle, parallel
matching).  All solves run to a relative residual of 1e-8.
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

import hazmath_b200 as hz
from hazmath_b200 import learn

DEV = "cuda"
COUPLING = {2: [[2.0, 0.5], [0.5, 1.0]],
            3: [[3.0, 0.5, 0.2], [0.5, 2.0, 0.3], [0.2, 0.3, 1.0]]}


def listed():
    return [
        # the smallest call: one exact Gauss-Seidel V(1,1) on a 2D grid
        {"name": "precond_2d_63_gs", "kind": "precond", "dim": 2, "m": 63, "eps": 1.0,
         "theta": 0.0, "precision": "fp64", "smoother": "gs"},
        # time steps of a small 3D diffusion problem
        {"name": "resolve_3d_48_mixed", "kind": "resolve", "dim": 3, "N": 48, "sigma": 1.0,
         "precision": "mixed", "smoother": "l1"},
        # a small 3D problem whose coefficient changes: latency of setup and solve
        {"name": "step_3d_33_mixed", "kind": "step", "dim": 3, "N": 33, "sigma": 1.0,
         "precision": "mixed", "smoother": "l1"},
        # an ordinary 3D problem of a million unknowns, 99^3 rows
        {"name": "step_3d_100_mixed", "kind": "step", "dim": 3, "N": 100, "sigma": 1.5,
         "precision": "mixed", "smoother": "l1"},
        # the benchmark's 256^3 system, the largest
        {"name": "step_3d_256_mixed", "kind": "step", "dim": 3, "N": 256, "sigma": 1.5,
         "precision": "mixed", "smoother": "l1"},
        # 2D anisotropic diffusion of a million unknowns: many iterations
        {"name": "step_2d_1022_mixed", "kind": "step", "dim": 2, "m": 1022, "eps": 0.1,
         "theta": 0.7, "precision": "mixed", "smoother": "l1"},
        # the drop-in's arithmetic on the 128^3 benchmark system
        {"name": "step_3d_128_fp64", "kind": "step", "dim": 3, "N": 128, "sigma": 1.0,
         "precision": "fp64", "smoother": "l1"},
        # the drop-in call of a HAZmath program: host arrays, 2D, Gauss-Seidel
        {"name": "dropin_2d_255_gs", "kind": "dropin", "dim": 2, "m": 255, "eps": 1.0,
         "theta": 0.0, "smoother": "gs", "krylov": "cg"},
        # independent systems of 1k to 60k unknowns solved together
        {"name": "batch_48", "kind": "batch", "nsys": 48, "lo": 1000, "hi": 60000,
         "shapes": 11},
        # a block system with 3 x 3 blocks
        {"name": "bsr_3d_24", "kind": "bsr", "N": 24, "nb": 3},
        # a training gradient of the learned weights on a 2D problem
        {"name": "learn_2d_300", "kind": "learn", "dim": 2, "m": 300, "eps": 0.01,
         "theta": 0.7},
        # assembly of a 4 million row matrix
        {"name": "assemble_160", "kind": "assemble", "N": 160, "sigma": 1.0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def problem(c, m, N, dim=None):
        c["dim"] = dim or rng.choice([2, 3])
        if c["dim"] == 2:
            c.update(m=size(*m), eps=round(math.exp(rng.uniform(math.log(0.03), 0.0)), 4),
                     theta=round(rng.uniform(0.0, math.pi), 3))
        else:
            c.update(N=size(*N), sigma=round(rng.uniform(0.5, 1.5), 2))
        return c

    kind = rng.choice(["assemble", "precond", "resolve", "step", "step", "step", "dropin",
                       "batch", "bsr", "learn"])
    c = {"kind": kind}
    if kind == "assemble":
        c.update(N=size(17, 200), sigma=round(rng.uniform(0.5, 1.5), 2))
    elif kind == "precond":
        problem(c, (50, 300), (14, 60))
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["smoother"] = "l1" if c["precision"] == "mixed" else rng.choice(["gs", "l1"])
    elif kind == "resolve":
        problem(c, (100, 700), (17, 100))
        c.update(precision=rng.choice(["fp64", "mixed"]), smoother="l1")
    elif kind == "step":
        c["precision"] = rng.choice(["fp64", "mixed", "mixed"])
        problem(c, (63, 1100) if c["precision"] == "mixed" else (63, 300),
                (17, 220) if c["precision"] == "mixed" else (17, 110))
        c["smoother"] = "l1"
    elif kind == "dropin":
        problem(c, (50, 255), (14, 40))
        c.update(smoother=rng.choice(["gs", "l1"]), krylov=rng.choice(["cg", "fgmres"]))
    elif kind == "batch":
        c.update(nsys=size(8, 64), lo=1000, hi=size(8000, 60000), shapes=rng.randrange(1000))
    elif kind == "bsr":
        c.update(N=size(9, 24), nb=rng.choice([2, 3]))
    else:
        problem(c, (127, 400), (24, 56))
    return c


# ---------------------------------------------------------------------------
# problems, on the device
# ---------------------------------------------------------------------------
def _stencil(shape, coefs):
    """Sorted CSR over a grid (x fastest) from {offset (x first): value per
    grid point or one number}; neighbours outside the grid are dropped."""
    dims = len(shape)
    n = math.prod(shape)
    idx = torch.arange(n, device=DEV, dtype=torch.int32)
    xs, rest = [], idx
    for d in range(dims):
        xs.append(rest % shape[d])
        rest = rest // shape[d]
    stride = [math.prod(shape[:d]) for d in range(dims)]
    offs = sorted(coefs, key=lambda o: sum(a * s for a, s in zip(o, stride)))
    mask = torch.ones((n, len(offs)), dtype=torch.bool, device=DEV)
    col = torch.empty((n, len(offs)), dtype=torch.int32, device=DEV)
    val = torch.empty((n, len(offs)), dtype=torch.float64, device=DEV)
    for k, o in enumerate(offs):
        for d in range(dims):
            if o[d] == 1:
                mask[:, k] &= xs[d] < shape[d] - 1
            elif o[d] == -1:
                mask[:, k] &= xs[d] > 0
        col[:, k] = idx + sum(a * s for a, s in zip(o, stride))
        c = coefs[o]
        val[:, k] = c.reshape(-1) if isinstance(c, torch.Tensor) else c
    ia = torch.zeros(n + 1, dtype=torch.int32, device=DEV)
    ia[1:] = torch.cumsum(mask.sum(1), 0)
    return ia, col[mask], val[mask]


def _field(N, sigma, corr, seed):
    """Per-cube log-normal coefficient exp(sigma g), [z, y, x]."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randn((N, N, N), dtype=torch.float64, device=DEV, generator=g)
    f = torch.fft.fftfreq(N, dtype=torch.float64, device=DEV)
    fx = torch.fft.rfftfreq(N, dtype=torch.float64, device=DEV)
    r2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + fx[None, None, :] ** 2
    w = torch.fft.irfftn(torch.fft.rfftn(w) * torch.exp(-2.0 * (math.pi * corr) ** 2 * r2),
                         s=(N, N, N))
    w -= w.mean()
    w /= w.std()
    return torch.exp(sigma * w).contiguous()


def _kuhn(N, k=None, K=None):
    """P1 stiffness of -div(k K grad u) on N^3 Kuhn cubes, interior vertices."""
    K = np.eye(3) if K is None else np.asarray(K, float)
    acc = {}
    for p in itertools.permutations(range(3)):
        v = [np.zeros(3, int)]
        for a in p:
            e = v[-1].copy()
            e[a] += 1
            v.append(e)
        G = np.zeros((4, 3))
        G[:, list(p)] = [[-1, 0, 0], [1, -1, 0], [0, 1, -1], [0, 0, 1]]
        E = (G @ K @ G.T) / (6.0 * N)
        for a in range(4):
            for b in range(4):
                o = tuple(int(t) for t in v[b] - v[a])
                x, y, z = (1 - int(t) for t in v[a])     # the cubes of interior vertices
                if k is None:
                    acc[o] = acc.get(o, 0.0) + float(E[a, b])
                else:
                    if o not in acc:
                        acc[o] = torch.zeros((N - 1,) * 3, dtype=torch.float64, device=DEV)
                    if E[a, b] != 0.0:
                        acc[o].add_(k[z:z + N - 1, y:y + N - 1, x:x + N - 1],
                                    alpha=float(E[a, b]))
    return _stencil((N - 1,) * 3, acc)


def _aniso2d(m, eps, theta):
    """P1 stiffness of -div(K grad u), K = R diag(1, eps) R^T, right triangles."""
    c, s = math.cos(theta), math.sin(theta)
    R = np.array([[c, -s], [s, c]])
    K = R @ np.diag([1.0, eps]) @ R.T
    acc = {}
    for tri in ([(0, 0), (1, 0), (1, 1)], [(0, 0), (1, 1), (0, 1)]):
        t = np.array(tri, float)
        B = np.array([t[1] - t[0], t[2] - t[0]]).T
        G = np.array([[-1, -1], [1, 0], [0, 1]], float) @ np.linalg.inv(B)
        E = 0.5 * abs(np.linalg.det(B)) * (G @ K @ G.T)
        for a in range(3):
            for b in range(3):
                o = (tri[b][0] - tri[a][0], tri[b][1] - tri[a][1])
                acc[o] = acc.get(o, 0.0) + float(E[a, b])
    return _stencil((m, m), acc)


def _rhs(n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.rand(n, dtype=torch.float64, device=DEV, generator=g) * 2.0 - 1.0


def _scalar_problem(case, seed):
    if case["dim"] == 2:
        ia, ja, val = _aniso2d(case["m"], case["eps"], case["theta"])
    else:
        ia, ja, val = _kuhn(case["N"], _field(case["N"], case["sigma"], 8.0, 2 * seed + 1))
    return ia, ja, val, _rhs(len(ia) - 1, 2 * seed)


def _batch_problem(case, seed):
    """Anisotropic 2D and 3D systems packed on one block diagonal."""
    rng = np.random.default_rng([case["shapes"], seed])
    shape_rng = np.random.default_rng(case["shapes"])      # sizes belong to the case
    ias, jas, vals, off, eo = [], [], [], [0], 0
    for _ in range(case["nsys"]):
        d = math.exp(shape_rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        flat = shape_rng.uniform() < 0.5
        eps, th = float(rng.uniform(0.01, 1.0)), float(rng.uniform(0.0, math.pi))
        if flat:
            ia, ja, val = _aniso2d(max(2, round(d ** 0.5)), eps, th)
        else:
            c, s = math.cos(th), math.sin(th)
            R = np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
            ia, ja, val = _kuhn(max(3, round(d ** (1 / 3)) + 1),
                                None, R @ np.diag([1.0, 1.0, eps]) @ R.T)
        ias.append(ia[:-1] + eo)
        jas.append(ja + off[-1])
        vals.append(val)
        eo += len(ja)
        off.append(off[-1] + len(ia) - 1)
    ias.append(torch.tensor([eo], dtype=torch.int32, device=DEV))
    return (np.asarray(off, np.int32), torch.cat(ias), torch.cat(jas), torch.cat(vals),
            _rhs(off[-1], 2 * seed))


def _bsr_problem(case, seed):
    """Block (I, J) = K_IJ B plus a random SPD term on the diagonal blocks."""
    nb = case["nb"]
    ia, ja, val = _kuhn(case["N"], _field(case["N"], 1.0, 8.0, 2 * seed + 1))
    n = len(ia) - 1
    B = torch.tensor(COUPLING[nb], dtype=torch.float64, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(seed)
    G = torch.randn((n, nb, nb), dtype=torch.float64, device=DEV, generator=g)
    blocks = val[:, None, None] * B
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (ia[1:] - ia[:-1]).long())
    diag = torch.nonzero(ja == rows)[:, 0]
    blocks[diag] += 0.1 * (G @ G.transpose(1, 2)) / nb
    return ia, ja, blocks.contiguous(), _rhs(n * nb, 2 * seed)


# ---------------------------------------------------------------------------
# the program
# ---------------------------------------------------------------------------
def _amg(smoother):
    if smoother == "gs":
        return hz.bench_amg()
    return hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2, postsmooth_iter=2)


def _it(krylov="cg"):
    kind = {"cg": hz.SOLVER_CG, "fgmres": hz.SOLVER_VFGMRES}[krylov]
    return hz.itsolver_param(linear_itsolver_type=kind, linear_precond_type=hz.PREC_AMG,
                             linear_tol=1e-8, linear_maxit=1000, linear_restart=100,
                             linear_stop_type=hz.STOP_REL_RES)


def _b200(precision):
    if precision == "mixed":
        return hz.b200_param(precision=hz.HZB_PREC_MIXED, matching=hz.HZB_MATCH_PARALLEL)
    return hz.b200_param()


def _ok(rc, what):
    if rc < 0:
        raise RuntimeError(f"{what}: {rc} {hz.last_error()}")
    return rc


def _setup(s):
    _ok(s["S"].setup_device(len(s["b"]), len(s["ja"]), s["ia"].data_ptr(), s["ja"].data_ptr(),
                            s["val"].data_ptr()), "setup")


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "assemble":
        N = case["N"]
        n = (N - 1) ** 3
        s.update(N=N, k=_field(N, case["sigma"], 8.0, seed),
                 ia=torch.empty(n + 1, dtype=torch.int32, device=DEV))
        rc, nnz = hz.assemble_p1_kuhn_device(N, s["k"].data_ptr(), s["ia"].data_ptr())
        _ok(rc, "assemble")
        s.update(ja=torch.empty(nnz, dtype=torch.int32, device=DEV),
                 val=torch.empty(nnz, dtype=torch.float64, device=DEV))
        return s
    if kind == "batch":
        s["off"], s["ia"], s["ja"], s["val"], s["b"] = _batch_problem(case, seed)
        s["S"] = hz.Solver(_amg("l1"), _it(), _b200("mixed"))
    elif kind == "bsr":
        s["ia"], s["ja"], s["val"], s["b"] = _bsr_problem(case, seed)
        s["nb"] = case["nb"]
        s["S"] = hz.Solver(hz.bench_amg(coarse_dof=100, coarse_solver=0), _it())
    else:
        s["ia"], s["ja"], s["val"], s["b"] = _scalar_problem(case, seed)
        if kind == "dropin":
            for k in ("ia", "ja", "val", "b"):
                s[k] = s[k].cpu().numpy()
            s.update(smoother=case["smoother"], krylov=case["krylov"])
            return s
        if kind == "learn":
            n, ns = len(s["b"]), 4
            s["S"] = learn.l1_solver()
            s["gnn"] = learn.GNN(weights=learn.WEIGHTS)
            s["E"] = torch.empty((ns, n), dtype=torch.float64, device=DEV)
            for k in ("om", "d4", "d2"):
                s[k] = torch.empty(n, dtype=torch.float32, device=DEV)
            s["seed"] = seed + 1
        else:
            s["S"] = hz.Solver(_amg(case["smoother"]), _it(), _b200(case["precision"]))
    s["x"] = torch.zeros_like(s["b"])
    if kind in ("precond", "resolve", "learn"):
        torch.cuda.synchronize()
        _setup(s)
    return s


def run(s):
    kind, S = s["kind"], s.get("S")
    if kind == "assemble":
        rc, _ = hz.assemble_p1_kuhn_device(s["N"], s["k"].data_ptr(), s["ia"].data_ptr(),
                                           s["ja"].data_ptr(), s["val"].data_ptr())
        _ok(rc, "assemble")
        return {"ia": s["ia"], "ja": s["ja"], "val": s["val"]}
    if kind == "dropin":
        x = np.zeros(len(s["b"]))
        _ok(hz.linear_solver_dcsr_krylov_amg(s["ia"], s["ja"], s["val"], s["b"], x,
                                             _it(s["krylov"]), _amg(s["smoother"])), "solve")
        return x
    x = s["x"]
    if kind == "precond":
        _ok(S.precond_device(s["b"].data_ptr(), x.data_ptr()), "precond")
        return x
    if kind == "learn":
        gnn, ns = s["gnn"], len(s["E"])
        gnn.infer(S, s["om"].data_ptr())
        learn.errors(S, ns, s["seed"], s["E"].data_ptr(), None, 0)
        l4 = learn.loss_grad(S, s["om"].data_ptr(), s["E"].data_ptr(), ns, s["d4"].data_ptr(), 4)
        l2 = learn.loss_grad(S, s["om"].data_ptr(), s["E"].data_ptr(), ns, s["d2"].data_ptr(), 2)
        dom = s["d4"] / l4 - s["d2"] / l2
        gnn.zero_grad()
        torch.cuda.current_stream().synchronize()   # the library has streams of its own
        gnn.backward(S, dom.data_ptr())
        return {"omega": s["om"], "loss": [l4, l2], "domega": dom, "grads": gnn.grads()}
    x.zero_()
    torch.cuda.current_stream().synchronize()       # the library has streams of its own
    if kind == "step":
        _setup(s)
    if kind in ("step", "resolve"):
        _ok(S.solve_device(s["b"].data_ptr(), x.data_ptr()), "solve")
    elif kind == "batch":
        _ok(S.batch_setup_device(s["off"], len(s["ja"]), s["ia"].data_ptr(), s["ja"].data_ptr(),
                                 s["val"].data_ptr()), "setup")
        _ok(S.batch_solve_device(s["b"].data_ptr(), x.data_ptr())[0], "solve")
    else:
        _ok(S.setup_bsr_device(len(s["ia"]) - 1, len(s["ja"]), s["nb"], s["ia"].data_ptr(),
                               s["ja"].data_ptr(), s["val"].data_ptr()), "setup")
        _ok(S.bsr_solve_device(s["b"].data_ptr(), x.data_ptr()), "solve")
    return x


def _sizes(case):
    """(rows, stored entries) of a scalar problem."""
    if case.get("dim") == 2:
        m = case["m"]
        return m * m, 7 * m * m - 8 * m + 2
    m = case["N"] - 1
    one, two = m * m * (m - 1), m * (m - 1) ** 2
    return m ** 3, m ** 3 + 6 * one + 6 * two + 2 * (m - 1) ** 3


def work(case):
    kind = case["kind"]
    if kind == "assemble":
        n, nnz = _sizes(case)
        return {"bytes": 8 * case["N"] ** 3 + 4 * (n + 1) + 12 * nnz, "flops": 2 * 96 * n}
    if kind == "batch":
        shape_rng = np.random.default_rng(case["shapes"])
        n = nnz = 0
        for _ in range(case["nsys"]):
            d = math.exp(shape_rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
            one = ({"dim": 2, "m": max(2, round(d ** 0.5))} if shape_rng.uniform() < 0.5 else
                   {"dim": 3, "N": max(3, round(d ** (1 / 3)) + 1)})
            a, b = _sizes(one)
            n, nnz = n + a, nnz + b
    else:
        n, nnz = _sizes(case)
    nb = case.get("nb", 1)
    # the matrix, the right-hand side and the solution once; a multiply-add per entry
    return {"bytes": nnz * (8 * nb * nb + 4) + 4 * (n + 1) + 16 * n * nb,
            "flops": 2 * nnz * nb * nb}


# ---------------------------------------------------------------------------
# the solutions in 64 bits, without the library
# ---------------------------------------------------------------------------
def _solve(ia, ja, val, b, tol=1e-13, maxit=20000):
    """Jacobi-preconditioned CG on a torch CSR matrix."""
    n = len(ia) - 1
    A = torch.sparse_csr_tensor(ia, ja, val, (n, n))
    rows = torch.repeat_interleave(torch.arange(n, device=DEV, dtype=torch.int32),
                                   ia[1:] - ia[:-1])
    d = torch.zeros_like(b)
    on = ja == rows
    d[rows[on].long()] = val[on]
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, rz = z.clone(), torch.dot(r, z)
    stop = tol * float(torch.linalg.vector_norm(b))
    for k in range(maxit):
        t = A @ p
        a = rz / torch.dot(p, t)
        x += a * p
        r -= a * t
        if k % 50 == 49 and float(torch.linalg.vector_norm(r)) < stop:
            return x
        z = r / d
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return None


def exact(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        ia, ja, val = _kuhn(case["N"], _field(case["N"], case["sigma"], 8.0, seed))
        return {"ia": ia, "ja": ja, "val": val}
    if kind in ("precond", "learn"):
        return None
    if kind == "batch":
        _, ia, ja, val, b = _batch_problem(case, seed)
    elif kind == "bsr":
        nb = case["nb"]
        ia, ja, blocks, b = _bsr_problem(case, seed)
        n = len(ia) - 1
        I = torch.repeat_interleave(torch.arange(n, device=DEV), (ia[1:] - ia[:-1]).long())
        e = torch.arange(nb, device=DEV)
        row = (I * nb)[:, None, None] + e[:, None] + 0 * e
        col = (ja.long() * nb)[:, None, None] + 0 * e[:, None] + e
        A = torch.sparse_coo_tensor(torch.stack([row.reshape(-1), col.reshape(-1)]),
                                    blocks.reshape(-1)).coalesce().to_sparse_csr()
        ia, ja, val = A.crow_indices().int(), A.col_indices().int(), A.values()
    else:
        ia, ja, val, b = _scalar_problem(case, seed)
    x = _solve(ia, ja, val, b)
    return x if x is None or kind != "dropin" else x.cpu().numpy()
