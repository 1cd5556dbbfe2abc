"""Batched independent systems (hzb_batch_setup_device / hzb_batch_solve_device):
every system reaches its own tolerance on its own true FP64 residual, each
system's answer is the one an independent solve gives and is within the
tolerance's order of the reference's solve of that system alone, one system
alone takes about the single-system path's iterations, and an entry that
couples two systems is rejected."""
import numpy as np
import pytest
import scipy.sparse as sp

import hazmath_b200 as hz
from hazmath_b200 import problems as P

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _amg():
    return hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2, postsmooth_iter=2)


def _it(tol=1e-8):
    return hz.itsolver_param(linear_itsolver_type=hz.SOLVER_CG, linear_precond_type=hz.PREC_AMG,
                             linear_tol=tol, linear_maxit=400, linear_stop_type=hz.STOP_REL_RES)


def _solver(prec=None):
    prec = hz.HZB_PREC_MIXED if prec is None else prec
    return hz.Solver(_amg(), _it(), hz.b200_param(precision=prec,
                                                  matching=hz.HZB_MATCH_PARALLEL))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _batch_solve(union, prec=None):
    off, ia, ja, val, b = union
    S = _solver(prec)
    dia, dja, dval, db = _dev(ia), _dev(ja), _dev(val), _dev(b)
    rc = S.batch_setup_device(off, int(ia[-1]), dia.data_ptr(), dja.data_ptr(), dval.data_ptr())
    assert rc == 0, hz.last_error()
    dx = torch.zeros_like(db)
    rc, its, rel, sec = S.batch_solve_device(db.data_ptr(), dx.data_ptr())
    st = S.stats()
    S.close()
    return rc, its, rel, sec, dx.cpu().numpy(), st


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_batch_each_system_converges(prec):
    systems, union = P.batch_anisotropic(24, seed=3, dof_lo=500, dof_hi=30000)
    p = hz.HZB_PREC_MIXED if prec == "mixed" else hz.HZB_PREC_FP64
    rc, its, rel, sec, x, st = _batch_solve(union, p)
    assert rc == its.max() > 0, (rc, hz.last_error())
    off = union[0]
    for k, (ia, ja, val, b) in enumerate(systems):
        A = sp.csr_matrix((val, ja, ia))
        xk = x[off[k]:off[k + 1]]
        true_rel = np.linalg.norm(b - A @ xk) / np.linalg.norm(b)
        assert true_rel < 1e-8, (k, true_rel)
        assert rel[k] == pytest.approx(true_rel, rel=1e-3, abs=1e-14)
        assert 0 < its[k] <= its.max()
    assert np.all(sec > 0) and sec.max() <= st.solve_seconds * 1.01
    # a system that needs more iterations finishes no earlier
    order = np.argsort(its, kind="stable")
    assert sec[order[-1]] >= sec[order[0]]


def test_batch_matches_independent_solves():
    systems, union = P.batch_anisotropic(6, seed=5, dof_lo=2000, dof_hi=20000)
    rc, its, rel, sec, x, _ = _batch_solve(union)
    assert rc > 0, hz.last_error()
    off = union[0]
    for k, (ia, ja, val, b) in enumerate(systems):
        S = _solver()
        xs = np.zeros(len(b))
        assert S.setup_host(ia, ja, val) == 0
        it1 = S.solve_host(b, xs)
        S.close()
        assert it1 > 0
        A = sp.csr_matrix((val, ja, ia))
        xk = x[off[k]:off[k + 1]]
        # both are 1e-8 residual solutions of the same system
        err = np.linalg.norm(xk - xs) / np.linalg.norm(xs)
        assert err < 1e-5, (k, err)
        # the union's hierarchy is deeper for a small system (coarsening runs
        # until the whole union is small), which costs iterations, not accuracy
        assert its[k] <= 2 * it1 + 10, (k, its[k], it1)


def test_single_system_batch_is_the_single_system_solve():
    k = P.lognormal_field(24, 1.0, 4.0, 9)
    ia, ja, val = P.kuhn3d_p1(24, k)
    b = P.rhs_uniform(len(ia) - 1, 4)
    off = np.array([0, len(b)], np.int32)
    rc, its, rel, sec, x, _ = _batch_solve((off, ia, ja, val, b))
    S = _solver()
    xs = np.zeros(len(b))
    assert S.setup_host(ia, ja, val) == 0
    it1 = S.solve_host(b, xs)
    S.close()
    # the batch ends a system's coarsening at 128 rows (a dense block solve),
    # the single-system solve at coarse_dof = 2000 rows; the cycles differ
    # below that, so the counts may differ by a few
    assert abs(int(its[0]) - it1) <= 3, (int(its[0]), it1)
    assert np.linalg.norm(x - xs) / np.linalg.norm(xs) < 1e-6


def test_batch_rejects_coupled_systems():
    systems, union = P.batch_anisotropic(3, seed=7, dof_lo=500, dof_hi=2000)
    off, ia, ja, val, b = union
    ja = ja.copy()
    r = off[1]                       # first row of system 1 points into system 0
    ja[ia[r]] = 0
    S = _solver()
    dia, dja, dval = _dev(ia), _dev(ja), _dev(val)
    rc = S.batch_setup_device(off, int(ia[-1]), dia.data_ptr(), dja.data_ptr(),
                              dval.data_ptr())
    S.close()
    assert rc == hz.ERROR_INPUT_PAR


@pytest.mark.parametrize("prec,max_it", [("mixed", 3), ("fp64", 1)])
def test_batch_terminal_block_sizes(prec, max_it):
    """Systems small enough to be dense blocks from the start (each size at an
    edge of the 32-wide register tiles, up to the largest block): 4.5 on the
    diagonal and -1 at the distances 1 and 7, so the condition number is at
    most 8.5 / 0.5 and the block's inverse solves the system at once in FP64;
    in FP32 its relative error is about 1e-6 a cycle, so two or three reach
    1e-8."""
    rng = np.random.default_rng(3)
    mats, rhs = [], []
    for m in (1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128):
        A = sp.diags([np.full(m, 4.5)], [0]).tolil()
        for d in (1, 7):
            if d < m:
                A += sp.diags([-np.ones(m - d), -np.ones(m - d)], [d, -d])
        mats.append(sp.csr_matrix(A))
        rhs.append(rng.uniform(-1.0, 1.0, m))
    U = sp.block_diag(mats, format="csr")
    U.sort_indices()
    off = np.cumsum([0] + [len(b) for b in rhs]).astype(np.int32)
    p = hz.HZB_PREC_MIXED if prec == "mixed" else hz.HZB_PREC_FP64
    rc, its, rel, sec, x, _ = _batch_solve(
        (off, U.indptr.astype(np.int32), U.indices.astype(np.int32), U.data,
         np.concatenate(rhs)), p)
    assert rc > 0, hz.last_error()
    assert its.max() <= max_it
    for k, (A, b) in enumerate(zip(mats, rhs)):
        want = np.linalg.solve(A.toarray(), b)
        assert np.linalg.norm(x[off[k]:off[k + 1]] - want) <= 1e-6 * np.linalg.norm(want), k


def test_batch_against_reference_per_system(golden):
    """Each of the 24 systems solved by the batch (FP32 cycle, parallel
    matching, per-system flexible CG to 1e-8) against the same system solved
    on its own by the reference (tests/golden/batch.npz: FP64 UA-AMG with
    HEM, l1-Jacobi V(2,2), PCG): the error against the reference's solve
    tightened to 1e-12 is of the tolerance's order (below 1e-6 relative),
    and the iteration counts are bounded against the reference's: a system
    the reference coarsens (more than coarse_dof = 2000 rows) needs at most
    2.5 times the reference's iterations; a smaller one the reference solves
    directly (one iteration), while the batch runs it through the union's
    hierarchy (at most 25 iterations)."""
    g = golden("batch.npz")
    systems, union = P.batch_anisotropic(24, seed=3, dof_lo=500, dof_hi=30000)
    rc, its, rel, sec, x, _ = _batch_solve(union)
    assert rc > 0, hz.last_error()
    off = union[0]
    st = int(g["stride"])
    worst, rows = 0.0, []
    for k in range(len(systems)):
        xs = g[f"{k}/x_sample"]
        xk = x[off[k]:off[k + 1]][::st]
        err = np.linalg.norm(xk - xs) / np.linalg.norm(xs)
        worst = max(worst, err)
        rows.append((k, len(systems[k][3]), int(its[k]), int(g[f"{k}/iters"]), err))
        assert err < 1e-6, (k, err)
    print("system, dofs, batch its, reference its, error vs reference 1e-12 solve:")
    for r in rows:
        print("  %2d %6d %4d %4d %.2e" % r)
    for k, n, ib, ir, _ in rows:
        assert ib <= (2.5 * ir if n > 2000 else 25), (k, n, ib, ir)
