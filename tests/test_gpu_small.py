"""The merged kernels of the l1-Jacobi V-cycle's small levels: the FP64 cycle bit for bit
against the same cycle put together from the kernel-level entry points, the
FP32 cycle against the FP64 one to FP32 rounding."""
import numpy as np
import pytest
import scipy.sparse as sp

import hazmath_b200 as hz
from hazmath_b200 import problems as P
from gpu_util import DevCSR, dev, host, ptr

pytestmark = pytest.mark.gpu


def _amg(pre, post, **kw):
    return hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=pre, postsmooth_iter=post,
                        **kw)


def _precond(S, r):
    d, z = dev(r), dev(np.zeros(len(r)))
    assert S.precond_device(ptr(d), ptr(z)) == 0, hz.last_error()
    return host(z)


def _sweeps(A, k, b, x):
    x = dev(x)
    assert hz.lib().hzb_smoother_device(hz.SMOOTHER_L1DIAG, 1, k, 1.0, *A.args(), ptr(dev(b)),
                                        ptr(x)) == 0
    return host(x)


def _cycle(S, l, pre, post, b):
    ia, ja, val, agg = S.level(l)
    if l == S.stats().num_levels - 1:
        # reported as its transpose, which is what is factored: a hierarchy of
        # its own transposes once more
        At = sp.csr_matrix((val, ja, ia)).T.tocsr()
        At.sort_indices()
        C = hz.Solver(hz.bench_amg(coarse_dof=len(ia)))
        assert C.setup_host(At.indptr, At.indices, At.data) == 0
        assert C.stats().num_levels == 1
        x = _precond(C, b)
        C.close()
        return x
    A = DevCSR(ia, ja, val)
    x = _sweeps(A, pre, b, np.zeros(len(b)))
    t = dev(np.zeros(len(b)))
    assert hz.lib().hzb_dcsr_mxv_device(*A.args(), ptr(dev(x)), ptr(t)) == 0
    w = b - host(t)
    bc = np.zeros(S.stats().rows[l + 1])
    for i in range(len(b)):
        if agg[i] >= 0:
            bc[agg[i]] += w[i]
    xc = _cycle(S, l + 1, pre, post, bc)
    return _sweeps(A, post, b, x + np.where(agg >= 0, xc[np.maximum(agg, 0)], 0.0))


PROBLEMS = {
    "2d_20": (lambda: P.poisson2d_5pt(20), 50),             # all levels
    "aniso_75": (lambda: P.aniso2d_p1(75, 0.1, 0.5), 300),
    "kuhn_28": (lambda: P.kuhn3d_p1(28, P.lognormal_field(28, 1.0, 4.0, 2)), 1500),
    "2d_257": (lambda: P.poisson2d_5pt(257), 2000),
    "2d_512": (lambda: P.poisson2d_5pt(512), 2000),         # 262144 rows, the FP32 limit; the
                                                            # FP64 levels start one below
    "2d_513": (lambda: P.poisson2d_5pt(513), 2000),
}


@pytest.mark.parametrize("name", sorted(PROBLEMS))
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2), (3, 2), (1, 2)])
def test_fp64_small_levels_bit_exact(name, pre, post):
    make, cdof = PROBLEMS[name]
    ia, ja, val = make()
    r = P.rhs_uniform(len(ia) - 1, 5)
    S = hz.Solver(_amg(pre, post, coarse_dof=cdof))
    assert S.setup_host(ia, ja, val) == 0, hz.last_error()
    assert S.stats().num_levels >= 2
    z = _precond(S, r)
    assert np.array_equal(z, _precond(S, r))
    assert np.array_equal(z, _cycle(S, 0, pre, post, r))
    S.close()


@pytest.mark.parametrize("name", sorted(PROBLEMS))
@pytest.mark.parametrize("pre,post", [(1, 1), (2, 2), (2, 3)])
def test_fp32_small_levels_to_rounding(name, pre, post):
    make, cdof = PROBLEMS[name]
    ia, ja, val = make()
    r = P.rhs_uniform(len(ia) - 1, 5)
    z = []
    for precision in (hz.HZB_PREC_FP64, hz.HZB_PREC_MIXED):
        S = hz.Solver(_amg(pre, post, coarse_dof=cdof), None,
                      hz.b200_param(precision=precision, matching=hz.HZB_MATCH_PARALLEL))
        assert S.setup_host(ia, ja, val) == 0, hz.last_error()
        if precision == hz.HZB_PREC_MIXED:
            it = S.solve_host(r, np.zeros(len(r)))
            assert it > 0
            om = dev(np.ones(len(r), np.float32))           # weights of one change nothing
            assert S.set_omega_device(ptr(om)) == 0
            assert S.solve_host(r, np.zeros(len(r))) == it
            z.append(S)
        else:
            z.append(_precond(S, r))
            S.close()
    S = z.pop()
    # one cycle: the first iterate of the flexible CG is alpha times it
    x = np.zeros(len(r))
    it1 = hz.itsolver_param(linear_itsolver_type=1, linear_precond_type=2, linear_tol=1e-30,
                            linear_maxit=1, linear_stop_type=1)
    T = hz.Solver(_amg(pre, post, coarse_dof=cdof), it1,
                  hz.b200_param(precision=hz.HZB_PREC_MIXED, matching=hz.HZB_MATCH_PARALLEL))
    assert T.setup_host(ia, ja, val) == 0
    T.solve_host(r, x)
    alpha = np.dot(x, z[0]) / np.dot(z[0], z[0])
    # a value passes about 20 rounded operations per sweep and level
    tol = 20 * 2 * (pre + post + 1) * S.stats().num_levels * 2.0 ** -24
    assert np.abs(x - alpha * z[0]).max() <= tol * np.abs(alpha * z[0]).max()
    S.close()
    T.close()


def _gs(A, pre, k, b, x):
    x = dev(x)
    assert hz.lib().hzb_smoother_device(hz.SMOOTHER_GS, pre, k, 1.0, *A.args(), ptr(dev(b)),
                                        ptr(x)) == 0
    return host(x)


@pytest.mark.parametrize("smoother", [hz.SMOOTHER_L1DIAG, hz.SMOOTHER_GS])
@pytest.mark.parametrize("make", [lambda: P.poisson2d_5pt(45), lambda: P.aniso2d_p1(50, 0.1, 0.5),
                                  lambda: P.kuhn3d_p1(14, P.lognormal_field(14, 1.0, 4.0, 2))],
                         ids=["2d_45", "aniso_50", "kuhn_14"])
def test_values_changed_in_the_callers_array(smoother, make):
    """A matrix in the caller's device arrays: level 0's sweeps and residual read
    its values as they are at the call (only the hierarchy and the Gauss-Seidel
    diagonals, which stay the same here, are the setup's)."""
    ia, ja, val = make()
    n = len(ia) - 1
    A = DevCSR(ia, ja, val)
    S = hz.Solver(hz.bench_amg(smoother=smoother, coarse_dof=n * 3 // 4))
    assert S.setup_device(*A.args()) == 0
    assert S.stats().num_levels == 2
    agg = S.level(0)[3]
    r = P.rhs_uniform(n, 5)
    _precond(S, r)                       # captured with the first values
    row = np.repeat(np.arange(n), np.diff(ia))
    new = np.where(ja == row, val, val * np.random.default_rng(1).uniform(0.4, 0.9, len(ja)))
    A.val.copy_(dev(new))
    got = _precond(S, r)
    sweep = _gs if smoother == hz.SMOOTHER_GS else lambda A, pre, k, b, x: _sweeps(A, k, b, x)
    x = sweep(A, 1, 1, r, np.zeros(n))
    t = dev(np.zeros(n))
    assert hz.lib().hzb_dcsr_mxv_device(*A.args(), ptr(dev(x)), ptr(t)) == 0
    w = r - host(t)
    bc = np.zeros(S.stats().rows[1])
    for i in range(n):
        if agg[i] >= 0:
            bc[agg[i]] += w[i]
    xc = _cycle(S, 1, 1, 1, bc)
    want = sweep(A, 0, 1, r, x + np.where(agg >= 0, xc[np.maximum(agg, 0)], 0.0))
    assert np.array_equal(got, want)
    S.close()


def _random_graph(n, deg, seed):
    rng = np.random.default_rng(seed)
    i, j = rng.integers(0, n, n * deg // 2), rng.integers(0, n, n * deg // 2)
    A = sp.coo_matrix((-rng.uniform(0.5, 1.5, len(i)), (i, j)), shape=(n, n)).tocsr()
    A = A + A.T
    A.setdiag(0)
    A.eliminate_zeros()
    A = (A + sp.diags(1.01 * -np.asarray(A.sum(1)).ravel() + 0.1)).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


# aggregates and rows on both sides of the merged kernels' rule
@pytest.mark.parametrize("agg", [hz.HEM, hz.HEC, hz.VMB])
@pytest.mark.parametrize("make", [lambda: P.poisson2d_5pt(90), lambda: _random_graph(5000, 8, 1),
                                  lambda: _random_graph(5000, 22, 2),
                                  lambda: _random_graph(5000, 40, 3)],
                         ids=["2d_90", "random_8", "random_22", "random_40"])
def test_fp64_cycle_by_aggregates_bit_exact(agg, make):
    ia, ja, val = make()
    r = P.rhs_uniform(len(ia) - 1, 5)
    S = hz.Solver(_amg(1, 2, coarse_dof=600, aggregation_type=agg))
    assert S.setup_host(ia, ja, val) == 0, hz.last_error()
    assert S.stats().num_levels >= 2
    assert np.array_equal(_precond(S, r), _cycle(S, 0, 1, 2, r))
    S.close()


@pytest.mark.parametrize("precision", [hz.HZB_PREC_FP64, hz.HZB_PREC_MIXED])
def test_large_aggregates_keep_the_separate_kernels(precision):
    """HEC aggregates of hundreds of long rows: an iteration takes no more than 3
    times one with pairs on the same matrix (merged, where a thread takes an
    aggregate's rows one after the other, 15 times)."""
    ia, ja, val = _random_graph(20000, 60, 1)
    b = P.rhs_uniform(len(ia) - 1, 5)
    t = {}
    for agg in (hz.HEC, hz.HEM):
        S = hz.Solver(_amg(2, 2, aggregation_type=agg), None, hz.b200_param(precision=precision))
        assert S.setup_host(ia, ja, val) == 0, hz.last_error()
        t[agg] = []
        for _ in range(4):
            assert S.solve_host(b, np.zeros(len(b))) > 0
            st = S.stats()
            t[agg].append(st.solve_seconds / st.iterations)
        S.close()
    assert min(t[hz.HEC]) < 3 * min(t[hz.HEM])
