"""The coarsest level's dense inverse alone: a matrix of at most coarse_dof
rows makes a hierarchy of one level, whose preconditioner application is the
inverse times r.  Compared with numpy's solve in FP64; sizes around the 32-row
panels, the 64-row tiles and the doubling steps' incomplete pairs."""
import numpy as np
import pytest

import hazmath_b200 as hz
from hazmath_b200 import problems as P
from gpu_util import dev, host, ptr

pytestmark = pytest.mark.gpu


def _shifted(n, seed):
    """SPD band matrix of n rows with unsymmetric-looking fill and a condition
    number of about 1e3."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for off in (1, 2, 7, 40):
        if off < n:
            w = -rng.uniform(0.1, 1.0, n - off)
            A += np.diag(w, off) + np.diag(w, -off)
    return A + np.diag(np.abs(A).sum(1) + 0.005 * rng.uniform(0.5, 1.0, n))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 129, 160, 257, 1024, 1025,
                               1999])
def test_dense_inverse_sizes(n):
    A = _shifted(n, n)
    rows, cols = np.nonzero(A)
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    S = hz.Solver(hz.bench_amg())
    assert S.setup_host(ia, cols.astype(np.int32), A[rows, cols]) == 0, hz.last_error()
    assert S.stats().num_levels == 1
    r = np.random.default_rng(n + 1).uniform(-1, 1, n)
    d, z = dev(r), dev(np.zeros(n))
    assert S.precond_device(ptr(d), ptr(z)) == 0
    x = np.linalg.solve(A, r)
    # forward error of a Cholesky-based inverse: a small multiple of n eps cond
    tol = 4.0 * max(n, 8) * np.finfo(float).eps * np.linalg.cond(A)
    assert np.abs(host(z) - x).max() <= tol * np.abs(x).max()
    S.close()


def test_indefinite_coarse_matrix_is_refused():
    ia, ja, val = P.poisson2d_5pt(20)
    val = val.copy()
    val[ja == np.repeat(np.arange(400), np.diff(ia))] = 1.0   # indefinite
    S = hz.Solver(hz.bench_amg())
    assert S.setup_host(ia, ja, val) == hz.ERROR_DATA_ZERODIAG
    S.close()
