"""The FP32 cycle's sliced-ELL schedule against the staged row bundles.

Both sum every row of a level in CSR order in FP32, one thread per row (the
bundles from shared memory, the sliced copy from its column-major slices), so
the mixed solve takes the same iterates bit for bit whichever of the two the
levels run.  HZB_FP32_LANES forces the schedule of every level of at least
4096 rows ("sell") or the bundles everywhere ("0").  The coarse levels of the
Kuhn hierarchy have ragged rows (4 to ~30 entries), so the slices carry
padding: zeros against the row's own last column, which must leave its sum as
it is."""
import numpy as np
import pytest
import scipy.sparse as sp

import hazmath_b200 as hz
from hazmath_b200 import problems as P
from gpu_util import dev, host, ptr

pytestmark = pytest.mark.gpu


def mixed_solve(monkeypatch, schedule, ia, ja, val, b):
    monkeypatch.setenv("HZB_FP32_LANES", schedule)
    S = hz.Solver(hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2,
                               postsmooth_iter=2),
                  b200=hz.b200_param(precision=hz.HZB_PREC_MIXED))
    assert S.setup_host(ia, ja, val) == 0, hz.last_error()
    x = np.zeros(len(b))
    it = S.solve_host(b, x)
    st = S.stats()
    levels = [(int(st.rows[l]), int(st.nnz[l])) for l in range(st.num_levels)]
    S.close()
    return it, x, levels


@pytest.mark.parametrize("N,sigma", [(24, 1.0), (40, 1.5)])
def test_sell_matches_bundles_bitwise(monkeypatch, N, sigma):
    ia, ja, val = P.kuhn3d_p1(N, P.lognormal_field(N, sigma, 8.0, 7))
    b = P.rhs_uniform(len(ia) - 1, 8)
    it_s, x_s, lv_s = mixed_solve(monkeypatch, "sell", ia, ja, val, b)
    it_b, x_b, lv_b = mixed_solve(monkeypatch, "0", ia, ja, val, b)
    assert lv_s == lv_b
    assert sum(1 for n, _ in lv_s if n >= 4096) >= 2   # the sliced copy ran on 2+ levels
    assert it_s == it_b > 0
    assert np.array_equal(x_s, x_b)
    A = sp.csr_matrix((val, ja, ia), shape=(len(b), len(b)))
    assert np.linalg.norm(b - A @ x_s) / np.linalg.norm(b) < 1e-8


@pytest.mark.parametrize("n,far", [(4097, 0), (150001, 70000), (150016, 149000)])
def test_sell_column_widths(monkeypatch, n, far):
    """Slices whose columns at one position span more than 16 bits (rows that
    couple over ``far`` beside rows that do not, forward beside backward) keep
    32-bit columns, the others 16-bit ones; the last window is partly or fully filled
    (n mod 256 = 1, 241 and 0), rows have odd and even lengths."""
    A = sp.diags([np.full(n, 4.25), -np.ones(n - 1), -np.ones(n - 1)], [0, 1, -1]).tocsr()
    if far:
        i = np.arange(0, n - far, 97)
        F = sp.coo_matrix((np.full(len(i), -0.5), (i, i + far)), shape=(n, n)).tocsr()
        A = (A + F + F.T).tocsr()
    A.sort_indices()
    ia, ja, val = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    b = P.rhs_uniform(n, 5)
    it_s, x_s, _ = mixed_solve(monkeypatch, "sell", ia, ja, val, b)
    it_b, x_b, _ = mixed_solve(monkeypatch, "0", ia, ja, val, b)
    assert it_s == it_b > 0
    assert np.array_equal(x_s, x_b)
    assert np.linalg.norm(b - A @ x_s) / np.linalg.norm(b) < 1e-8


def test_many_partial_sums(monkeypatch):
    """More partial sums of the outer product than one CTA adds (above 16384 of
    at most 256 rows each), the last of them of a part of its rows: the solve
    still ends at its true residual, in the same bits on both schedules."""
    n = 16384 * 256 + 4099
    A = sp.diags([np.full(n, 4.25), -np.ones(n - 1), -np.ones(n - 1)], [0, 1, -1]).tocsr()
    ia, ja, val = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data
    b = P.rhs_uniform(n, 5)
    out = []
    for schedule in ("sell", "0"):
        monkeypatch.setenv("HZB_FP32_LANES", schedule)
        S = hz.Solver(hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2,
                                   postsmooth_iter=2),
                      b200=hz.b200_param(precision=hz.HZB_PREC_MIXED,
                                         matching=hz.HZB_MATCH_PARALLEL))
        assert S.setup_host(ia, ja, val) == 0, hz.last_error()
        x = np.zeros(n)
        out.append((S.solve_host(b, x), x))
        S.close()
    assert out[0][0] == out[1][0] > 0
    assert np.array_equal(out[0][1], out[1][1])
    assert np.linalg.norm(b - A @ out[0][1]) / np.linalg.norm(b) < 1e-8


@pytest.mark.parametrize("N", [48, 64])
def test_fp64_sliced_levels_bitwise(N):
    """An FP64 solve whose large levels run from zero-free sliced copies: set up
    from host arrays (level 0 too) and from device arrays (level 0 stays in the
    caller's), the same iterates bit for bit."""
    torch = pytest.importorskip("torch")
    ia, ja, val = P.kuhn3d_p1(N, P.lognormal_field(N, 1.0, 8.0, 7))
    b = P.rhs_uniform(len(ia) - 1, 8)
    amg = hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2, postsmooth_iter=2)
    par = hz.b200_param(precision=hz.HZB_PREC_FP64, matching=hz.HZB_MATCH_PARALLEL)
    S = hz.Solver(amg, b200=par)
    assert S.setup_host(ia, ja, val) == 0, hz.last_error()
    x = np.zeros(len(b))
    it = S.solve_host(b, x)
    S.close()
    D = hz.Solver(amg, b200=par)
    dia, dja, dval, db = (torch.from_numpy(np.ascontiguousarray(a)).cuda()
                          for a in (ia, ja, val, b))
    dx = torch.zeros_like(db)
    assert D.setup_device(len(b), len(ja), dia.data_ptr(), dja.data_ptr(),
                          dval.data_ptr()) == 0, hz.last_error()
    assert D.solve_device(db.data_ptr(), dx.data_ptr()) == it > 0
    D.close()
    assert np.array_equal(x, dx.cpu().numpy())


@pytest.mark.parametrize("N", [48, 64])
def test_fp64_sliced_and_staged_levels_bitwise(monkeypatch, N):
    """The two forms of the FP64 cycle's large levels, each forced by
    HZB_FP64_SELL (the bytes that hzb_time_kernel counts tell which one a level
    has): the same iterates bit for bit."""
    ia, ja, val = P.kuhn3d_p1(N, P.lognormal_field(N, 1.0, 8.0, 7))
    b = P.rhs_uniform(len(ia) - 1, 8)
    out = []
    for form in ("1", "0"):
        monkeypatch.setenv("HZB_FP64_SELL", form)
        S = hz.Solver(hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, presmooth_iter=2,
                                   postsmooth_iter=2),
                      b200=hz.b200_param(precision=hz.HZB_PREC_FP64,
                                         matching=hz.HZB_MATCH_PARALLEL))
        assert S.setup_host(ia, ja, val) == 0, hz.last_error()
        x = np.zeros(len(b))
        it = S.solve_host(b, x)
        st = S.stats()
        large = [l for l in range(st.num_levels - 1) if st.nnz[l] > 1250000]
        out.append((it, x, [S.time_kernel(hz.HZB_K_L1_64, l, 1)[1] for l in large]))
        S.close()
    (it_s, x_s, by_s), (it_b, x_b, by_b) = out
    assert len(by_s) == len(by_b) >= (2 if N == 64 else 1)
    assert all(s != t for s, t in zip(by_s, by_b))
    assert it_s == it_b > 0
    assert np.array_equal(x_s, x_b)


def test_infinite_x_beside_padding(monkeypatch):
    """Rows shorter than their slice are filled up with zeros against a column of
    their own: an infinite x there leaves their result what the row's own entries
    make it (infinite, not NaN).  The rows of very different lengths below are
    coupled too weakly to aggregate, so nothing but the sweeps reaches them; a
    few have no entries but stored zeros, which the sliced copy drops."""
    rng = np.random.default_rng(4)
    ia, ja, val = P.kuhn3d_p1(48, P.lognormal_field(48, 1.0, 8.0, 7))
    G = sp.csr_matrix((val, ja, ia))
    m, k = len(ia) - 1, 1000
    i = np.repeat(np.arange(k), rng.integers(0, 25, k))
    j = rng.integers(0, k, len(i))
    W = sp.coo_matrix((np.full(len(i), -1e-3), (i, j)), shape=(k, k)).tocsr()
    W = W + W.T
    W.setdiag(10.0)
    A = sp.block_diag([G, W]).tocsr()
    A.sort_indices()
    ia, ja, val = A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data.copy()
    hit = m + np.arange(3, k, 7)
    for q in range(m + 502, m + 520):   # the columns too: the matrix stays symmetric
        if q not in hit:
            val[ia[q]:ia[q + 1]] = 0.0
            val[ja == q] = 0.0
    r = P.rhs_uniform(m + k, 3)
    r[hit] = np.inf
    z = []
    for form in ("1", "0"):
        monkeypatch.setenv("HZB_FP64_SELL", form)
        S = hz.Solver(hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG, strong_coupled=0.1),
                      b200=hz.b200_param(precision=hz.HZB_PREC_FP64,
                                         matching=hz.HZB_MATCH_PARALLEL))
        assert S.setup_host(ia, ja, val) == 0, hz.last_error()
        d, o = dev(r), dev(np.zeros(m + k))
        assert S.precond_device(ptr(d), ptr(o)) == 0, hz.last_error()
        z.append(host(o))
        S.close()
    assert np.isfinite(z[1][:m]).all()
    assert np.isinf(z[1][m:]).sum() > len(hit)       # the neighbours of the rows hit
    assert np.array_equal(z[0], z[1], equal_nan=True)
