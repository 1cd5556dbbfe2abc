"""Kernel-level parity of the CUDA library against the reference's outputs
(golden fixtures) and the CPU oracle, through the C ABI on device arrays.
Integer outputs and every FP64 kernel are compared bit for bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import hazmath_b200 as hz
from hazmath_b200 import problems as P
from gpu_util import DevCSR, dev, host, ptr

pytestmark = pytest.mark.gpu


def test_mxv_aAxpy_bit_exact(golden):
    g = golden("smoothers.npz")
    A = DevCSR(g["ia"], g["ja"], g["val"])
    x = dev(g["x0"])
    y = dev(np.zeros(A.n))
    assert hz.lib().hzb_dcsr_mxv_device(*A.args(), ptr(x), ptr(y)) == 0
    assert np.array_equal(host(y), g["mxv"])
    for alpha, key in ((-1.0, "aAxpy_m1"), (0.7, "aAxpy_07")):
        y = dev(g["b"])
        assert hz.lib().hzb_dcsr_aAxpy_device(alpha, *A.args(), ptr(x), ptr(y)) == 0
        assert np.array_equal(host(y), g[key])


@pytest.mark.parametrize("N", [9, 40])
def test_mxv_kuhn_vs_oracle(port, N):
    """15-point Kuhn pattern with explicit zeros; N = 40 exercises bundles
    of 128 rows x 15 entries staged in shared memory."""
    ia, ja, val = P.kuhn3d_p1(N, P.lognormal_field(N, 1.0, 4.0, 7))
    x = np.random.default_rng(1).uniform(-1, 1, len(ia) - 1)
    A = DevCSR(ia, ja, val)
    y = dev(np.zeros(A.n))
    assert hz.lib().hzb_dcsr_mxv_device(*A.args(), ptr(dev(x)), ptr(y)) == 0
    assert np.array_equal(host(y), port.mxv(ia, ja, val, x))


@pytest.mark.parametrize("sm", [1, 2, 3, 5, 6, 7, 8, 10])
@pytest.mark.parametrize("pre", [1, 0])
def test_smoothers_bit_exact(golden, sm, pre):
    """GS/SGS/SOR through the level-scheduled exact sweep; Jacobi and
    l1-Jacobi row-parallel: all equal to the reference's sequential loops."""
    g = golden("smoothers.npz")
    A = DevCSR(g["ia"], g["ja"], g["val"])
    x = dev(g["x0"])
    rc = hz.lib().hzb_smoother_device(sm, pre, 2, 1.2, *A.args(), ptr(dev(g["b"])), ptr(x))
    assert rc == 0, hz.last_error()
    assert np.array_equal(host(x), g[f"s{sm}_pre{pre}"])


@pytest.mark.parametrize("sm", [6, 7, 8])
@pytest.mark.parametrize("pre", [1, 0])
def test_combined_smoothers_vs_oracle(port, sm, pre):
    ia, ja, val = P.aniso2d_p1(23, 0.03, 0.4)
    rng = np.random.default_rng(sm * 10 + pre)
    b, x0 = rng.uniform(-1, 1, len(ia) - 1), rng.uniform(-1, 1, len(ia) - 1)
    A = DevCSR(ia, ja, val)
    x = dev(x0)
    assert hz.lib().hzb_smoother_device(sm, pre, 1, 1.15, *A.args(), ptr(dev(b)), ptr(x)) == 0
    assert np.array_equal(host(x), port.smooth(sm, pre, 1, ia, ja, val, b, x0, relax=1.15))


def _hem(ia, ja, val, theta):
    A = DevCSR(ia, ja, val)
    agg = dev(np.zeros(A.n, np.int32))
    nc = C.c_int()
    rc = hz.lib().hzb_aggregation_hem_device(*A.args(), theta, ptr(agg), C.byref(nc))
    assert rc == 0, hz.last_error()
    return nc.value, host(agg)


@pytest.mark.parametrize("case", ["aniso2d_31", "kuhn_12", "theta_p2d_40"])
def test_hem_matches_reference_level0(golden, case):
    z = golden("small_cases.npz")
    theta = float(z[f"{case}/dparams"][0])
    nc, agg = _hem(z[f"{case}/A_ia"], z[f"{case}/A_ja"], z[f"{case}/A_val"], theta)
    assert np.array_equal(agg, z[f"{case}/agg0"])
    assert nc == int(z[f"{case}/info"][0][2])


@pytest.mark.parametrize("seed", range(4))
def test_hem_random_vs_oracle(port, seed):
    rng = np.random.default_rng(seed)
    m = int(rng.integers(15, 60))
    ia, ja, val = P.aniso2d_p1(m, float(10 ** rng.uniform(-4, 0)), float(rng.uniform(0, np.pi)))
    theta = float(rng.choice([0.0, 0.1, 0.3]))
    nc, agg = _hem(ia, ja, val, theta)
    nc_o, agg_o = port.hem(ia, ja, val, theta)
    assert nc == nc_o and np.array_equal(agg, agg_o)


@pytest.mark.parametrize("path", [1, 2, 3, 4])
def test_hem_implementations_agree(golden, port, monkeypatch, path):
    # ranked lists + byte ring, ranked lists + bit ring, bit ring over the raw
    # rows, state in global memory: the same aggregates as the reference
    monkeypatch.setenv("HZB_HEM_PATH", str(path))
    z = golden("small_cases.npz")
    for case in ["aniso2d_31", "kuhn_12", "theta_p2d_40"]:
        theta = float(z[f"{case}/dparams"][0])
        nc, agg = _hem(z[f"{case}/A_ia"], z[f"{case}/A_ja"], z[f"{case}/A_val"], theta)
        assert np.array_equal(agg, z[f"{case}/agg0"]), case
        assert nc == int(z[f"{case}/info"][0][2])
    k = P.lognormal_field(14, 1.0, 3.0, 7)
    ia, ja, val = P.kuhn3d_p1(14, k)
    rows = np.repeat(np.arange(len(ia) - 1), np.diff(ia))
    val = val * (1.0 + 0.01 * ((rows + ja + path) % 3))   # symmetric ties and near-ties
    nc, agg = _hem(ia, ja, val, 0.05)
    nc_o, agg_o = port.hem(ia, ja, val, 0.05)
    assert nc == nc_o and np.array_equal(agg, agg_o)


def _random_graph(n, deg, seed, symmetric):
    """Random CSR with negative off-diagonals of few distinct weights (ties),
    wide rows and any bandwidth."""
    rng = np.random.default_rng(seed)
    m = max(1, n * deg // 2)
    i, j = rng.integers(0, n, m), rng.integers(0, n, m)
    i, j = i[i != j], j[i != j]
    w = -rng.integers(1, 6, len(i)).astype(float)
    if symmetric:
        i, j, w = np.r_[i, j], np.r_[j, i], np.r_[w, w]
    key, first = np.unique(i * n + j, return_index=True)
    k = np.r_[key, np.arange(n) * (n + 1)]
    v = np.r_[w[first], np.full(n, 50.0)]
    order = np.argsort(k)
    k, v = k[order], v[order]
    ia = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(k // n, minlength=n), out=ia[1:])
    return ia.astype(np.int32), (k % n).astype(np.int32), v


@pytest.mark.parametrize("n,deg,symmetric", [
    (2, 2, True), (1024, 6, True), (1025, 6, True), (2049, 5, False), (8193, 40, True),
    (16384, 6, True), (16385, 6, True), (40000, 7, False), (200001, 8, True)])
def test_hem_rounds_vs_oracle(port, n, deg, symmetric):
    """One CTA, clusters of 2 to 8, the grid, a window smaller than the graph;
    rows without a partner and graphs that are not symmetric."""
    ia, ja, val = _random_graph(n, deg, n, symmetric)
    nc_o, agg_o = port.hem(ia, ja, val, 0.0)
    nc, agg = _hem(ia, ja, val, 0.0)
    assert nc == nc_o and np.array_equal(agg, agg_o)


def test_rap_bit_exact(golden):
    g = golden("rap.npz")
    A = DevCSR(g["ia"], g["ja"], g["val"])
    nc = int(g["nc"])
    nnz = C.c_int()
    pia, pja, pval = C.c_void_p(), C.c_void_p(), C.c_void_p()
    rc = hz.lib().hzb_rap_agg_device(*A.args(), nc, ptr(dev(g["agg"])), C.byref(nnz),
                                     C.byref(pia), C.byref(pja), C.byref(pval))
    assert rc == 0, hz.last_error()
    out = []
    for p, n, dt in ((pia, nc + 1, np.int32), (pja, nnz.value, np.int32),
                     (pval, nnz.value, np.float64)):
        h = np.empty(n, dt)
        assert hz.lib().hzb_copy_to_host(C.c_void_p(h.ctypes.data), p,
                                         C.c_size_t(h.nbytes)) == 0
        hz.lib().hzb_free_device(p)
        out.append(h)
    assert np.array_equal(out[0], g["cia"])
    assert np.array_equal(out[1], g["cja"])
    assert np.array_equal(out[2], g["cval"])


def _rap_plain(ia, ja, val, nc, agg):
    """A_c = R A P in the reference's slot order: the diagonal first (from
    0.0), other columns where they are first met, sums in traversal order."""
    members = [[] for _ in range(nc)]
    for i, c in enumerate(agg):
        if c >= 0:
            members[c].append(i)
    cia, cja, cval = [0], [], []
    for c in range(nc):
        slot, vals = {c: 0}, [0.0]
        for i in members[c]:
            for k in range(ia[i], ia[i + 1]):
                cc = int(agg[ja[k]])
                if cc < 0:
                    continue
                if cc in slot:
                    vals[slot[cc]] += val[k]
                else:
                    slot[cc] = len(vals)
                    vals.append(float(val[k]))
        cja += list(slot)
        cval += vals
        cia.append(len(cja))
    return np.array(cia, np.int32), np.array(cja, np.int32), np.array(cval)


@pytest.mark.parametrize("n,lens,members", [
    (40, (0, 3), 2),           # rows of at most 32 entries together, empty rows
    (300, (14, 18), 2),        # around 32 entries: with and without the table
    (300, (30, 33), 2),        # around 64: the first list's bound
    (200, (60, 130), 2),       # around 256: the second list
    (400, (1, 3), 40),         # more than 32 fine rows in an aggregate
    (1500, (900, 1100), 2),    # around 2048: the scratch rows
])
def test_rap_row_sizes_bit_exact(n, lens, members):
    rng = np.random.default_rng(n + lens[1])
    m = rng.integers(lens[0], lens[1] + 1, n)
    ia = np.zeros(n + 1, np.int32)
    np.cumsum(m, out=ia[1:])
    ja = np.concatenate([rng.permutation(n)[:k] for k in m]).astype(np.int32)
    val = rng.uniform(-1.0, 1.0, len(ja))
    val[rng.random(len(val)) < 0.05] = -0.0
    nc = n // members
    agg = np.r_[np.arange(nc), rng.integers(0, nc, n - nc)].astype(np.int32)
    agg[nc:][rng.random(n - nc) < 0.05] = -1
    A = DevCSR(ia, ja, val)
    nnz = C.c_int()
    pia, pja, pval = C.c_void_p(), C.c_void_p(), C.c_void_p()
    rc = hz.lib().hzb_rap_agg_device(*A.args(), nc, ptr(dev(agg)), C.byref(nnz), C.byref(pia),
                                     C.byref(pja), C.byref(pval))
    assert rc == 0, hz.last_error()
    cia, cja, cval = _rap_plain(ia, ja, val, nc, agg)
    got = []
    for q, like in ((pia, cia), (pja, cja), (pval, cval)):
        a = np.empty_like(like)
        assert nnz.value == len(cja)
        assert hz.lib().hzb_copy_to_host(a.ctypes.data, q, a.nbytes) == 0
        hz.lib().hzb_free_device(q)
        got.append(a)
    assert np.array_equal(got[0], cia) and np.array_equal(got[1], cja)
    assert np.array_equal(got[2].view(np.int64), cval.view(np.int64))


def _wide(n, seed):
    """Rows of 0 to 40 off-diagonal entries to both sides, unsorted, the
    diagonal anywhere."""
    rng = np.random.default_rng(seed)
    ia, ja, val = [0], [], []
    for i in range(n):
        c = rng.choice(n, size=min(n, int(rng.integers(0, 41))), replace=False)
        c = rng.permutation(np.r_[c[c != i], i])
        ja.extend(c)
        val.extend(np.where(c == i, 60.0, rng.uniform(-1.0, 1.0, len(c))))
        ia.append(len(ja))
    return np.array(ia, np.int32), np.array(ja, np.int32), np.array(val)


GS_PROBLEMS = {
    "one_row": lambda: P.poisson2d_5pt(1),
    "2d_16": lambda: P.poisson2d_5pt(16),
    "2d_256": lambda: P.poisson2d_5pt(256),      # sets of up to 256 rows: the last that stream
    "2d_257": lambda: P.poisson2d_5pt(257),      # runs of sets in the row kernels
    "aniso_61": lambda: P.aniso2d_p1(61, 0.1, 0.5),
    "kuhn_17": lambda: P.kuhn3d_p1(17, P.lognormal_field(17, 1.0, 4.0, 7)),
    "wide_300": lambda: _wide(300, 5),
}


@pytest.mark.parametrize("name", sorted(GS_PROBLEMS))
@pytest.mark.parametrize("sm,pre", [(2, 1), (2, 0), (3, 1), (5, 1), (5, 0), (6, 1)])
def test_streamed_gauss_seidel_vs_oracle(port, name, sm, pre):
    """GS, SGS (which leaves the last row out of its way back), SOR and SSOR on
    schedules with small sets, both directions, several sweeps."""
    ia, ja, val = GS_PROBLEMS[name]()
    n = len(ia) - 1
    rng = np.random.default_rng(n + sm)
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    A = DevCSR(ia, ja, val)
    x = dev(x0)
    assert hz.lib().hzb_smoother_device(sm, pre, 2, 1.15, *A.args(), ptr(dev(b)), ptr(x)) == 0
    assert np.array_equal(host(x), port.smooth(sm, pre, 2, ia, ja, val, b, x0, relax=1.15))


def _stencil(N, ny, centre, side, corner):
    """5- or 9-point stencil on N x ny points, row by row; ny = 1: a chain."""
    ia, ja, val = [0], [], []
    for i in range(N * ny):
        y, x = divmod(i, N)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                v = centre if dx == dy == 0 else corner * (1 + 0.1 * dx) if dx and dy else side
                if v and 0 <= y + dy < ny and 0 <= x + dx < N:
                    ja.append((y + dy) * N + x + dx)
                    val.append(v)
        ia.append(len(ja))
    return np.array(ia, np.int32), np.array(ja, np.int32), np.array(val)


GS_WIDTHS = {
    "chain_2": lambda: _stencil(2, 1, 2.5, -1.0, 0.0),     # fewer sets than take turns
    "chain_4": lambda: _stencil(4, 1, 2.5, -1.0, 0.0),
    "chain_700": lambda: _stencil(700, 1, 2.5, -1.0, 0.0),  # 2 entries a row, sets of one row
    "five_70": lambda: _stencil(70, 70, 4.5, -1.0, 0.0),   # 4
    "seven_40": lambda: P.aniso2d_p1(40, 0.1, 0.5),        # 6
    "nine_64": lambda: _stencil(64, 64, 9.0, -1.0, -0.5),  # 8
}


@pytest.mark.parametrize("name", sorted(GS_WIDTHS))
@pytest.mark.parametrize("sm,pre", [(2, 1), (3, 1), (6, 0)])
def test_streamed_gauss_seidel_row_widths(port, name, sm, pre):
    """Schedules streamed with one width for all sets, for each width."""
    ia, ja, val = GS_WIDTHS[name]()
    n = len(ia) - 1
    rng = np.random.default_rng(n + sm)
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    A = DevCSR(ia, ja, val)
    x = dev(x0)
    assert hz.lib().hzb_smoother_device(sm, pre, 3, 1.15, *A.args(), ptr(dev(b)), ptr(x)) == 0
    assert np.array_equal(host(x), port.smooth(sm, pre, 3, ia, ja, val, b, x0, relax=1.15))


def _periodic(nx, ny, px, py):
    """5-point matrix of a grid periodic in x or y, CSR rows ascending."""
    def line(m, per):
        d = sp.diags([np.full(m - 1, -1.0), np.full(m - 1, -1.0)], [-1, 1], format="lil")
        if per:
            d[0, m - 1] = d[m - 1, 0] = -0.75
        return d.tocsr()
    a = sp.kron(sp.eye(ny), line(nx, px)) + sp.kron(line(ny, py), sp.eye(nx)) * 1.25
    a = (a + sp.eye(nx * ny) * 4.75).tocsr()
    a.sort_indices()
    return a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data


# far couplings: the ring grows, and the choice of stages goes through the small
# groups down to two stages of one set (from 153 points a side on), which the
# single sequence takes
@pytest.mark.parametrize("nx,ny,px,py", [
    (100, 100, 0, 1), (127, 127, 1, 0), (137, 137, 0, 1), (145, 145, 1, 1), (151, 151, 1, 1),
    (153, 153, 1, 0), (153, 153, 0, 1), (154, 154, 1, 1), (100, 242, 0, 1)])
@pytest.mark.parametrize("sm,pre", [(2, 1), (2, 0), (6, 1)])
def test_streamed_gauss_seidel_far_couplings(port, nx, ny, px, py, sm, pre):
    ia, ja, val = _periodic(nx, ny, px, py)
    n = len(ia) - 1
    rng = np.random.default_rng(n + sm)
    b, x0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    A = DevCSR(ia, ja, val)
    x = dev(x0)
    assert hz.lib().hzb_smoother_device(sm, pre, 2, 1.15, *A.args(), ptr(dev(b)), ptr(x)) == 0
    assert np.array_equal(host(x), port.smooth(sm, pre, 2, ia, ja, val, b, x0, relax=1.15))


def _strip(nx, ny, seed=None, periodic=False):
    """5-point graph of nx x ny points (ny = 1: a chain), weights 1 or random."""
    i = np.arange(nx * ny).reshape(ny, nx)
    pairs = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:])]
    if periodic:
        pairs.append((i[:, :1], i[:, -1:]))
    a = np.concatenate([p.ravel() for p, _ in pairs])
    b = np.concatenate([q.ravel() for _, q in pairs])
    w = np.ones(len(a)) if seed is None else np.random.default_rng(seed).uniform(0.5, 1.5, len(a))
    n = nx * ny
    A = sp.coo_matrix((-w, (a, b)), shape=(n, n)).tocsr()
    A = (A + A.T + sp.eye(n) * 5.0).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


# rows that can only be decided one after the other: the rounds give way to the
# walk (chains, strips of a few rows), or do not (wider ones); with couplings
# beyond the byte ring (65,504 rows) and beyond the bit ring, where the rounds
# go on to their end
@pytest.mark.parametrize("nx,ny,kw", [
    (500, 1, {}), (2001, 1, {"seed": 1}), (16384, 1, {}), (16385, 1, {}), (100000, 1, {"seed": 2}),
    (2, 20000, {}), (4, 9000, {"seed": 3}), (16, 3000, {}), (64, 700, {}), (9000, 4, {}),
    (70000, 1, {"periodic": True}), (530000, 1, {"periodic": True, "seed": 4})])
def test_hem_chains_and_strips(port, nx, ny, kw):
    ia, ja, val = _strip(nx, ny, **kw)
    nc, agg = _hem(ia, ja, val, 0.0)
    nc_o, agg_o = port.hem(ia, ja, val, 0.0)
    assert nc == nc_o and np.array_equal(agg, agg_o)


def test_hem_chain_no_slower_than_the_walk(monkeypatch):
    """A chain of 100,000 rows, one decision after the other: 3 times the walk's
    time at most (the rounds to their end take 20 times)."""
    import time
    ia, ja, val = _strip(100000, 1)
    best = {}
    for path in ("0", "2"):
        monkeypatch.setenv("HZB_HEM_PATH", path)
        _hem(ia, ja, val, 0.0)
        best[path] = 1e9
        for _ in range(3):
            t = time.perf_counter()
            _hem(ia, ja, val, 0.0)
            best[path] = min(best[path], time.perf_counter() - t)
    assert best["0"] < 3 * best["2"]


@pytest.mark.parametrize("nx,ny", [(64, 64), (4097, 1), (64, 128), (2731, 3), (128, 128)])
def test_hem_rounds_of_cluster_and_grid(port, monkeypatch, nx, ny):
    """Both sides of the sizes where the walk, the cluster and the grid take over
    (4096 and 8192 rows), the rounds to their end too."""
    ia, ja, val = _strip(nx, ny, seed=5)
    nc_o, agg_o = port.hem(ia, ja, val, 0.0)
    for path in ("0", "1"):
        monkeypatch.setenv("HZB_HEM_PATH", path)
        nc, agg = _hem(ia, ja, val, 0.0)
        assert nc == nc_o and np.array_equal(agg, agg_o)


def test_hem_rounds_are_not_given_up_on_a_growing_front(monkeypatch):
    """The first coarse level of a 2D grid of 600^2 points, whose sweep front
    builds up for hundreds of rounds: no more than 1.3 times the rounds to their
    end (given up by the pace of the first rounds alone, 2.3 times)."""
    import time
    ia, ja, val = P.aniso2d_p1(600, 1.0, 0.0)
    S = hz.Solver(hz.bench_amg(smoother=hz.SMOOTHER_L1DIAG))
    assert S.setup_host(ia, ja, val) == 0
    A = DevCSR(*S.level(1)[:3])
    S.close()
    agg, nc = dev(np.zeros(A.n, np.int32)), C.c_int()
    best = {}
    for path in ("0", "1"):
        monkeypatch.setenv("HZB_HEM_PATH", path)
        times = []
        for _ in range(4):
            t = time.perf_counter()
            assert hz.lib().hzb_aggregation_hem_device(*A.args(), 0.0, ptr(agg), C.byref(nc)) == 0
            times.append(time.perf_counter() - t)
        best[path] = min(times)
    assert best["0"] < 1.3 * best["1"]
