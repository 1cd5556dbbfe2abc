"""The deterministic parallel matching (matching = HZB_MATCH_PARALLEL) against
a plain restatement of its rules: rounds of mutual choice, handshake rounds on
hashed coins, leftovers to their first aggregated neighbour (all pairs have two
members), aggregates numbered by their smallest vertex."""
import numpy as np
import pytest

import hazmath_b200 as hz
from hazmath_b200 import problems as P

pytestmark = pytest.mark.gpu

M32 = 0xFFFFFFFF
LEAD, ROUNDS, IDLE = 4, 100, 4


def _mix(x):
    x ^= x >> 16
    x = x * 0x7feb352d & M32
    x ^= x >> 15
    x = x * 0x846ca68b & M32
    return x ^ (x >> 16)


def _edge(i, j):
    lo, hi = min(i, j), max(i, j)
    return _mix((lo * 0x9e3779b1 & M32) ^ ((hi + 0x7f4a7c15 + (lo << 6) + (lo >> 2)) & M32))


def _red(k, r):
    return (_mix((k * 2654435761 + r * 0x632be5ab) & M32) >> 7) & 1


def match_rules(ia, ja, val, theta):
    n = len(ia) - 1
    diag = np.zeros(n)
    for i in range(n):
        for k in range(ia[i], ia[i + 1]):
            if ja[k] == i:
                diag[i] = val[k]
                break
    rows, state = [], np.full(n, -2)
    for i in range(n):
        strong = [(int(j), float(np.float32(abs(v)))) for j, v in
                  zip(ja[ia[i]:ia[i + 1]], val[ia[i]:ia[i + 1]])
                  if j == i or (v * v >= theta * theta * abs(diag[i] * diag[j]) and v < 0)]
        if len(strong) > 1:
            state[i] = -1
        rows.append([e for e in strong if e[0] != i])
    npair, idle, r = 0, 0, 0

    def best_of(k, ok):
        b = None
        for j, w in rows[k]:
            if ok(j):
                key = (w, _edge(k, j), j)
                if b is None or key > b:
                    b = key
        return -1 if b is None else b[2]

    while r < ROUNDS and idle < IDLE:
        mutual = r < LEAD
        ptr = [best_of(k, lambda j: state[j] == -1 and (mutual or not _red(j, r)))
               if state[k] == -1 and (mutual or _red(k, r)) else -1 for k in range(n)]
        pairs = []
        for j in range(n):
            if state[j] != -1:
                continue
            if mutual:
                p = ptr[j]
                if 0 <= p < j and ptr[p] == j:
                    pairs.append((j, p))
            elif not _red(j, r):
                i = best_of(j, lambda i: ptr[i] == j)
                if i >= 0:
                    pairs.append((j, i))
        for j, i in pairs:
            state[j] = state[i] = npair
            npair += 1
        idle = 0 if pairs or mutual else idle + 1
        r += 1
    agg = state.copy()
    for k in range(n):
        if state[k] == -1:
            agg[k] = next((state[j] for j, _ in rows[k] if state[j] >= 0), -1)
            if agg[k] < 0:
                agg[k] = npair
                npair += 1
    number = {}
    for k in range(n):
        if agg[k] >= 0:
            agg[k] = number.setdefault(int(agg[k]), len(number))
        else:
            agg[k] = -1
    return agg, len(number)


def _asymmetric(n, seed):
    """Rows of 0 to 12 off-diagonal entries, few distinct weights, positive
    ones among them, columns in no order, isolated rows that others name."""
    rng = np.random.default_rng(seed)
    ia, ja, val = [0], [], []
    for i in range(n):
        m = int(rng.integers(0, 13))
        c = rng.choice(n, size=min(m, n), replace=False)
        c = c[c != i]
        e = np.r_[c, i]
        v = np.r_[rng.integers(-4, 2, len(c)).astype(float), 9.0]
        o = rng.permutation(len(e))
        ja.extend(e[o])
        val.extend(v[o])
        ia.append(len(ja))
    return np.array(ia, np.int32), np.array(ja, np.int32), np.array(val)


CASES = {
    "2d": (P.poisson2d_5pt(40), 0.0),
    "aniso": (P.aniso2d_p1(37, 0.02, 0.8), 0.1),
    "kuhn": (P.kuhn3d_p1(12, P.lognormal_field(12, 1.0, 3.0, 3)), 0.0),
    "one_cta": (P.poisson2d_5pt(22), 0.0),
    "asymmetric": (_asymmetric(1500, 1), 0.0),
    "asymmetric_theta": (_asymmetric(513, 2), 0.2),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_parallel_matching_rules(case):
    (ia, ja, val), theta = CASES[case]
    agg_o, nc = match_rules(ia, ja, val, theta)
    amg = hz.bench_amg(smoother=hz.SMOOTHER_JACOBI, strong_coupled=theta, coarse_dof=10,
                       max_levels=2, coarse_solver=0)
    S = hz.Solver(amg, None, hz.b200_param(matching=hz.HZB_MATCH_PARALLEL))
    assert S.setup_host(ia, ja, val) == 0, hz.last_error()
    assert S.stats().num_levels == 2 and S.stats().rows[1] == nc
    assert np.array_equal(S.level(0)[3], agg_o)
    S.close()
