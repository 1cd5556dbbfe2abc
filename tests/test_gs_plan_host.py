"""The stages of a streamed Gauss-Seidel schedule (csrc/hzb_gs_plan.h), on the CPU.

A sweep in turns fetches set s when the sets up to s - 3 are complete, and waits
for the copy into its stage by the parity of the copy's round; so the copy of the
round before has to have landed by then."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "hazmath_b200", "csrc")
SHIM = r"""
#include "hzb_gs_plan.h"
#include <cstring>
extern "C" int places(int ns, const int *ptr, int *start) {
    std::vector<int> p(ptr, ptr + ns + 1), st;
    const int n = hzb::gs_places(p, &st);
    if (n) std::memcpy(start, st.data(), sizeof(int) * ns);
    return n;
}
extern "C" void plan(int ns, const int *ptr, const int *start, int places, const int *width,
                     int dist, long long *out) {
    std::vector<int> p(ptr, ptr + ns + 1), st(start, start + ns), w(width, width + ns);
    const hzb::GsPlan P = hzb::gs_plan(p, st, places, w, dist);
    out[0] = P.uniform; out[1] = P.group; out[2] = P.stages; out[3] = P.ring;
    out[4] = (long long)hzb::gs_smem(ns, P.E, P.R, P.ring, P.stages);
    out[5] = (long long)hzb::GS_SMEM; out[6] = hzb::GS_TURNS;
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("gs_plan")
    src, so = str(d / "shim.cpp"), str(d / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", so],
                   check=True)
    return C.CDLL(so)


def grid(nx, ny, px=False, py=False, corners=False):
    """Neighbour lists of a 5-point grid, periodic in x or y, or with one
    coupling between its first and last point."""
    i = np.arange(nx * ny).reshape(ny, nx)
    pairs = [(i[:, :-1], i[:, 1:]), (i[:-1], i[1:])]
    if px:
        pairs.append((i[:, :1], i[:, -1:]))
    if py:
        pairs.append((i[:1], i[-1:]))
    if corners:
        pairs.append((i[:1, :1], i[-1:, -1:]))
    a = np.concatenate([p.ravel() for p, _ in pairs])
    b = np.concatenate([q.ravel() for _, q in pairs])
    nb = [[] for _ in range(nx * ny)]
    for u, v in zip(a.tolist(), b.tolist()):
        nb[u].append(v)
        nb[v].append(u)
    return nb


def plan_of(lib, nb, backward=False):
    n = len(nb)
    lev = [0] * n
    for r in range(n):
        lo = [lev[j] for j in nb[r] if j < r]
        lev[r] = 1 + max(lo) if lo else 0
    lev = np.array(lev)
    if backward:
        lev = lev.max() - lev
    rows = np.lexsort((np.arange(n), lev))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(lev))]).astype(np.int32)
    ns = len(ptr) - 1
    start = np.zeros(ns, np.int32)
    ip = lambda a: a.ctypes.data_as(C.c_void_p)
    places = lib.places(ns, ip(ptr), ip(start))
    if not places:
        return None
    place = np.empty(n, np.int64)
    width = np.zeros(ns, np.int32)
    for k in range(ns):
        m = rows[ptr[k]:ptr[k + 1]]
        place[m] = start[k] + np.arange(len(m))
        width[k] = (max(len(nb[r]) for r in m) + 1) // 2 * 2
    dist = max(abs(int(place[r]) - int(place[j])) for r in range(n) for j in nb[r])
    out = np.zeros(7, np.int64)
    lib.plan(ns, ip(ptr), ip(start), places, ip(width), dist, ip(out))
    return dict(ns=ns, uniform=int(out[0]), group=int(out[1]), stages=int(out[2]),
                ring=int(out[3]), smem=int(out[4]), limit=int(out[5]), turns=int(out[6]))


# group and stages of each, 0: no stream.  The last ones leave room for two
# stages of one set, which only the single sequence may take.
CASES = [
    (dict(nx=40, ny=40), (4, 8, 3)),
    (dict(nx=255, ny=255), None),
    (dict(nx=100, ny=100, py=True), None),
    (dict(nx=127, ny=127, py=True), None),
    (dict(nx=137, ny=137, px=True), None),
    (dict(nx=145, ny=145, px=True, py=True), (4, 1, 4)),
    (dict(nx=151, ny=151, px=True, py=True), (4, 1, 3)),
    (dict(nx=153, ny=153, px=True), (0, None, None)),
    (dict(nx=153, ny=153, py=True), (0, None, None)),
    (dict(nx=154, ny=154, px=True, py=True), (0, None, None)),
    (dict(nx=154, ny=154, corners=True), (0, None, None)),
    (dict(nx=100, ny=242, py=True), (0, None, None)),
    (dict(nx=140, ny=168, py=True), (0, None, None)),
    (dict(nx=200, ny=200, py=True), (0, 0, 0)),
]


@pytest.mark.parametrize("backward", [False, True])
@pytest.mark.parametrize("kw,want", CASES, ids=["-".join(map(str, c[0].values())) for c in CASES])
def test_stages_outlast_the_turns(planner, kw, want, backward):
    p = plan_of(planner, grid(**kw), backward)
    assert p is not None
    if p["stages"]:
        assert p["smem"] <= p["limit"] and p["ring"] <= 0xff00 and p["ring"] % 256 == 0
    if p["stages"] and p["uniform"]:
        # the copy before the one that set s waits for was into the group
        # `stages` earlier; its first set has to be complete
        s = np.arange(p["ns"])
        before = (s // p["group"] - p["stages"]) * p["group"]
        assert (before[before >= 0] <= s[before >= 0] - p["turns"]).all()
    if want:
        for got, w in zip((p["uniform"], p["group"], p["stages"]), want):
            assert w is None or got == w
