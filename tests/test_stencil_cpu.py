"""Bin stencils (csrc/d3_geometry.cpp) against a brute-force distance between bins: every
offset whose closest point pair lies within the cutoff is in its row, and no offset beyond
the neighbours of a borderline one is added."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "lasp-d3_b200", "csrc")
DRIVER = r"""
#include "d3_geometry.h"
#include <cstdio>
using namespace d3;
int main() {
    double h[9], r;
    int nb[3], gy, gz;
    while (scanf("%lf%lf%lf%lf%lf%lf%lf%lf%lf%lf%d%d%d%d%d", h, h + 1, h + 2, h + 3, h + 4, h + 5, h + 6, h + 7, h + 8, &r, nb,
                 nb + 1, nb + 2, &gy, &gz) == 15) {
        const auto st = build_stencil(make_geom(h), nb, r);
        const auto bl = merge_block_stencil(st, gy, gz);
        printf("%zu %zu\n", st.size(), bl.size());
        for (const auto &x : st) printf("%d %d %d %d\n", x.dy, x.dz, x.dxlo, x.dxhi);
        for (const auto &x : bl) printf("%d %d %d %d\n", x.dy, x.dz, x.dxlo, x.dxhi);
    }
}
"""


def min_dist2(G, d):
    """min over u in [-1,1]^3 of (d+u)^T G (d+u) by the 27 active sets."""
    best = np.full(len(d), np.inf)
    for code in range(27):
        st = np.array([code % 3, code // 3 % 3, code // 9])
        v = d + np.where(st == 1, -1.0, np.where(st == 2, 1.0, 0.0))
        fr, fx = np.nonzero(st == 0)[0], np.nonzero(st != 0)[0]
        ok = np.ones(len(d), bool)
        if len(fr):
            x = -np.linalg.solve(G[np.ix_(fr, fr)], G[np.ix_(fr, fx)] @ v[:, fx].T).T if len(fx) else np.zeros((len(d), 3))
            ok = (np.abs(x - d[:, fr]) <= 1.0).all(1)
            v[:, fr] = x
        q = np.einsum("ni,ij,nj->n", v, G, v)
        best = np.where(ok, np.minimum(best, q), best)
    return best


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("stencil")
    (d / "driver.cpp").write_text(DRIVER)
    exe = str(d / "driver")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "driver.cpp"), os.path.join(CSRC, "d3_geometry.cpp"),
                           "-o", exe])
    return exe


@pytest.mark.parametrize("seed", range(12))
def test_stencil_matches_brute_force(driver, seed):
    rng = np.random.default_rng(seed)
    nb = rng.integers(1, 7, 3)
    h = np.diag(rng.uniform(6.0, 30.0, 3)) + (rng.uniform(-12.0, 12.0, (3, 3)) if seed % 3 else 0.0)
    if seed % 4 == 1:
        h = h[[1, 0, 2]]  # left-handed
    if abs(np.linalg.det(h)) < 200.0:
        h = np.diag([9.0, 14.0, 7.0])
    r = rng.uniform(3.0, 40.0)
    gy, gz = rng.integers(1, 5, 2)
    args = " ".join(repr(float(x)) for x in h.ravel()) + " %r %d %d %d %d %d\n" % (float(r), *nb, gy, gz)
    out = subprocess.run([driver], input=args, capture_output=True, text=True, check=True).stdout.split()
    n, nblk = int(out[0]), int(out[1])
    rows = np.array(out[2:], int).reshape(-1, 4)
    assert len(rows) == n + nblk
    st = {(y, z): (lo, hi) for y, z, lo, hi in rows[:n].tolist()}
    assert len(st) == n
    M = h / nb[:, None]
    G = M @ M.T
    height = 1.0 / np.linalg.norm(np.linalg.inv(h), axis=0) / nb
    ext = np.ceil(r / height).astype(int) + 2
    grid = np.stack(np.meshgrid(*[np.arange(-e, e + 1) for e in ext], indexing="ij"), -1).reshape(-1, 3)
    q = min_dist2(G, grid.astype(float))
    lo = np.array([st.get((y, z), (1, 0))[0] for _, y, z in grid.tolist()])
    hi = np.array([st.get((y, z), (1, 0))[1] for _, y, z in grid.tolist()])
    has = (grid[:, 0] >= lo) & (grid[:, 0] <= hi)
    assert has[q <= r * r].all()
    assert not has[q > (r * (1 + 1e-8) + 1e-5) ** 2].any()
    # block stencil: the union of the member rows' ranges, each row offset once
    blk = {}
    for oz in range(gz):
        for oy in range(gy):
            for (y, z), (a, b) in st.items():
                a0, b0 = blk.get((y + oy, z + oz), (a, b))
                blk[(y + oy, z + oz)] = (min(a, a0), max(b, b0))
    assert {(y, z): (a, b) for y, z, a, b in rows[n:].tolist()} == blk
