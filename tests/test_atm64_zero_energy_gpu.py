"""Triplets at the angle where the ATM energy vanishes (1 + 3 cos cos cos = 0) still have
forces: an atom whose only triplet has an energy of exactly zero gets them all the same."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import D3Batch

pytestmark = pytest.mark.gpu

BOHR = 0.52917726


def angular(pos):
    a, b, c = pos
    t = lambda u, v: u @ v / np.linalg.norm(u) / np.linalg.norm(v)  # noqa: E731
    return 1.0 + 3.0 * t(b - a, c - a) * t(a - b, c - b) * t(a - c, b - c)


def zero_triplet(rng):
    """Three copper atoms with sides of 4.5 to 6.5 bohr at the first atom and the opening angle
    solved by bisection; coordinates near the origin, so that separations round little."""
    r1, r2 = rng.uniform(4.5, 6.5, 2)
    u, v = np.linalg.qr(rng.normal(size=(3, 2)))[0].T
    at = lambda th: np.array([np.zeros(3), r1 * u, r2 * (np.cos(th) * u + np.sin(th) * v)])  # noqa: E731
    lo, hi = 0.55 * np.pi, 0.95 * np.pi
    lo, hi = (lo, hi) if angular(at(lo)) > 0 else (hi, lo)
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if angular(at(mid)) > 0 else (lo, mid)
    p = at(lo)
    return {"pos": (p - p.min(0)) * BOHR, "Z": np.array([29, 29, 29]), "cell": np.eye(3) * 30.0}


def test_forces_of_triplets_without_energy():
    rc = dict(rc=40.0, rc_cn=20.0, rc_atm=20.0)
    rng = np.random.default_rng(1)
    edge = (80 / 0.1) ** (1.0 / 3.0)
    # a dense structure beside them keeps the evaluation on block pairs
    parts = [S.random_box(80, edge * np.eye(3), seed=2)] + [zero_triplet(rng) for _ in range(64)]
    assert max(abs(angular(s["pos"])) for s in parts[1:]) < 1e-13
    b = D3Batch([1, 6, 7, 8, 29], len(parts), sum(len(s["Z"]) for s in parts), **rc)
    b.set_structures(parts)
    e, f, st = b.compute()
    b.close()
    for k, s in enumerate(parts):
        r = oracle.compute(s["pos"], s["Z"], s["cell"], c6_mode=1, **rc)
        assert abs(e[k] - r["energy"]) <= 1e-9 * abs(r["energy"])
        assert np.abs(f[k] - r["forces"]).max() <= 1e-7
        assert np.abs(st[k] - r["stress"]).max() <= 1e-7
