"""Order of the ATM half lists: each triplet once, from its highest atom, where the
reference's image box cannot cut a pair within rc_ATM, and the reference's own order where
it can. Both forms against the FP64 oracle, at their parity bars, and the triplet count of
the reference's enumeration."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_PAIR_KERNEL, OPT_PRECISION, D3

pytestmark = pytest.mark.gpu


def tri(n, seed, density=0.09):
    edge = (n / density) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [-0.2, 0.15, 1.0]]), seed=seed)


def system(kind):
    rng = np.random.default_rng(5)
    rc = 60.0
    if kind == "inside":
        s = tri(60, 3)
    elif kind == "drifted":  # a little outside the cell on all sides
        s = tri(60, 3)
        s["pos"] = s["pos"] + rng.uniform(-1.0, 1.0, s["pos"].shape)
    elif kind == "scattered":  # cells away: the image box cuts pairs within rc_ATM
        s = tri(40, 4)
        s["pos"] = s["pos"] + rng.integers(-3, 4, s["pos"].shape) @ s["cell"]
    elif kind == "short_box":  # pair cutoffs below rc_ATM: the box cuts pairs within rc_ATM
        s, rc = tri(30, 6), 16.0
    elif kind == "ties":  # perfect lattice: many equal heights
        s = S.gtest_bcc_fe()
    elif kind == "left_handed":
        s = tri(50, 7)
        s["cell"] = s["cell"][[1, 0, 2]]
    else:  # thin along the third vector
        s = tri(48, 8)
        s = {"pos": s["pos"] * [2.0, 2.0, 0.25], "Z": s["Z"], "cell": s["cell"] * [2.0, 2.0, 0.25]}
    return s, rc


@pytest.mark.parametrize("precision,pair_kernel", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("kind", ["inside", "drifted", "scattered", "short_box", "ties", "left_handed", "thin"])
def test_order_matches_reference_enumeration(kind, precision, pair_kernel):
    s, rc = system(kind)
    rc_cn, rc_atm = min(rc, 30.0), 28.0
    d = D3(s["Z"], len(s["Z"]), rc=rc, rc_cn=rc_cn, rc_atm=rc_atm)
    d.set_option(OPT_PRECISION, precision)
    d.set_option(OPT_PAIR_KERNEL, pair_kernel)
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    e, f, st = d.compute()
    _, cnt = d.pass_times()
    d.pass_terms()  # diagnostics rebuild the lists in the reference's order
    e2, f2, _ = d.compute()
    _, cnt2 = d.pass_times()
    d.close()
    r = oracle.compute(s["pos"], s["Z"], s["cell"], rc=rc, rc_cn=rc_cn, rc_atm=rc_atm, c6_mode=1)
    triplets = oracle.counts(s["pos"], s["cell"], rc=rc, rc_cn=rc_cn, rc_atm=rc_atm)[2]
    e_rel, f_abs, s_abs = (1e-6, 1e-4, 1e-6) if precision else (1e-9, 1e-7, 1e-7)
    assert abs(e - r["energy"]) <= e_rel * abs(r["energy"])
    assert np.abs(f - r["forces"]).max() <= f_abs
    assert np.abs(st - r["stress"]).max() <= s_abs
    for c in (cnt, cnt2):
        assert abs(int(c[0]) - 2 * triplets) <= (2 * triplets * 1e-5 if precision else 0)
    assert abs(e2 - e) <= e_rel * abs(e) and np.abs(f2 - f).max() <= f_abs
