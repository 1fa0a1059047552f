"""FP64 block-pair ATM kernel at the edges of its blocks and of the rule that chooses it,
against the FP64 oracle and against the other FP64 schedule (bar of the plain form: energy
1e-9 relative, forces and stress 1e-7)."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_ATM_FORCE_SCALED, OPT_ATM_SCHEDULE, D3

pytestmark = pytest.mark.gpu

ONE = (("C", 1.0),)
SEVEN = (("H", 0.3), ("C", 0.2), ("N", 0.1), ("O", 0.1), ("Si", 0.1), ("Fe", 0.1), ("Cu", 0.1))


def evaluate(s, rc_atm, ext, scaled, schedule):
    d = D3(s["Z"], len(s["Z"]), rc=50.0, rc_cn=25.0, rc_atm=rc_atm, table=1 if ext else 0)
    d.set_option(OPT_ATM_SCHEDULE, schedule)
    d.set_option(OPT_ATM_FORCE_SCALED, int(scaled))
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    e, f, st = d.compute()
    _, cnt = d.pass_times()
    d.close()
    return e, f, st, int(cnt[0])


def box(n, density, mix, seed):
    edge = (n / density) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [-0.11, 1.0, 0], [0.06, 0.09, 1.0]]), mix, seed=seed)


@pytest.mark.parametrize("n,density,rc_atm,mix,ext,scaled", [
    (36, 0.1, 20.0, S.MIX_HCNOCU, False, False),   # just below the apex count of the rule
    (37, 0.1, 20.0, S.MIX_HCNOCU, False, False),   # and just at it
    (64, 0.1, 11.0, ONE, False, False),            # lists about 32 long: one and two blocks
    (64, 0.1, 12.6, ONE, False, True),             # and about 64, the short-list rule's line
    (50, 0.1, 17.0, SEVEN, False, False),          # 128 entries: the sort grid changes
    (50, 0.1, 17.0, SEVEN, True, False),           # rows of seven types and references: fewer warps fit
    (150, 0.1, 33.0, S.MIX_HCNOCU, False, False),  # 1,024 entries: the sort grid changes
    (900, 0.02, 21.0, S.MIX_HCNOCU, False, False), # weight-free box
])
def test_blockpair_matches_oracle(n, density, rc_atm, mix, ext, scaled):
    s = box(n, density, mix, seed=n)
    r = oracle.compute(s["pos"], s["Z"], s["cell"], rc=50.0, rc_cn=25.0, rc_atm=rc_atm, extended=ext,
                       atm_force_scaled=scaled, c6_mode=1)
    triplets = oracle.counts(s["pos"], s["cell"], rc=50.0, rc_cn=25.0, rc_atm=rc_atm)[2]
    for schedule in (0, 1):
        e, f, st, visits = evaluate(s, rc_atm, ext, scaled, schedule)
        assert visits == 2 * triplets
        assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
        assert np.abs(f - r["forces"]).max() <= 1e-7
        assert np.abs(st - r["stress"]).max() <= 1e-7


def test_lists_on_both_sides_of_the_capacity():
    """Half lists around 4,096 entries: some apexes by block pairs, the longer ones by rows."""
    s = box(40, 0.1, S.MIX_HCNOCU, seed=5)
    s["pos"] = s["pos"] * [1.0, 1.0, 0.8]  # denser lower part of the cell: uneven lists
    a, b = evaluate(s, 51.0, False, False, 0), evaluate(s, 51.0, False, False, 1)
    assert a[3] == b[3]
    assert abs(a[0] - b[0]) <= 1e-9 * abs(b[0])
    assert np.abs(a[1] - b[1]).max() <= 1e-7 and np.abs(a[2] - b[2]).max() <= 1e-7


@pytest.mark.parametrize("mix,ext", [(ONE, False), (ONE, True), (SEVEN, False), (SEVEN, True)])
def test_weight_free_boxes_of_one_and_many_types(mix, ext):
    """Both ends of the shared-memory rule in weight-free boxes (two CTAs per SM, one, or the
    other schedule)."""
    s = box(700, 0.02, mix, seed=9)
    a, b = evaluate(s, 20.0, ext, False, 0), evaluate(s, 20.0, ext, False, 1)
    r = oracle.compute(s["pos"], s["Z"], s["cell"], rc=50.0, rc_cn=25.0, rc_atm=20.0, extended=ext, c6_mode=1)
    for e, f, st, visits in (a, b):
        assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
        assert np.abs(f - r["forces"]).max() <= 1e-7 and np.abs(st - r["stress"]).max() <= 1e-7
    assert a[3] == b[3]
