"""Which FP64 ATM kernel takes a call (block pairs add one launch to an evaluation, so the
launch count tells), lists on both sides of the block pairs' capacity, and weight-free and
weighted structures in one launch."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_ATM_SCHEDULE, D3, D3Batch

BOHR = 0.52917726
ONE = (("C", 1.0),)


def box(n, density, mix=S.MIX_HCNOCU, seed=5):
    edge = (n / density) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [-0.11, 1.0, 0], [0.06, 0.09, 1.0]]), mix, seed=seed)


def uneven():
    s = box(40, 0.1)
    return dict(s, pos=s["pos"] * [1.0, 1.0, 0.8])  # denser lower part of the cell


def half_list_lengths(s, rc_atm):
    """Entries before each atom within rc_atm (bohr): by height along the third lattice vector
    (T_z, then the fractional coordinate), images of the atom itself by T_y, T_x."""
    pos, cell = s["pos"] / BOHR, s["cell"] / BOHR
    frac = pos @ np.linalg.inv(cell)
    frac -= np.floor(frac)
    x = frac @ cell
    reach = np.ceil(rc_atm * np.linalg.norm(np.linalg.inv(cell), axis=0)).astype(int) + 1
    T = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in reach], indexing="ij"), -1).reshape(-1, 3)
    out = []
    for a in range(len(x)):
        d2 = ((x[None, :, :] + (T @ cell)[:, None, :] - x[a]) ** 2).sum(-1)
        low = T[:, 2][:, None] + frac[None, :, 2] < frac[a, 2]
        low[:, a] = (T[:, 2] < 0) | ((T[:, 2] == 0) & ((T[:, 1] < 0) | ((T[:, 1] == 0) & (T[:, 0] < 0))))
        out.append(int(((d2 <= rc_atm ** 2) & low).sum()))
    return np.array(out)


def test_uneven_lists_lie_on_both_sides_of_the_capacity():
    m = half_list_lengths(uneven(), 51.0)
    assert (m > 4096).sum() >= 8 and (m <= 4096).sum() >= 8


def blocks(d):
    d.set_option(OPT_ATM_SCHEDULE, 1)
    rows_only = d.launches_per_eval()
    d.set_option(OPT_ATM_SCHEDULE, 0)
    return d.launches_per_eval() - rows_only


@pytest.mark.gpu
@pytest.mark.parametrize("n,density,rc_atm,mix,table,want", [
    (36, 0.1, 20.0, S.MIX_HCNOCU, 0, 0),   # fewer apexes than a quarter of the 148 SMs
    (37, 0.1, 20.0, S.MIX_HCNOCU, 0, 1),
    (64, 0.1, 11.3, ONE, 0, 0),            # 45 entries expected per list, the rule's line is 48
    (64, 0.1, 11.8, ONE, 0, 1),            # 51
    (40, 0.1, 51.0, S.MIX_HCNOCU, 0, 1),
    (700, 0.02, 20.0, S.MIX_HCNOCU, 0, 1), # weight-free
])
def test_rule_of_the_block_pairs(n, density, rc_atm, mix, table, want):
    s = box(n, density, mix)
    d = D3(s["Z"], n, rc=60.0, rc_cn=25.0, rc_atm=rc_atm, table=table)
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    assert blocks(d) == want
    d.close()


# rows of (2 NR + 2) doubles per type for 32 partners and warp: 10 warps fit six types of the
# 5-reference table or five of the other (weighted structures 10 and 9)
@pytest.mark.gpu
@pytest.mark.parametrize("table,most", [(0, 6), (1, 5)])
@pytest.mark.parametrize("density", [0.02, 0.1])  # weight-free and weighted
def test_rule_of_the_warps(table, most, density):
    elements = [1, 6, 7, 8, 29, 14, 26]
    for types in (most, most + 1):
        s = box(600, density, ONE)
        s["Z"] = np.resize(elements[:types], 600)
        rc = dict(rc=50.0, rc_cn=25.0, rc_atm=20.0)
        d = D3(s["Z"], 600, table=table, **rc)
        d.set_cell(s["cell"])
        d.set_atoms(s["pos"], s["Z"])
        assert blocks(d) == (1 if types == most else 0)
        e, f, st = d.compute()
        d.close()
        r = oracle.compute(s["pos"], s["Z"], s["cell"], c6_mode=1, extended=bool(table), **rc)
        assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
        assert np.abs(f - r["forces"]).max() <= 1e-7
        assert np.abs(st - r["stress"]).max() <= 1e-7


@pytest.mark.gpu
@pytest.mark.parametrize("order", [(0, 1, 0), (1, 0, 1)])
def test_both_kinds_in_one_batch(order):
    """Structures with cells longer and shorter than 2 rc_ATM in one evaluation: two
    launches of the block-pair kernel, each taking its own apexes."""
    rc = dict(rc=50.0, rc_cn=25.0, rc_atm=17.0)
    kinds = [box(120, 0.02, seed=3), box(60, 0.1, seed=4)]  # edges 34 and 16 bohr
    parts = [kinds[k] for k in order]
    b = D3Batch(sorted({int(z) for s in parts for z in s["Z"]}), 3, 400, **rc)
    b.set_structures(parts)
    assert blocks(b) == 1
    e, f, st = b.compute()
    visits = int(b.pass_times()[1][0])
    b.close()
    want = 0
    for k, s in enumerate(parts):
        r = oracle.compute(s["pos"], s["Z"], s["cell"], c6_mode=1, **rc)
        want += 2 * oracle.counts(s["pos"], s["cell"], **rc)[2]
        assert abs(e[k] - r["energy"]) <= 1e-9 * abs(r["energy"])
        assert np.abs(f[k] - r["forces"]).max() <= 1e-7
        assert np.abs(st[k] - r["stress"]).max() <= 1e-7
    assert visits == want
