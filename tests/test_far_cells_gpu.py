"""Atoms given many cells away from the origin: the reference's image box still cuts pairs
within rc_ATM between atoms of different cells, and moving every atom by the same number of
cells changes nothing. Against the FP64 oracle on the structure at the origin, at the parity
bars of the two forms."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_PRECISION, D3

pytestmark = pytest.mark.gpu

RC = dict(rc=60.0, rc_cn=30.0, rc_atm=28.0)


def scattered():
    edge = (40 / 0.09) ** (1.0 / 3.0)
    s = S.random_box(40, edge * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [-0.2, 0.15, 1.0]]), seed=4)
    cells = np.random.default_rng(5).integers(-3, 4, s["pos"].shape)
    return s, s["pos"] + cells @ s["cell"]


# positions of 1e4 (1e6) cells carry 2e-11 (2e-9) A of rounding, against forces that vary by
# well under 1 eV/A^2: below the bars
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("cells", [(0, 0, 0), (15990, 0, 0), (20000, 20000, 20000), (-20000, 0, 16001), (0, 999990, -999990)])
def test_image_box_cuts_far_from_the_origin(cells, precision):
    s, pos = scattered()
    d = D3(s["Z"], len(s["Z"]), **RC)
    d.set_option(OPT_PRECISION, precision)
    d.set_cell(s["cell"])
    d.set_atoms(pos + np.array(cells) @ s["cell"], s["Z"])
    e, f, st = d.compute()
    _, cnt = d.pass_times()
    d.close()
    r = oracle.compute(pos, s["Z"], s["cell"], c6_mode=1, **RC)
    triplets = oracle.counts(pos, s["cell"], **RC)[2]
    e_rel, f_abs, s_abs = (1e-6, 1e-4, 1e-6) if precision else (1e-9, 1e-7, 1e-7)
    assert abs(e - r["energy"]) <= e_rel * abs(r["energy"])
    assert np.abs(f - r["forces"]).max() <= f_abs
    assert np.abs(st - r["stress"]).max() <= s_abs
    assert abs(int(cnt[0]) - 2 * triplets) <= (2 * triplets * 1e-5 if precision else 0)
