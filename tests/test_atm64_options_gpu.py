"""FP64 row kernel at every number of CTAs per SM that can be asked for, with one and with the
most element types a handle takes, against the FP64 oracle (bar of the plain form)."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_ATM_CTAS_PER_SM, OPT_ATM_SCHEDULE, OPT_ATM_TILE, D3

pytestmark = pytest.mark.gpu

RC = dict(rc=40.0, rc_cn=25.0, rc_atm=22.0)


@pytest.mark.parametrize("ext", [False, True])
@pytest.mark.parametrize("types", [1, 32])
def test_ctas_per_sm(types, ext):
    edge = (70 / 0.1) ** (1.0 / 3.0)
    s = S.random_box(70, edge * np.array([[1.0, 0, 0], [0.1, 1.0, 0], [0.05, -0.1, 1.0]]), (("C", 1.0),), seed=8)
    s["Z"] = np.resize(np.arange(1, 2 * types, 2), 70) if types > 1 else s["Z"]
    r = oracle.compute(s["pos"], s["Z"], s["cell"], extended=ext, c6_mode=1, **RC)
    d = D3(s["Z"], 70, table=1 if ext else 0, **RC)
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    d.set_option(OPT_ATM_SCHEDULE, 1)
    for ctas in (0, 1, 2, 3, 4, 5, 6, 7, 8, 50):
        for tile in (0, 32):
            d.set_option(OPT_ATM_CTAS_PER_SM, ctas)
            d.set_option(OPT_ATM_TILE, tile)
            e, f, st = d.compute()
            assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
            assert np.abs(f - r["forces"]).max() <= 1e-7
            assert np.abs(st - r["stress"]).max() <= 1e-7
    d.close()
