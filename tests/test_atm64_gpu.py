"""FP64 ATM kernel at the edges of its tiles, row lists, type groups and splits, against
the FP64 oracle (the parity bar of the plain form: energy 1e-9 relative, forces and stress
1e-7)."""
import numpy as np
import pytest

import d3_systems as S
import oracle
from d3_b200 import OPT_ATM_CTAS_PER_SM, OPT_ATM_FORCE_SCALED, OPT_ATM_TILE, D3

pytestmark = pytest.mark.gpu

MIX2 = (("H", 0.6), ("O", 0.4))


def box(n, density, seed, mix=S.MIX_HCNOCU):
    edge = (n / density) ** (1.0 / 3.0)
    return S.random_box(n, edge * np.array([[1.0, 0, 0], [0.09, 1.0, 0], [0.05, 0.07, 1.0]]), mix, seed=seed)


@pytest.mark.parametrize("n,density,rc_atm,tile,ctas,ext,scaled", [
    (1, 0.02, 18.0, 0, 0, False, False),      # one atom: only its own images
    (2, 0.05, 25.0, 0, 0, True, False),       # far fewer apexes than CTAs: most splits
    (5, 0.1, 58.0, 0, 0, False, False),       # lists longer than the row list and one tile
    (33, 0.08, 12.0, 0, 4, False, False),     # lists shorter than a warp's 32 partners
    (97, 0.1, 30.0, 128, 0, False, True),     # smallest tile: several per list
    (160, 0.1, 24.0, 256, 2, True, False),
    (700, 0.02, 20.0, 0, 0, False, False),    # weight-free box (heights above 2 rc_ATM)
    (700, 0.02, 20.0, 128, 4, True, False),
])
def test_atm64_matches_oracle(n, density, rc_atm, tile, ctas, ext, scaled):
    s = box(n, density, seed=n, mix=S.MIX_HCNOCU if n > 2 else MIX2)
    d = D3(s["Z"], n, rc=60.0, rc_cn=30.0, rc_atm=rc_atm, table=1 if ext else 0)
    d.set_option(OPT_ATM_TILE, tile)
    d.set_option(OPT_ATM_CTAS_PER_SM, ctas)
    d.set_option(OPT_ATM_FORCE_SCALED, int(scaled))
    d.set_cell(s["cell"])
    d.set_atoms(s["pos"], s["Z"])
    e, f, st = d.compute()
    _, cnt = d.pass_times()
    d.close()
    r = oracle.compute(s["pos"], s["Z"], s["cell"], rc=60.0, rc_cn=30.0, rc_atm=rc_atm, extended=ext,
                       atm_force_scaled=scaled, c6_mode=1)
    triplets = oracle.counts(s["pos"], s["cell"], rc=60.0, rc_cn=30.0, rc_atm=rc_atm)[2]
    assert int(cnt[0]) == 2 * triplets
    assert abs(e - r["energy"]) <= 1e-9 * abs(r["energy"])
    assert np.abs(f - r["forces"]).max() <= 1e-7
    assert np.abs(st - r["stress"]).max() <= 1e-7
