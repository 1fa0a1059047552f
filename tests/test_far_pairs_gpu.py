"""Pairs hundreds of bohr apart in the FP32 form: the force of a pair keeps FP32 accuracy out
to the cutoff (powers of the distance up to r^-16 would leave the FP32 range)."""
import numpy as np
import pytest

from d3_b200 import OPT_PRECISION, D3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("damping", [0, 1])
@pytest.mark.parametrize("r", [40.0, 320.0, 900.0, 1800.0])
def test_pair_force_in_fp32_matches_fp64(r, damping):
    cell = np.eye(3) * 4000.0 * 0.52917726  # no image within the cutoff
    axis = np.array([1.0, 0.02, -0.03])
    a = np.array([10.0, 20.0, 30.0])
    pos = np.array([a, a + axis / np.linalg.norm(axis) * r * 0.52917726])
    out = []
    for precision in (0, 1):
        d = D3([29, 79], 2, rc=1.1 * r + 16.0, rc_cn=20.0, damping=damping)
        d.set_option(OPT_PRECISION, precision)
        d.set_cell(cell)
        d.set_atoms(pos, [29, 79])
        d.compute()
        t = d.pass_terms()
        out.append((t[:, 0], t[:, 2:5]))
        d.close()
    (e0, f0), (e1, f1) = out
    # FP32: both positions (below r + 60 bohr) round by 2^-24 relative and the force varies as
    # r^-7; about 30 roundings of 6e-8 on top
    tol = 7 * 2 * (r + 60.0) * 2.0 ** -24 / r + 2e-6
    assert np.abs(e1 - e0).max() <= tol * np.abs(e0).max()
    assert np.abs(f1 - f0).max() <= tol * np.abs(f0).max()
