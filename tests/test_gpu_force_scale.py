"""FP32 gradients with charges or LJ radii far from the ordinary: the sums of the ligand's forces must not lose
digits to a unit that fits the largest force that could occur.  Parameters that no atom has, a radius close to
0 that some atoms have, and a huge charge that no pose comes near, against the oracle (1e-4 of the largest
component, as for ordinary parameters).  The oracle's gradient stays finite in all of them."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["unused radius", "unused depth", "small radius", "far charge", "large charges"])
@pytest.mark.parametrize("n", [6, 200])
def test_gradients_keep_their_digits(what, n, tables):
    c = sd.SyntheticComplex(700, 90, n, 1, 2, 2, seed=12)
    eps, sigma = np.array(tables[1]), np.array(tables[2])
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] *= 0.8
    if what.startswith("unused"):
        c.rec_lj[:] = np.where(c.rec_lj == 7, 8, c.rec_lj)
        c.lig_lj[:] = np.where(c.lig_lj == 7, 8, c.lig_lj)
        eps[7], sigma[7] = (0.1, 1e-9) if what == "unused radius" else (-1.0, 3.0)
    elif what == "small radius":
        sigma[7] = 1e-7
    elif what == "far charge":
        c.rec_xyz[5] = (0.0, 0.0, 5000.0)
        c.rec_charge[5] = 1e20
    else:
        c.rec_charge[:] *= 3e3
        c.lig_charge[:] *= 1e-3
        c.lig_charge[4] = 1e3
    t = (tables[0], eps, sigma)
    osys = OracleSystem(c, t, scoring=1)
    grad = np.array([oracle_grad(osys, p, 10) for p in poses])
    assert np.isfinite(grad).all()
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    with sd.Docking([c], t, scoring=sd.SD_SCORING_PYDOCK) as dk:
        _, g = dk.pydock_grad(0, poses, sd.SD_PREC_MIXED)
    assert (np.abs(g - grad) / top[:, None]).max() <= 1e-4
