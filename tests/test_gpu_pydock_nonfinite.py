"""pyDock scoring with a charge that is not finite: poses without an atom within the cutoff of it keep finite
energies and gradients, the oracle's.  The ligand lies next to the charge's group of 8 atoms, so that the
charge is listed with it and only the cutoff keeps it out."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_energy, oracle_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("charge", [np.nan, np.inf])
def test_charge_beyond_the_cutoff(charge, tables):
    n = 64
    c = sd.SyntheticComplex(8, 3, n, 1, 0, 0, seed=4)
    rng = np.random.default_rng(1)
    c.rec_xyz[:] = rng.normal(scale=0.5, size=(8, 3))
    c.rec_xyz[0] = (-6.0, 0.0, 0.0)  # the charge, at the far side of its group
    c.lig_xyz[:] = rng.normal(scale=0.2, size=(3, 3))
    c.rec_charge[0] = charge
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] = rng.normal(scale=0.5, size=(n, 3)) + (11.5, 0.0, 0.0)
    osys = OracleSystem(c, tables, scoring=1)
    ref = np.array([oracle_energy(osys, p) for p in poses])
    grad = np.array([oracle_grad(osys, p, 6) for p in poses])
    assert np.isfinite(ref).all() and np.isfinite(grad).all() and np.abs(ref).min() > 1e-6
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    scale = np.maximum(np.abs(ref), top)
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        for precision, etol, gtol in ((sd.SD_PREC_FP64, 1e-10, 1e-10), (sd.SD_PREC_MIXED, 1e-5, 1e-4)):
            _, e = dk.score_poses(0, poses, precision)
            eg, g = dk.pydock_grad(0, poses, precision)
            assert (np.abs(e - ref) / scale).max() <= etol
            assert (np.abs(eg - ref) / scale).max() <= etol
            assert (np.abs(g - grad) / top[:, None]).max() <= gtol
        poses[:, 0] -= 8.0  # within the cutoff of the charge
        for precision in (sd.SD_PREC_FP64, sd.SD_PREC_MIXED):
            _, e = dk.score_poses(0, poses, precision)
            assert not np.isfinite(e).any()
