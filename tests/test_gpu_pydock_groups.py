"""The pyDock scorer and adjoint at the edges of their groups (8 receptor atoms), tiles and chunks (32
atoms) and candidate lists (128 places, so dense overlapping poses refill them), against the oracle.

Tolerances: FP64 as in test_gpu_pydock.py (1e-10 of the value); FP32 gradients within 1e-4 of their
largest component, and FP32 energies within 1e-5 of the larger of the energy and that component (a
coordinate rounded at 30 A moves by 2e-6 A, and an energy by that times its gradient)."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_energy, oracle_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rec,n_lig,modes", [(1, 1, 0), (7, 33, 10), (8, 31, 3), (9, 32, 10), (33, 97, 1),
                                               (65, 700, 10), (200, 161, 10)])
def test_groups_and_lists(n_rec, n_lig, modes, tables):
    n = 9
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, n_modes_rec=modes, n_modes_lig=modes, seed=n_rec + 7 * n_lig)
    poses = np.array(c.poses.reshape(n, -1))
    poses[::3, :3] *= 0.05  # overlapping: whole molecules inside the cutoff
    poses[1::3, :3] *= 0.6
    osys = OracleSystem(c, tables, scoring=1)
    ref = np.array([oracle_energy(osys, p) for p in poses])
    grad = np.array([oracle_grad(osys, p, 6 + 2 * modes) for p in poses])
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        for prec, etol, gtol in ((sd.SD_PREC_FP64, 1e-10, 1e-10), (sd.SD_PREC_MIXED, 1e-5, 1e-4)):
            _, e = dk.score_poses(0, poses, prec)
            eg, g = dk.pydock_grad(0, poses, prec)
            scale = np.maximum(np.abs(ref), top)
            assert (np.abs(e - ref) / scale).max() <= etol
            assert (np.abs(eg - ref) / scale).max() <= etol
            assert (np.abs(g - grad) / top[:, None]).max() <= gtol
