"""Groups of receptor atoms of which one is displaced far by its ANM extent: the bounding box of such a
group is large, and its FP32 centre and extent are rounded by more than the margin of the box test.  The
ligand atom sits just inside the cutoff of an atom at the near side of the box, so a box that is too small
loses the pair.  Against the oracle: DFIRE FP64 bit for bit and mixed to rounding (8 values), pyDock within
1e-10 (FP64) of the larger of 1 and the largest energy."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_scores
from pydock_util import oracle_energy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [1e2, 3e3, 1e5, 1e6, 7e6])
def test_pair_at_the_near_side_of_a_large_box(extent, tables):
    n = 600
    c = sd.SyntheticComplex(8, 1, n, 1, 1, 0, seed=2)
    rng = np.random.default_rng(int(extent))
    c.rec_xyz[:] = rng.normal(scale=2e-4, size=(8, 3))  # the box ends at the atoms that do not move
    c.lig_xyz[:] = 0.0
    c.rec_mask[:], c.lig_mask[:] = 0, 0
    c.rec_mask[5] = 1
    c.rec_modes[0] = 0.0
    c.rec_modes[0, 5] = (1.0, 0.7, 0.9)
    poses = np.array(c.poses.reshape(n, -1))
    d = -np.abs(rng.normal(size=(n, 3)))  # the box opens away from the ligand atom on each axis
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    at = np.array(c.rec_xyz)[rng.choice([0, 1, 2, 3, 4, 6, 7], size=n)]
    poses[:, :3] = at + d * (15.0 - rng.uniform(0.0, 0.05, size=(n, 1)) ** 2)
    poses[:, 7] = extent * rng.uniform(0.5, 1.0, size=n)
    _, ref = oracle_scores(OracleSystem(c, tables), poses)
    assert (ref != 0.0).mean() > 0.9
    with sd.Docking([c], tables) as dk:
        _, en = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.array_equal(en, ref)
        _, en = dk.score_poses(0, poses, sd.SD_PREC_MIXED)
        assert np.abs(en - ref).max() <= 1e-12
    osys = OracleSystem(c, tables, scoring=1)
    poses[:, :3] = at + d * 14.97  # inside the electrostatics' switch
    ref = np.array([oracle_energy(osys, p) for p in poses])
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        _, en = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.abs(en - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
        eg, _ = dk.pydock_grad(0, poses, sd.SD_PREC_FP64)
        assert np.abs(eg - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
