"""DFIRE poses whose ANM extents displace atoms beyond what FP32 can settle or even hold (the FP32 error
bound of the culled scorers is then wider than a bin, or infinite), beside atoms that the mask keeps in
place and that do meet: the oracle's energies, FP64 bit for bit.  Odd sizes, so that lists and chunks end
in padding.

Tolerance of mixed: the same FP64 table values (|v| < 6 here) in another order of summation, at most
n * 2^-53 * sum|v| <= 6 n^2 2^-53 for n pairs."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_bins, oracle_scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [1e4, 3e5, 1e6, 1e19, 1e37, 1e39, 1e150])
@pytest.mark.parametrize("n_rec,n_lig", [(9, 33), (70, 65), (700, 97)])
def test_displacements_beyond_fp32(n_rec, n_lig, extent, tables):
    n = 24
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, n_modes_rec=2, n_modes_lig=3, seed=n_rec)
    c.rec_mask[:], c.lig_mask[:] = np.arange(n_rec) % 3 == 0, np.arange(n_lig) % 2 == 0
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] *= 0.2  # overlapping
    poses[:, 7:] = 0.0
    poses[0::3, 7] = extent   # receptor displaced
    poses[1::3, 9] = extent   # ligand displaced
    poses[2::3, 7:] = extent  # both
    _, ref = oracle_scores(OracleSystem(c, tables), poses)
    assert (ref != 0.0).all()
    tol = 6.0 * (n_rec * n_lig) ** 2 * 2.0 ** -53 + 1e-12
    assert np.abs(tables[0]).max() < 6.0
    with sd.Docking([c], tables) as dk:
        for k in (n, 5):
            _, en = dk.score_poses(0, poses[:k], sd.SD_PREC_FP64)
            assert np.array_equal(en, ref[:k])
            _, en = dk.score_poses(0, poses[:k], sd.SD_PREC_MIXED)
            assert np.abs(en - ref[:k]).max() <= tol


@pytest.mark.parametrize("extent", [0.0, 3.0, 1e4, 3e5, 1e6, 1e37, 1e39])
def test_atoms_displaced_together(extent, tables):
    """Receptor and ligand atoms displaced by the same vector, beyond what FP32 holds from 1e39 on: they meet
    there, and the bins of the pairs, by the steps of each precision's scorer, are the oracle's."""
    c = sd.SyntheticComplex(70, 41, 1, 1, n_modes_rec=1, n_modes_lig=1, seed=8)
    c.rec_mask[:], c.lig_mask[:] = np.arange(70) % 2 == 0, np.arange(41) % 3 == 0
    c.rec_modes[:], c.lig_modes[:] = (1.0, 0.0, 0.0), (1.0, 0.0, 0.0)
    pose = np.zeros(c.pose_len)
    pose[:3], pose[3], pose[7:] = (2.0, -1.0, 0.5), 1.0, extent
    osys = OracleSystem(c, tables)
    want, _, _, _, _ = oracle_bins(osys, pose)
    both = np.ix_(c.rec_mask == 1, c.lig_mask == 1)
    assert (want[both] >= 0).any()
    _, ref = oracle_scores(osys, pose[None])
    with sd.Docking([c], tables) as dk:
        for precision in (sd.SD_PREC_FP64_REF, sd.SD_PREC_FP64, sd.SD_PREC_MIXED):
            assert np.array_equal(dk.dfire_bins(0, pose, precision), want)
        _, en = dk.score_poses(0, pose[None], sd.SD_PREC_FP64)
        assert np.array_equal(en, ref)
        _, en = dk.score_poses(0, pose[None], sd.SD_PREC_MIXED)
        assert np.abs(en - ref).max() <= 6.0 * want.size ** 2 * 2.0 ** -53
