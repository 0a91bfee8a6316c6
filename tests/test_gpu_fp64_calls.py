"""The culled FP64 scorer in calls whose number of poses selects each of its shapes (few poses: many warps a
pose; many: small CTAs), held to the oracle's bits on some of the poses, and to one another on all."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_scores

pytestmark = pytest.mark.gpu


# 4x6, 6x4, 8x3 and 12x2 warps x CTAs for large calls of these sizes
@pytest.mark.parametrize("n_rec,n_lig", [(90, 60), (757, 481), (1000, 800), (1200, 1400), (3002, 1274)])
def test_every_number_of_poses_gives_the_same_bits(n_rec, n_lig, tables):
    n = 1000
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, 3, 3, seed=n_rec)
    poses = np.array(c.poses.reshape(n, -1))
    poses[::2, :3] *= 0.8
    pick = np.array([0, 1, 2, 147, 148, 295, 296, 443, 591, 887, 998, 999])
    sc, ref = oracle_scores(OracleSystem(c, tables), poses[pick])
    with sd.Docking([c], tables) as dk:
        s_all, e_all = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.array_equal(e_all[pick], ref) and np.array_equal(s_all[pick], sc)
        for k in (1, 148, 149, 296, 297, 444, 592, 640, 888, 960):
            _, e = dk.score_poses(0, poses[:k], sd.SD_PREC_FP64)
            assert np.array_equal(e, e_all[:k]), f"{k} poses"


@pytest.mark.parametrize("n_rec,n_lig", [(1024, 2500), (1025, 2048), (1025, 2049), (2000, 4700)])
def test_large_ligands_of_few_poses(n_rec, n_lig, tables):
    """24 warps a pose from 2,049 ligand and 1,025 receptor atoms on, else 16."""
    c = sd.SyntheticComplex(n_rec, n_lig, 4, 1, 3, 3, seed=n_lig)
    poses = np.array(c.poses.reshape(4, -1))
    poses[:, :3] *= 0.8
    _, ref = oracle_scores(OracleSystem(c, tables), poses)
    with sd.Docking([c], tables) as dk:
        _, e = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.array_equal(e, ref)
