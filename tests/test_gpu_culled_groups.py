"""The culled DFIRE scorers at the edges of their groups (8 receptor atoms), tiles and chunks (32
atoms), candidate lists (so dense overlapping poses refill them), two-pose batches and kernel shapes,
against the oracle: FP64 bit for bit, mixed within a tolerance.

Tolerance of mixed: both sides add the same FP64 table values (|v| < 6 here) in different orders, so they
differ by at most n * 2^-53 * sum|v| <= 6 n^2 2^-53 for n pairs; a wrong bin moves an energy by a
difference of N(0,1) values."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rec,n_lig", [(1, 1), (7, 33), (8, 31), (9, 32), (33, 97), (65, 700), (200, 161)])
@pytest.mark.parametrize("modes", [0, 3, 10])
def test_groups_lists_and_pose_pairs(n_rec, n_lig, modes, tables):
    n = 1501  # above two rounds of the largest grid: pose pairs first, then single poses, odd
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, n_modes_rec=modes, n_modes_lig=modes, seed=n_rec + 7 * n_lig)
    poses = np.array(c.poses.reshape(n, -1))
    poses[::3, :3] *= 0.05  # overlapping: whole molecules inside the cutoff
    poses[1::7, :3] *= 0.6
    _, ref = oracle_scores(OracleSystem(c, tables), poses)
    tol = 6.0 * (n_rec * n_lig) ** 2 * 2.0 ** -53 + 1e-12
    assert tol < 1e-4 and np.abs(tables[0]).max() < 6.0
    with sd.Docking([c], tables) as dk:
        for k in (n, 5):
            _, en = dk.score_poses(0, poses[:k], sd.SD_PREC_MIXED)
            assert np.abs(en - ref[:k]).max() <= tol
            _, en = dk.score_poses(0, poses[:k], sd.SD_PREC_FP64)
            assert np.array_equal(en, ref[:k])


@pytest.mark.parametrize("n_rec,n_lig", [(6001, 1766), (15999, 333), (17307, 1125), (21500, 500)])
def test_fp64_kernel_shapes(n_rec, n_lig, tables):
    """Receptors whose partial sums leave room for one CTA of 24, 16 or 8 warps per SM."""
    c = sd.SyntheticComplex(n_rec, n_lig, 4, 1, seed=n_rec)
    poses = c.poses.reshape(4, -1)
    sc, ref = oracle_scores(OracleSystem(c, tables), poses)
    with sd.Docking([c], tables) as dk:
        got, en = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.array_equal(en, ref) and np.array_equal(got, sc)
