"""DFIRE poses whose ANM extents displace atoms beyond what FP32 can settle or even hold (the FP32 error
bound of the culled scorers is then wider than a bin, or infinite), beside atoms that the mask keeps in
place and that do meet: the oracle's energies, FP64 bit for bit.  Odd sizes, so that lists and chunks end
in padding.

Tolerance of mixed: the same FP64 table values (|v| < 6 here) in another order of summation, at most
n * 2^-53 * sum|v| <= 6 n^2 2^-53 for n pairs."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_scores

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
