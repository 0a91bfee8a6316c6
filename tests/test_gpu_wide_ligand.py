"""Mixed DFIRE scoring of ligands whose atoms lie far from the ligand frame's origin: the FP32 error bound,
and with it the window around a bin's edge in which a pair is decided in FP64, grows with that distance, so
tiles meet more such pairs than a warp can note.  Each of them is decided by itself: the oracle's energies,
and no more FP64 decisions than there are pairs within 15.1 A (the cutoff and every window beyond it).

Tolerance: the same FP64 table values (|v| < 6 here) in another order of summation, at most
n * 2^-53 * sum|v| <= 6 n^2 2^-53 for n pairs."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_scores

pytestmark = pytest.mark.gpu


def rotations(q):
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]]).transpose(2, 0, 1)


def far_complex(n_rec, n_lig, n, offset):
    """Rigid molecules, the ligand moved by offset along x in its frame and each pose moved back; the poses
    overlap.  Returns the complex, the poses and the pairs within 15.1 A of each."""
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, 0, 0, seed=n_rec + n_lig)
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] *= 0.3
    R = rotations(poses[:, 3:7])
    c.lig_xyz[:, 0] += offset
    poses[:, :3] -= offset * R[:, :, 0]
    close = []
    for p, r in zip(poses, R):
        lig = np.array(c.lig_xyz) @ r.T + p[:3]
        d2 = (np.array(c.rec_xyz)[:, None, 0] - lig[None, :, 0]) ** 2
        for k in (1, 2):
            d2 += (np.array(c.rec_xyz)[:, None, k] - lig[None, :, k]) ** 2
        close.append(int((d2 <= 15.1 ** 2).sum()))
    return c, poses, np.array(close)


def tolerance(pairs):
    return 6.0 * pairs.max() ** 2 * 2.0 ** -53 + 1e-12


@pytest.mark.parametrize("offset", [60.0, 500.0, 4000.0, 16000.0])
@pytest.mark.parametrize("variant", range(sd.mixed_variant_count()))
def test_far_ligand_pairs_are_decided_one_by_one(variant, offset, tables, monkeypatch):
    monkeypatch.setenv("SPARKLE_MIXED_VARIANT", str(variant))
    n = 400
    c, poses, close = far_complex(757, 481, n, offset)
    sc, ref = oracle_scores(OracleSystem(c, tables), poses)
    with sd.Docking([c], tables) as dk:
        dk.init_state(0, poses.reshape(c.poses.shape))
        dk.set_draws(0, sd.gso_draws(1, n, 1, 1))
        dk.step(1)
        assert dk.tuning()["variant"] == variant
        assert np.abs(dk.get_state(0).scoring.ravel() - sc).max() <= 0.0157 * tolerance(close) + 1e-12
        done = dk.stats()["pairs_fallback"]
        assert 0 < done <= close.sum()
        for k in (20, n):  # at most one pose per SM, and more
            _, en = dk.score_poses(0, poses[:k])
            assert np.abs(en - ref[:k]).max() <= tolerance(close)
            now = dk.stats()["pairs_fallback"]
            assert now - done <= close[:k].sum()
            done = now


def test_far_ligand_beyond_shared_memory(tables):
    n = 3
    c, poses, close = far_complex(70, 13000, n, 2000.0)
    _, ref = oracle_scores(OracleSystem(c, tables), poses)
    with sd.Docking([c], tables) as dk:
        _, en = dk.score_poses(0, poses)
        assert np.abs(en - ref).max() <= tolerance(close)
        assert 0 < dk.stats()["pairs_fallback"] <= close.sum()
