"""Clustering at its limit of 4 A: translations that put the backbone RMSD of pairs exactly at, and a few
rounding errors on either side of, the limit, beside clear ones; equal to the oracle, whose sums are in
the reference's order."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem, oracle_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_lig,every", [(40, 1), (33, 8), (700, 1), (2000, 3)])
def test_rmsd_at_the_limit(n_lig, every, tables):
    G = 40
    cx = sd.SyntheticComplex(50, n_lig, 3, G, 0, 0, seed=n_lig)
    rng = np.random.default_rng(5)
    poses = np.array(cx.poses)
    poses[:, :, 3:7] = poses[:, :1, 3:7]  # one orientation per swarm: an RMSD is a distance of translations
    for s in range(3):
        for g in range(1, G):
            d = rng.normal(size=3) if s else np.array([1.0, 0.0, 0.0])
            r = 4.0 * rng.integers(1, 3) * (1.0 + rng.integers(-3, 4) * [0.0, 2.0 ** -52, 2.0 ** -45][s])
            poses[s, g, :3] = poses[s, rng.integers(0, g), :3] + d / np.linalg.norm(d) * r
    rb = np.zeros(cx.n_rec, np.int32)  # receptor atoms do not move, so only ligand atoms are flagged
    lb = (np.arange(n_lig) % every == 0).astype(np.int32)
    with sd.Docking([cx], tables, precision=sd.SD_PREC_FP64) as dk:
        dk.init_state(0, poses)
        st = dk.get_state(0)
        st.scoring[:] = rng.normal(size=st.scoring.shape)
        dk.set_state(0, st)
        got = dk.cluster(0, rb, lb)
    ref = oracle_cluster(OracleSystem(cx, tables), poses, st.scoring, rb, lb)
    assert np.array_equal(got["n_clusters"], ref["n_clusters"]) and np.array_equal(got["member"], ref["member"])
    for s, n in enumerate(ref["n_clusters"]):
        assert np.array_equal(got["rep"][s, :n], ref["rep"][s, :n])
        assert np.array_equal(got["size"][s, :n], ref["size"][s, :n])


@pytest.mark.parametrize("n_swarms,glowworms,modes", [(1, 1, 10), (1, 3, 0), (3, 21, 7), (2, 130, 10)])
def test_ragged_swarms(n_swarms, glowworms, modes, tables):
    """Final poses in batches over swarm boundaries, the last one short; receptor and ligand atoms."""
    cx = sd.SyntheticComplex(100, 70, n_swarms, glowworms, modes, modes, seed=glowworms)
    rng = np.random.default_rng(glowworms)
    poses = np.array(cx.poses)
    poses[:, :, :3] = poses[:, :1, :3] + rng.normal(size=poses[:, :, :3].shape)  # some pairs within 4 A
    rb, lb = (np.arange(100) % 3 == 0).astype(np.int32), (np.arange(70) % 2 == 0).astype(np.int32)
    with sd.Docking([cx], tables, precision=sd.SD_PREC_FP64) as dk:
        dk.init_state(0, poses)
        st = dk.get_state(0)
        st.scoring[:] = rng.normal(size=st.scoring.shape)
        dk.set_state(0, st)
        got = dk.cluster(0, rb, lb)
    ref = oracle_cluster(OracleSystem(cx, tables), poses, st.scoring, rb, lb)
    assert np.array_equal(got["n_clusters"], ref["n_clusters"]) and np.array_equal(got["member"], ref["member"])
