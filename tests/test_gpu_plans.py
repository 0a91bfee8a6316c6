"""Launch plans of a context that scores by more than one kernel shape.  A call of at most one pose per
SM on a receptor of more than 640 atoms takes a CTA of more warps than a larger call, so each needs its
own grid and shared memory, in whichever order the calls come and at every precision.

Tolerances: FP64 1e-10 and FP32 1e-5, of the larger of the energy and its gradient's largest component (a
coordinate rounded to FP32 at 30 A moves by 2e-6 A, and an energy by that times its gradient)."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_energy, oracle_grad

pytestmark = pytest.mark.gpu
N_REC, N_LIG, MANY, FEW = 700, 90, 400, 20


@pytest.mark.parametrize("precision,tol", [(sd.SD_PREC_FP64_REF, 1e-10), (sd.SD_PREC_FP64, 1e-10),
                                           (sd.SD_PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("first", ["many", "few", "step"])
def test_pydock_calls_of_both_shapes(first, precision, tol, tables):
    c = sd.SyntheticComplex(N_REC, N_LIG, MANY // 20, 20, 3, 3, seed=5)
    poses = np.array(c.poses.reshape(MANY, -1))
    poses[:, :3] *= 0.7  # closer, so that every energy counts
    osys = OracleSystem(c, tables, scoring=1)
    ref = np.array([oracle_energy(osys, p) for p in poses])
    top = np.array([np.abs(oracle_grad(osys, p, 12)).max() for p in poses])
    scale = np.maximum(np.maximum(np.abs(ref), top), 1.0)
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK, precision=precision) as dk:
        if first == "step":
            dk.init_state(0, poses.reshape(c.poses.shape))
            dk.set_draws(0, sd.gso_draws(1, c.n_swarms, 1, c.n_glowworms))
            dk.step(1)
            assert (np.abs(-dk.get_state(0).scoring.ravel() - ref) / scale).max() <= tol
        for n in (MANY, FEW, MANY, FEW) if first != "few" else (FEW, MANY, FEW):
            _, e = dk.score_poses(0, poses[:n], precision)
            assert (np.abs(e - ref[:n]) / scale[:n]).max() <= tol, f"{n} poses"


@pytest.mark.parametrize("n", [1, 40, 5000])
def test_results_of_repeated_calls(n, tables):
    """Scores and energies, energies and gradients come to the host in one copy where they are small, through
    pinned memory from the 16th call of a context on, and one by one where they are not (5,000 poses)."""
    c = sd.SyntheticComplex(120, 60, n, 1, 10, 10, seed=3)
    poses = c.poses.reshape(n, -1)
    with sd.Docking([c], tables) as dk:
        sc, en = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        assert np.array_equal(sc, -(0.0157 * en - 4.7)) and np.unique(en).size > n // 2
        for _ in range(18):
            s, e = dk.score_poses(0, poses, sd.SD_PREC_FP64)
            assert np.array_equal(s, sc) and np.array_equal(e, en)
    osys = OracleSystem(c, tables, scoring=1)
    pick = np.unique([0, n // 2, n - 1])
    ref = np.array([oracle_energy(osys, poses[k]) for k in pick])
    grad = np.array([oracle_grad(osys, poses[k], 26) for k in pick])
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        for _ in range(18):
            e, g = dk.pydock_grad(0, poses, sd.SD_PREC_FP64)
            assert (np.abs(e[pick] - ref) / np.maximum(np.abs(ref), top)).max() <= 1e-10
            assert (np.abs(g[pick] - grad) / top[:, None]).max() <= 1e-10
