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
