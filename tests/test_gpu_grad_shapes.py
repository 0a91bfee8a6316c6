"""FP32 gradients at the sizes where their kernel's shape changes (4, 8 or 12 warps per CTA, by what fits on an
SM beside a pose's arrays), in a context of their own and beside a larger complex, against the oracle: 1e-4 of
the largest component, energies 1e-5 of the larger of energy and component."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_energy, oracle_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rec,n_lig", [(5, 3), (60, 40), (300, 512), (300, 544), (300, 576), (300, 608), (500, 1216),
                                         (500, 1280), (500, 1312), (500, 1344), (400, 1984), (400, 2048), (400, 2240),
                                         (400, 2336), (400, 4800), (400, 4900)])
@pytest.mark.parametrize("beside", [False, True])
def test_shapes(n_rec, n_lig, beside, tables):
    n = 200  # above one pose per SM
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, 2, 3, seed=n_rec + n_lig)
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] *= 0.7
    pick = [0, 1, 77, 199]
    osys = OracleSystem(c, tables, scoring=1)
    ref = np.array([oracle_energy(osys, poses[k]) for k in pick])
    grad = np.array([oracle_grad(osys, poses[k], 11) for k in pick])
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    others = [sd.SyntheticComplex(900, 3000, 1, 1, 0, 0, seed=1)] if beside else []
    with sd.Docking(others + [c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        for _ in range(2):
            e, g = dk.pydock_grad(len(others), poses, sd.SD_PREC_MIXED)
            assert (np.abs(g[pick] - grad) / top[:, None]).max() <= 1e-4
            assert (np.abs(e[pick] - ref) / np.maximum(np.abs(ref), top)).max() <= 1e-5
            if beside:  # between calls on the other complex
                o = others[0].poses.reshape(1, -1)
                dk.pydock_grad(0, np.repeat(o, n, axis=0), sd.SD_PREC_MIXED)


@pytest.mark.parametrize("n_rec,n_lig", [(50, 1472), (50, 1536), (700, 1504), (47, 3456), (47, 3503), (47, 3560)])
@pytest.mark.parametrize("n", [148, 149, 400])
def test_fp64_beside_one_cta(n_rec, n_lig, n, tables):
    """FP64 gradients where an SM's shared memory holds two CTAs' arrays, one, or none."""
    c = sd.SyntheticComplex(n_rec, n_lig, n, 1, 2, 3, seed=n_rec + n_lig)
    poses = np.array(c.poses.reshape(n, -1))
    poses[:, :3] *= 0.7
    pick = [0, 77, n - 1]
    osys = OracleSystem(c, tables, scoring=1)
    ref = np.array([oracle_energy(osys, poses[k]) for k in pick])
    grad = np.array([oracle_grad(osys, poses[k], 11) for k in pick])
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    with sd.Docking([c], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        e, g = dk.pydock_grad(0, poses, sd.SD_PREC_FP64)
        assert (np.abs(g[pick] - grad) / top[:, None]).max() <= 1e-10
        assert (np.abs(e[pick] - ref) / np.maximum(np.abs(ref), top)).max() <= 1e-10
