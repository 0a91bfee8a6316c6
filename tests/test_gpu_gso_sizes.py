"""The GSO update at the edges of its shapes (a warp per glowworm up to 512 glowworms, a thread above;
words of 32 neighbours): every state field bit-identical to the oracle, with many neighbours per
glowworm (a vision range of 30 A), draws of 0 and near 1, identical poses and unequal mode counts."""
import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleState, OracleSystem, oracle_step

pytestmark = pytest.mark.gpu
FIELDS = (("pos", "pos"), ("scoring", "scoring"), ("luciferin", "luciferin"), ("vision_range", "vision"),
          ("step", "step"), ("moved", "moved"), ("nnei_len", "nnei"), ("select", "select"),
          ("ligand_reference_pose", "ref"))


@pytest.mark.parametrize("G,modes", [(1, (10, 10)), (2, (0, 3)), (31, (10, 0)), (32, (1, 1)), (33, (10, 10)),
                                     (200, (10, 10)), (511, (5, 10)), (512, (10, 10)), (513, (10, 10))])
def test_swarm_sizes(G, modes, tables):
    steps = 3
    cx = sd.SyntheticComplex(60, 40, 3, G, *modes, seed=40 + G)
    osys = OracleSystem(cx, tables)
    st = OracleState(cx.n_swarms, G, cx.pose_len, cx.poses)
    if G > 2:
        st.pos[1, 1] = st.pos[1, 0]  # equal poses: equal scores, no neighbours of each other
    U = np.array(sd.gso_draws(5, cx.n_swarms, steps, G))
    U[0, 1, :] = 0.0
    U[2, 2, :] = 1.0 - 2.0 ** -53
    with sd.Docking([cx], tables, precision=sd.SD_PREC_FP64) as dk:
        for t in range(steps):
            st.vision[:] = 30.0
            dk.set_state(0, sd.State(st.pos.copy(), st.scoring.copy(), st.luciferin.copy(), st.vision.copy(),
                                     st.step.copy(), st.moved.copy(), st.nnei.copy(), st.select.copy(), st.ref.copy()))
            dk.set_draws(0, U[:, t:t + 1, :])
            oracle_step(osys, st, U[:, t, :])
            dk.step(1)
            g = dk.get_state(0)
            for f, o in FIELDS:
                assert np.array_equal(getattr(g, f), getattr(st, o)), f"step {t}: {f} differs"
