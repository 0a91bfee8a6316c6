"""What a context holds of the device's memory after calls with large workspaces: at most 256 MiB of each, and
32 MiB beside them (mode-free complexes, so that the states themselves are small beside that)."""
import numpy as np
import pytest

import sparkledock_b200 as sd

pytestmark = pytest.mark.gpu
HELD = (256 + 32 + 8) << 20  # 8 MiB for allocations of the driver


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_clustering_gives_its_workspace_back(tables):
    S, G = 300, 200
    cx = sd.SyntheticComplex(600, 300, S, G, 0, 0, seed=9)  # 60,000 poses x 900 atoms x 24 bytes: 1.3 GB, 1 GiB kept
    with sd.Docking([cx], tables, precision=sd.SD_PREC_FP64) as dk:
        dk.init_state(0, cx.poses)
        before = free_bytes()
        first = dk.cluster(0, np.ones(600, np.int32), np.ones(300, np.int32))
        assert before - free_bytes() <= HELD
        again = dk.cluster(0, np.ones(600, np.int32), np.ones(300, np.int32))
    assert all(np.array_equal(first[k][:, :1] if first[k].ndim > 1 else first[k],
                              again[k][:, :1] if again[k].ndim > 1 else again[k]) for k in first)


def test_starting_poses_are_not_kept_twice(tables):
    cx = sd.SyntheticComplex(40, 30, 8000, 200, 10, 10, seed=9)  # 1.6 M poses of 216 bytes: 346 MB
    with sd.Docking([cx], tables) as dk:
        before = free_bytes()
        dk.init_state(0, cx.poses)
        assert before - free_bytes() <= HELD
        assert np.array_equal(dk.get_state(0).pos, cx.poses)
