"""Sizes at which a scorer's arrays just fit in a CTA's shared memory.  The no-allocation call must take them
without an allocating call before it, whatever shape the number of poses selects; its energies equal the
allocating call's (pyDock within 1e-10: its sums follow the order in which warps take tiles)."""
import ctypes as C

import numpy as np
import pytest

import sparkledock_b200 as sd
from sparkledock_b200 import _abi

pytestmark = pytest.mark.gpu


def noalloc_energies(dk, poses, precision):
    import torch
    n = poses.shape[0]
    d_pose = torch.from_numpy(np.ascontiguousarray(poses)).cuda()
    d_sc, d_en = (torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    d_ref = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = _abi.lib().sd_score_poses_noalloc(dk._ctx, 0, C.c_void_p(d_pose.data_ptr()), n, precision,
                                           C.c_void_p(d_sc.data_ptr()), C.c_void_p(d_en.data_ptr()),
                                           C.c_void_p(d_ref.data_ptr()), 1)
    assert rc == 0, _abi.lib().sd_last_error()
    return d_en.cpu().numpy()


# 24 warps' buffers, their static arrays (12.6 KiB) and a ligand of 4,800 slots: too much for one CTA by up to
# 608 bytes; and one tile of 32 receptor atoms on either side
@pytest.mark.parametrize("n_rec,n_lig", [(800, 4790), (896, 4790), (928, 4790), (1500, 4790), (2560, 4790), (4000, 4750)])
def test_few_poses_at_the_shape_limit(n_rec, n_lig, tables):
    cx = sd.SyntheticComplex(n_rec, n_lig, 8, 1, 0, 0, seed=n_rec)
    poses = cx.poses.reshape(8, -1)
    for precision in (sd.SD_PREC_FP64, sd.SD_PREC_FP64_REF):
        with sd.Docking([cx], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
            en = noalloc_energies(dk, poses, precision)
            _, ref = dk.score_poses(0, poses, precision)
            assert (np.abs(en - ref) / np.maximum(np.abs(ref), 1.0)).max() <= 1e-10
