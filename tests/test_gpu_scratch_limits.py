"""Sizes at which a scorer's arrays just fit in a CTA's shared memory.  The no-allocation call must take them
without an allocating call before it, whatever shape the number of poses selects; its energies equal the
allocating call's (pyDock within 1e-10: its sums follow the order in which warps take tiles)."""
import ctypes as C

import numpy as np
import pytest

import sparkledock_b200 as sd
from oracle_bind import OracleSystem
from pydock_util import oracle_energy, oracle_grad
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
@pytest.mark.parametrize("n_rec,n_lig", [(800, 4790), (896, 4790), (928, 4790), (1500, 4790), (2560, 4790),
                                         (4000, 4750)])
def test_few_poses_at_the_shape_limit(n_rec, n_lig, tables):
    cx = sd.SyntheticComplex(n_rec, n_lig, 8, 1, 0, 0, seed=n_rec)
    poses = cx.poses.reshape(8, -1)
    for precision in (sd.SD_PREC_FP64, sd.SD_PREC_FP64_REF):
        with sd.Docking([cx], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
            en = noalloc_energies(dk, poses, precision)
            _, ref = dk.score_poses(0, poses, precision)
            assert (np.abs(en - ref) / np.maximum(np.abs(ref), 1.0)).max() <= 1e-10


# the arrays fit by themselves, but not beside the buffers of the warps
@pytest.mark.parametrize("n_rec,n_lig,scoring", [(23100, 300, sd.SD_SCORING_DFIRE), (25900, 300, sd.SD_SCORING_DFIRE),
                                                 (27600, 1, sd.SD_SCORING_DFIRE), (24000, 640, sd.SD_SCORING_DFIRE),
                                                 (200000, 4600, sd.SD_SCORING_PYDOCK),
                                                 (200000, 4880, sd.SD_SCORING_PYDOCK)])
def test_arrays_at_the_shared_memory_limit(n_rec, n_lig, scoring, tables):
    cx = sd.SyntheticComplex(n_rec, n_lig, 2, 1, 0, 0, seed=n_rec)
    poses = np.array(cx.poses.reshape(2, -1))
    poses[:, :3] *= 0.9
    for precision in (sd.SD_PREC_FP64, sd.SD_PREC_FP64_REF) if scoring == sd.SD_SCORING_PYDOCK else (sd.SD_PREC_FP64,):
        with sd.Docking([cx], tables, scoring=scoring) as dk:
            en = noalloc_energies(dk, poses, precision)
            _, ref = dk.score_poses(0, poses, precision)
        assert np.isfinite(ref).all() and (ref != 0.0).any()
        if scoring == sd.SD_SCORING_DFIRE:
            assert np.array_equal(en, ref)
        else:
            assert (np.abs(en - ref) / np.maximum(np.abs(ref), 1.0)).max() <= 1e-10


@pytest.mark.parametrize("n_rec,extent", [(16384, 0.0), (16384, 1e4), (16385, 1e4), (20000, 0.0), (20000, 1e4)])
def test_more_near_tiles_than_are_ordered(n_rec, extent, tables):
    """pyDock orders up to 512 near tiles by distance; a receptor displacement bound of hundreds of A makes
    every tile near."""
    cx = sd.SyntheticComplex(n_rec, 40, 3, 1, 1, 0, seed=n_rec)
    cx.rec_mask[:] = np.arange(n_rec) % 5 == 0
    poses = np.array(cx.poses.reshape(3, -1))
    poses[:, :3] *= 0.8
    poses[:, 7] = extent
    osys = OracleSystem(cx, tables, scoring=1)
    ref = np.array([oracle_energy(osys, p) for p in poses])
    grad = np.array([oracle_grad(osys, p, 7) for p in poses])
    top = np.maximum(np.abs(grad).max(axis=1), 1.0)
    with sd.Docking([cx], tables, scoring=sd.SD_SCORING_PYDOCK) as dk:
        e, g = dk.pydock_grad(0, poses, sd.SD_PREC_FP64)
        _, s = dk.score_poses(0, poses, sd.SD_PREC_FP64)
        for en in (e, s):
            assert (np.abs(en - ref) / np.maximum(np.abs(ref), top)).max() <= 1e-10
        assert (np.abs(g - grad) / top[:, None]).max() <= 1e-10
