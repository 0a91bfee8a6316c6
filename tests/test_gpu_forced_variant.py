"""A forced variant of the mixed DFIRE kernel (SPARKLE_MIXED_VARIANT) runs in calls of few poses too: the names
of the kernels that a call launches, as the profiler of torch records them."""
import numpy as np
import pytest

import sparkledock_b200 as sd

pytestmark = pytest.mark.gpu
SHAPES = ["12, 2", "14, 2", "8, 3", "6, 4"]  # warps and CTAs per SM, by variant


def scorers_of(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
        call()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "dfire_score" in e.name]


@pytest.mark.parametrize("variant", range(sd.mixed_variant_count()))
def test_few_poses_with_a_forced_variant(variant, tables, monkeypatch):
    monkeypatch.setenv("SPARKLE_MIXED_VARIANT", str(variant))
    cx = sd.SyntheticComplex(757, 481, 1, 16, 3, 3, seed=6)
    poses = np.ascontiguousarray(cx.poses.reshape(16, -1))
    with sd.Docking([cx], tables) as dk:
        dk.init_state(0, cx.poses)
        dk.set_draws(0, sd.gso_draws(1, 1, 1, 16))
        dk.step(1)
        assert (dk.tuning()["warps"], dk.tuning()["min_blocks"]) == tuple(int(v) for v in SHAPES[variant].split(","))
        names = scorers_of(lambda: dk.score_poses(0, poses))
    if not names:
        pytest.skip("no kernel records (another profiler is attached)")
    assert len(names) == 1 and f"dfire_score_mixed_kernel<{SHAPES[variant]}," in names[0], names
