"""gba_autotune in FP64: its baseline is what item sizes left to the library
(option 0) give, and a size that stays at that is returned as 0."""
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


def ms_per_iteration(gba, s, **sizes):
    opt = abi.make_options(max_iterations=2, eps1=-1.0, eps2=-1.0, precision=abi.PRECISION_FP64, use_cuda_graph=1,
                           **sizes)
    plan = gba.Plan(s, opt)
    best = float("inf")
    for r in range(5):
        plan.run()
        plan.synchronize()
        if r:
            best = min(best, plan.last_run_ms())
    plan.close()
    return best / 2


def test_baseline_is_option_0():
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=10, num_points=1000, seed=7)
    t = gba.autotune([s], abi.make_options(precision=abi.PRECISION_FP64, max_iterations=10))
    assert t["pair_item"] in (0, 256, 512, 1024, 2048, 4096)
    assert t["image_item"] in (0, 256, 512, 1024)
    assert t["key_item"] in (0, 256, 512, 1024, 2048)
    assert 0 < t["ms_per_iteration"] <= t["default_ms_per_iteration"]
    auto = ms_per_iteration(gba, s)
    fixed = ms_per_iteration(gba, s, pair_item=1024, image_item=512, key_item=1024)
    assert auto < 0.8 * fixed          # (the sizes this small problem is cut to)
    assert t["default_ms_per_iteration"] < 0.5 * (auto + fixed)
    tuned = ms_per_iteration(gba, s, pair_item=t["pair_item"], image_item=t["image_item"], key_item=t["key_item"])
    assert tuned < 0.5 * (auto + fixed)
