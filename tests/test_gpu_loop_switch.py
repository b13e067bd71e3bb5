"""Whether a plan's iterations run in a device-side loop is decided once, when
the plan is made: GBA_UNROLLED set or cleared between a plan's runs changes
neither its results nor its launch counts."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("unrolled_first", [False, True])
def test_switch_between_runs(graph, unrolled_first, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=9, num_points=400, seed=3)
    opt = abi.make_options(max_iterations=30, use_cuda_graph=graph)
    want, _ = gba.solve(s, opt)

    def env(on):
        if on:
            monkeypatch.setenv("GBA_UNROLLED", "1")
        else:
            monkeypatch.delenv("GBA_UNROLLED", raising=False)

    env(unrolled_first)
    plan = gba.Plan(s, opt)
    counts = []
    for on in (unrolled_first, not unrolled_first, unrolled_first):
        env(on)
        before = gba.kernel_launch_count()
        plan.run()
        plan.synchronize()
        counts.append((plan.launches(), gba.kernel_launch_count() - before))
        assert np.array_equal(plan.x(0), want)
    plan.close()
    assert counts[0] == counts[1] == counts[2] and counts[0][0] > 0
