"""Launch counts of runs that iterate in a device-side loop: right whenever
they are asked for, and complete for runs that nothing waited for."""
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, dict(precision=abi.PRECISION_MIXED), dict(linear_solver=abi.LINEAR_PCG)])
@pytest.mark.parametrize("graph", [0, 1])
def test_counts_without_a_wait(graph, kw):
    from hs_sfm_gb300 import gba
    s = synthetic.grid_scene(num_images=60, num_points=5000, seed=2)
    plan = gba.Plan(s, abi.make_options(max_iterations=30, use_cuda_graph=graph, **kw))
    plan.run()
    plan.synchronize()
    c0 = gba.kernel_launch_count()
    plan.run()
    plan.synchronize()
    one, full = plan.launches(), gba.kernel_launch_count() - c0
    assert one == full > 0
    plan.run()
    assert plan.launches() == one          # asked while it runs
    if "linear_solver" in kw:              # (the inner loop's passes are counted when a run is waited for)
        plan.close()
        return
    c0 = gba.kernel_launch_count()
    for _ in range(3):                     # one after the other, no wait between
        plan.run()
    plan.synchronize()
    assert plan.launches() == one
    assert gba.kernel_launch_count() - c0 == 3 * full
    plan.close()
