"""gba_estimate_device_bytes (which the server admits by) bounds what a plan
asks for also where the key pairs, placed on the device, are most of it."""
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
@pytest.mark.parametrize("kind", ["grid", "long_tracks", "many_images"])
def test_estimate_bounds_pairs(kind, precision):
    from hs_sfm_gb300 import gba
    s = {"grid": lambda: synthetic.grid_scene(num_images=120, num_points=30000, seed=2),
         "long_tracks": lambda: synthetic.ring_scene(num_images=60, num_points=4000, obs_per_point=30, seed=3),
         "many_images": lambda: synthetic.ring_scene(num_images=700, num_points=4000, obs_per_point=4, seed=4)}[kind]()
    plan = gba.Plan(s, abi.make_options(precision=precision, max_iterations=1))
    held = plan.device_bytes()
    plan.close()
    assert held <= gba.estimate_device_bytes(s, precision) <= 3 * held + (2 << 20)
