"""gba_plan_device_bytes counts what a plan takes from the device's memory
pool, and gba_estimate_device_bytes (which the server admits by) bounds it."""
import ctypes

import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


def pool_used():
    """Bytes in use of the device's default memory pool."""
    with open("/proc/self/maps") as fh:
        path = next(line.split()[-1] for line in fh if "libcudart" in line)
    rt = ctypes.CDLL(path)
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(used)) == 0   # cudaMemPoolAttrUsedMemCurrent
    return used.value


SCENES = {
    "tiny": lambda: synthetic.ring_scene(num_images=4, num_points=50, obs_per_point=3),
    "small": lambda: synthetic.ring_scene(num_images=10, num_points=1000),
    "window": lambda: synthetic.ring_scene(num_images=22, num_points=4000, obs_range=(3, 8), seed=4),
    "cameras": lambda: synthetic.full_model_scene(seed=4, num_images=12, num_points=1500, num_cameras=12,
                                                  obs_per_point=4),
    "gcp": lambda: synthetic.gcp_scene(seed=5, num_images=20, num_points=3000, num_gcps=10),
    "grid": lambda: synthetic.grid_scene(num_images=120, num_points=30000, seed=2),
}


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
@pytest.mark.parametrize("kind", list(SCENES))
def test_held_bytes(kind, precision):
    from hs_sfm_gb300 import gba
    s = SCENES[kind]()
    opt = abi.make_options(precision=precision, max_iterations=2)
    gba.solve(s, opt)
    before = pool_used()
    plan = gba.Plan(s, opt)
    plan.run()
    plan.synchronize()
    plan.get_all()
    held, counted = pool_used() - before, plan.device_bytes()
    plan.close()
    # (the pool rounds each allocation to 512 bytes; a plan makes at most 200)
    assert held <= counted + 200 * 512, (held, counted)
    assert gba.estimate_device_bytes(s, precision) >= counted
