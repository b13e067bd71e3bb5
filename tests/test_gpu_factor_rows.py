"""The dataflow factorization's layouts give the bits of the per-column
launches at their edges: row CTAs with helpers up to 38 tile rows (152 SMs),
row CTAs without helpers to 76, the common scheduler above; and a last tile
row of every fill."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("images", [2, 5, 6, 16, 37, 42, 43, 48, 49])
def test_small_systems_alone(images, monkeypatch):
    """One small mixed-precision system (up to nine tile rows) in one launch:
    the bits of the per-column launches."""
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=images, num_points=60 * images, obs_per_point=min(4, images), seed=images)
    opt = abi.make_options(max_iterations=4, precision=abi.PRECISION_MIXED, eps1=0.0, eps2=0.0, shared_device=1)
    x, r = gba.solve(s, opt)
    monkeypatch.setenv("GBA_CHOL_COLUMNS", "1")
    xc, rc = gba.solve(s, opt)
    assert r.status == rc.status == abi.GBA_OK and r.final_cost == rc.final_cost
    assert np.array_equal(x, xc)


@pytest.mark.parametrize("images,precision", [(16, 0), (16, 1), (27, 0), (27, 1), (64, 0), (64, 1), (202, 0), (202, 1),
                                              (203, 1), (229, 0), (405, 1), (406, 1)])
def test_layouts_equal_per_column_launches(images, precision):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=images, num_points=40 * images, obs_per_point=4, seed=300 + images)
    opt = dict(max_iterations=3, precision=precision, eps1=0.0, eps2=0.0)
    x, r = gba.solve(s, abi.make_options(**opt))
    xc, rc = gba.solve(s, abi.make_options(shared_device=1, **opt))
    assert r.status == rc.status == abi.GBA_OK and r.accepted == rc.accepted
    assert np.array_equal(x, xc)
