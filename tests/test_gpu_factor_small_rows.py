"""The factorization's kernels against the per-column launches (both arms named:
GBA_CHOL_COLUMNS on the other): systems alone of two to nine tile rows, in both
precisions, so the one-CTA launch and the dataflow launch each meet another."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
@pytest.mark.parametrize("images", [6, 11, 16, 21, 22, 27, 37, 42, 43, 48])
def test_alone_equals_per_column_launches(images, precision, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=images, num_points=40 * images, obs_per_point=4, seed=500 + images)
    opt = dict(max_iterations=3, precision=precision, eps1=0.0, eps2=0.0)
    plan = gba.Plan(s, abi.make_options(**opt))
    tile_rows = (6 * images + 31) // 32
    small = precision == abi.PRECISION_MIXED and tile_rows <= 4
    assert plan.structure()["factor_schedule"] == (2 if small else 1)
    plan.close()
    x, r = gba.solve(s, abi.make_options(**opt))
    monkeypatch.setenv("GBA_CHOL_COLUMNS", "1")
    columns = abi.make_options(shared_device=1, **opt)
    plan = gba.Plan(s, columns)
    assert plan.structure()["factor_schedule"] == 0
    plan.close()
    xc, rc = gba.solve(s, columns)
    assert r.status == rc.status == abi.GBA_OK and r.accepted == rc.accepted and r.final_cost == rc.final_cost
    assert np.array_equal(x, xc)
