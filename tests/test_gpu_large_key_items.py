"""Key items longer than the cost kernel keeps in shared memory (a caller's
key_item): the records it forms from the residuals it has just written are
those of a separate linearization, bit for bit."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_item", [1024, 1025, 2048, 4000])
@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
def test_records_of_large_items(key_item, precision, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=24, num_points=6000, obs_per_point=7, seed=8)
    opt = abi.make_options(max_iterations=8, eps1=0.0, eps2=0.0, precision=precision, key_item=key_item,
                           loss=abi.LOSS_HUBER)
    x, r = gba.solve(s, opt)
    monkeypatch.setenv("GBA_SEPARATE_LINEARIZE", "1")
    xs, rs = gba.solve(s, opt)
    assert r.status == rs.status == abi.GBA_OK
    assert r.final_cost == rs.final_cost and np.array_equal(x, xs)
