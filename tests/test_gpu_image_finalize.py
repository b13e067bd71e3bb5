"""The FP64 image sums over every number of work items an image's four chains
can have left over: 0 to a few rounds of four items in flight a chain."""
import math

import numpy as np
import pytest

from hs_sfm_gb300 import abi
from test_gpu_image_sums import scene, two_product

pytestmark = pytest.mark.gpu

ITEM = 64


@pytest.mark.parametrize("items", [1, 2, 3, 4, 5, 8, 15, 16, 17, 20, 31, 33, 48, 65])
def test_items(items):
    from hs_sfm_gb300 import gba
    s, rng = scene(items, ITEM * (items - 1) + 1 + 62 * (items % 2))
    keys = len(s.points)
    f = gba.vector_function(s, s.x0)[:2 * keys]
    s.near_y = f + rng.normal(0, 1, 2 * keys)
    r = (f - s.near_y).reshape(-1, 2)
    _, ji = gba.jacobian(s, s.x0)
    # stops at the first gradient, which the report gives
    _, rep = gba.solve(s, abi.make_options(max_iterations=1, eps1=1e30, image_item=ITEM,
                                           precision=abi.PRECISION_FP64))
    assert rep.stop_reason == abi.STOP_SMALL_GRADIENT
    exact, mags = [], []
    for a in range(6):
        p0, e0 = two_product(ji[:, 0, a], r[:, 0])
        p1, e1 = two_product(ji[:, 1, a], r[:, 1])
        exact.append(math.fsum(np.concatenate([p0, e0, p1, e1])))
        mags.append(np.abs(p0).sum() + np.abs(p1).sum())
    a = int(np.argmax(np.abs(exact)))
    # a term goes through four products and additions in its lane and four
    # levels of the lanes' tree, each rounding once; what follows is compensated
    assert abs(rep.final_gradient_inf_norm - abs(exact[a])) <= 10 * 2.0 ** -53 * mags[a]
