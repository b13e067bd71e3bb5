"""A track's point has the same bits in a batch of any size (by which the lanes
per track are chosen)."""
import dataclasses

import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


def first(b, n):
    m = int(b.track_offsets[n])
    return dataclasses.replace(b, track_offsets=b.track_offsets[:n + 1].copy(), track_views=b.track_views[:m].copy(),
                               track_keys=b.track_keys[:m].copy(), points=b.points[:n].copy())


@pytest.mark.parametrize("views,longest,distortion", [(24, 12, True), (90, 70, False)])
def test_bits_do_not_depend_on_the_batch(views, longest, distortion):
    from hs_sfm_gb300 import gba
    b = synthetic.triangulation_batch(seed=9, num_points=25000, num_views=views, views_range=(2, longest), noise=0.7,
                                      distortion=distortion)
    P, st = gba.triangulate(b)
    assert np.all(st == abi.GBA_OK)
    for n in (1, 3, 100, 4864, 4865, 9728, 9729, 19456, 19457):
        Pn, stn = gba.triangulate(first(b, n))
        assert np.array_equal(stn, st[:n])
        assert np.array_equal(Pn, P[:n]), n
