"""Lanes per track (8, 4, 2, 1 by the batch's size) and the order by track
length: the points of the oracle at the edges of each, with tracks longer than
the order's 64 lengths and two-view tracks beside them."""
import numpy as np
import pytest

import oracle
from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,views,longest", [(1, 20, 8), (33, 90, 80), (4864, 24, 8), (4865, 24, 8), (9729, 24, 5),
                                             (19456, 30, 12), (19457, 30, 12), (20000, 90, 70)])
def test_layouts_match_oracle(n, views, longest):
    from hs_sfm_gb300 import gba
    b = synthetic.triangulation_batch(seed=n, num_points=n, num_views=views, views_range=(2, longest))
    P, st = gba.triangulate(b)
    Pr, sr = oracle.triangulate(b)
    assert np.array_equal(st, sr) and np.all(st == abi.GBA_OK)
    # the tolerances of tests/test_gpu_triangulate.py: FP64 on both sides, an
    # LM that may stop one step apart on a flat direction
    assert np.max(np.abs(P - Pr)) < 1e-6

    def cost(X):
        r = synthetic.project_views(b.intrinsics, b.extrinsics, b.track_views,
                                    np.repeat(X, np.diff(b.track_offsets), axis=0)) - b.track_keys
        return np.add.reduceat(np.sum(r * r, axis=1), b.track_offsets[:-1])

    c, cr = cost(P), cost(Pr)
    assert np.all(np.abs(c - cr) <= 1e-9 * cr + 1e-12)


def test_short_tracks_in_every_layout():
    """Tracks of no and one view keep their status between good ones."""
    from hs_sfm_gb300 import gba
    for n in (40, 6000, 12000, 25000):
        b = synthetic.triangulation_batch(seed=n, num_points=n)
        k = np.diff(b.track_offsets).copy()
        keep = np.ones(len(b.track_views), dtype=bool)
        for j, left in ((0, 0), (n // 2, 1), (n - 1, 1)):
            keep[b.track_offsets[j] + left:b.track_offsets[j + 1]] = False
            k[j] = left
        b.track_views, b.track_keys = b.track_views[keep], b.track_keys[keep]
        b.track_offsets = np.concatenate([[0], np.cumsum(k)]).astype(np.int64)
        P, st = gba.triangulate(b)
        bad = np.zeros(n, dtype=bool)
        bad[[0, n // 2, n - 1]] = True
        assert np.all(st[bad] == abi.GBA_ERR_INVALID) and np.all(st[~bad] == abi.GBA_OK)
        assert np.all(P[bad] == 0.0)
