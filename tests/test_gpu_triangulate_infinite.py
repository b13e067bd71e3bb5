"""A track whose smallest singular vector is a point at infinity is refused,
also when the homogeneous coordinate decouples from the others exactly (the
start of an inverse iteration is then an eigenvector, but not the smallest)."""
import numpy as np
import pytest

import oracle
from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 5000, 10000, 20000])
def test_decoupled_point_at_infinity(copies):
    from hs_sfm_gb300 import gba
    # four parallel cameras; keys x of the origin moved by (3, -5, 5, -3):
    # A^T A = diag(4 f^2, 4 f^2, 1088, 68 depth^2), all exact
    f, depth = 1024.0, 8.0
    views = np.zeros((4, 10))
    views[:, 0] = f
    views[:, 4] = 1.0
    ext = np.zeros((4, 6))
    ext[:, 3] = [-17 * depth / f] * 2 + [17 * depth / f] * 2
    ext[:, 5] = -depth
    keys = np.array([[20.0, 0.0], [12.0, 0.0], [-12.0, 0.0], [-20.0, 0.0]])
    b = synthetic.TriangulationBatch(intrinsics=views, extrinsics=ext,
                                     track_offsets=4 * np.arange(copies + 1, dtype=np.int64),
                                     track_views=np.tile(np.arange(4, dtype=np.int64), copies),
                                     track_keys=np.tile(keys, (copies, 1)), points=np.zeros((copies, 3)))
    P, st = gba.triangulate(b)
    one = synthetic.TriangulationBatch(intrinsics=views, extrinsics=ext, track_offsets=np.array([0, 4]),
                                       track_views=np.arange(4), track_keys=keys, points=np.zeros((1, 3)))
    Pr, sr = oracle.triangulate(one)
    assert sr[0] != abi.GBA_OK
    assert np.all(st == sr[0]) and np.array_equal(P, np.repeat(Pr, copies, axis=0))


def test_nearly_decoupled_matches_oracle():
    """The same tracks with depths below (the origin is found) and above."""
    from hs_sfm_gb300 import gba
    f = 1024.0
    for depth in (1.0, 2.0, 3.5):
        views = np.zeros((4, 10))
        views[:, 0] = f
        views[:, 4] = 1.0
        ext = np.zeros((4, 6))
        ext[:, 3] = [-17 * depth / f] * 2 + [17 * depth / f] * 2
        ext[:, 5] = -depth
        keys = np.array([[20.0, 0.0], [12.0, 0.0], [-12.0, 0.0], [-20.0, 0.0]])
        b = synthetic.TriangulationBatch(intrinsics=views, extrinsics=ext, track_offsets=np.array([0, 4]),
                                         track_views=np.arange(4), track_keys=keys, points=np.zeros((1, 3)))
        opt = abi.make_options(max_iterations=0)
        P, st = gba.triangulate(b, opt)
        Pr, sr = oracle.triangulate(b, opt)
        assert st[0] == sr[0] == abi.GBA_OK and np.max(np.abs(P - Pr)) < 1e-9
