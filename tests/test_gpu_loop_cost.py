"""A run with stopping tests that uses up its iterations takes about what the
plain sequence takes (GBA_UNROLLED=1), and one that stops early much less."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


def compare(gba, s, monkeypatch, **kw):
    """Device time under the default rule over that of the plain sequence."""
    plans = []
    for env in (False, True):
        if env:
            monkeypatch.setenv("GBA_UNROLLED", "1")
        plans.append(gba.Plan(s, abi.make_options(**kw)))
    monkeypatch.delenv("GBA_UNROLLED")
    ms = [[], []]
    for r in range(26):   # in turn
        for q, p in enumerate(plans):
            p.run()
            p.synchronize()
            if r > 1:
                ms[q].append(p.last_run_ms())
    its = plans[0].report().iterations
    [p.close() for p in plans]
    return np.median(ms[0]) / np.median(ms[1]), its


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("limit", [4, 5, 10, 20, 50])
def test_used_up(limit, graph, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=22, num_points=4000, obs_range=(2, 5), seed=4)
    ratio, its = compare(gba, s, monkeypatch, max_iterations=limit, precision=abi.PRECISION_MIXED, eps1=1e-300,
                         eps2=1e-300, use_cuda_graph=graph)
    # (replays from the host scatter by 2% themselves)
    assert its == limit and ratio < 1.04, ratio


@pytest.mark.parametrize("graph", [0, 1])
def test_stopped_early(graph, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=10, num_points=1000, seed=0)
    ratio, its = compare(gba, s, monkeypatch, max_iterations=50, use_cuda_graph=graph)
    assert its < 12 and ratio < 0.8, ratio
