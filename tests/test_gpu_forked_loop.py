"""The forked iteration (GBA_FORK: the image sums and the loop's control on a
second stream) inside the device-side loop: the bits, reports and launch counts
of the unrolled launches and of one stream."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu

FIELDS = ("status", "stop_reason", "iterations", "accepted", "rejected", "factor_failures", "pcg_iterations",
          "initial_cost", "final_cost", "final_rmse", "final_mu", "final_gradient_inf_norm")

CASES = [("grid", {}), ("grid", dict(precision=abi.PRECISION_MIXED)), ("grid", dict(max_iterations=4)),
         ("grid", dict(precision=abi.PRECISION_MIXED, function_tolerance=1e-6, eps1=0.0, eps2=0.0)),
         ("cameras", {}), ("cameras", dict(precision=abi.PRECISION_MIXED)),
         ("grid", dict(linear_solver=abi.LINEAR_PCG, loss=abi.LOSS_HUBER)),
         ("grid", dict(linear_solver=abi.LINEAR_PCG, precision=abi.PRECISION_MIXED)), ("batch", {})]


def scenes(kind):
    if kind == "batch":
        return [synthetic.ring_scene(num_images=5 + 3 * q, num_points=200 + 90 * q, obs_range=(3, 6), seed=q)
                for q in range(4)]
    if kind == "cameras":
        return [synthetic.full_model_scene(seed=5, num_images=10, num_points=400, obs_per_point=4)]
    return [synthetic.grid_scene(num_images=60, num_points=5000, seed=2)]


@pytest.mark.parametrize("kind,kw", CASES)
def test_forked_loop(kind, kw, monkeypatch):
    from hs_sfm_gb300 import gba
    ss = scenes(kind)
    opt = abi.make_options(**{**dict(max_iterations=30), **kw})

    def runs():
        plan = gba.Plan(ss, opt)
        forked = plan.structure()["forked"]
        out = []
        for _ in range(2):
            plan.run()
            plan.synchronize()
            xs, reps = plan.get_all()
            out.append((xs, reps, plan.launches()))
        plan.close()
        xs, reps = gba.solve_batch(ss, opt)
        return forked, out + [(xs, reps, None)]

    monkeypatch.setenv("GBA_FORK", "1")
    forked, loop = runs()
    assert forked == 1
    monkeypatch.setenv("GBA_UNROLLED", "1")
    forked, flat = runs()
    assert forked == 1
    monkeypatch.delenv("GBA_UNROLLED")
    monkeypatch.setenv("GBA_ONE_STREAM", "1")
    forked, single = runs()
    assert forked == 0
    for other in (flat, single):
        for (xa, ra, _), (xb, rb, _) in zip(loop, other):
            for a, b in zip(xa, xb):
                assert np.array_equal(a, b)
            for a, b in zip(ra, rb):
                assert [getattr(a, f) for f in FIELDS] == [getattr(b, f) for f in FIELDS]
    assert loop[0][2] == loop[1][2]


def test_large_plan_forks_and_loops(monkeypatch):
    """The default of a large scene (300,000 keys or more)."""
    from hs_sfm_gb300 import gba
    s = synthetic.grid_scene(num_images=80, num_points=60000, seed=6)
    opt = abi.make_options(max_iterations=12, precision=abi.PRECISION_MIXED, function_tolerance=1e-6)
    plan = gba.Plan(s, opt)
    assert plan.structure()["forked"] == 1
    plan.close()
    x, r = gba.solve(s, opt)
    monkeypatch.setenv("GBA_UNROLLED", "1")
    monkeypatch.setenv("GBA_ONE_STREAM", "1")
    xf, rf = gba.solve(s, opt)
    assert np.array_equal(x, xf) and [getattr(r, f) for f in FIELDS] == [getattr(rf, f) for f in FIELDS]
