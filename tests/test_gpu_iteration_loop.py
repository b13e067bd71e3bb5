"""Runs with stopping tests iterate in a device-side loop (a CUDA-graph while
node): the same bits, reports and stop reasons as the unrolled launches
(GBA_UNROLLED=1), alone and in batches whose problems stop at different
iterations, in one-shot solves and resident plans, with PCG inside the body."""
import numpy as np
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu

FIELDS = ("status", "stop_reason", "iterations", "accepted", "rejected", "factor_failures", "pcg_iterations",
          "initial_cost", "final_cost", "final_rmse", "final_mu", "final_gradient_inf_norm")


def scenes(kind):
    if kind == "one":
        return [synthetic.ring_scene(num_images=9, num_points=400, seed=3)]
    if kind == "batch":   # different sizes and convergence
        return [synthetic.ring_scene(num_images=5 + 3 * q, num_points=200 + 90 * q, obs_range=(3, 6), seed=q)
                for q in range(5)]
    if kind == "many":    # more problems than the loop's control has threads
        return [synthetic.ring_scene(num_images=4, num_points=40, obs_per_point=4, seed=q) for q in range(300)]
    if kind == "cameras":
        return [synthetic.full_model_scene(seed=5, num_images=10, num_points=400, obs_per_point=4)]
    return [synthetic.grid_scene(num_images=60, num_points=5000, seed=2)]


CASES = [("one", {}), ("one", dict(max_iterations=5)), ("one", dict(eps1=1e12)), ("batch", {}),
         ("batch", dict(precision=abi.PRECISION_MIXED)), ("batch", dict(function_tolerance=1e-6, eps1=0.0, eps2=0.0)),
         ("many", dict(precision=abi.PRECISION_MIXED)), ("cameras", {}), ("grid", {}),
         ("grid", dict(precision=abi.PRECISION_MIXED)),
         ("grid", dict(linear_solver=abi.LINEAR_PCG, loss=abi.LOSS_HUBER))]


@pytest.mark.parametrize("kind,kw", CASES)
def test_loop_equals_unrolled(kind, kw, monkeypatch):
    from hs_sfm_gb300 import gba
    ss = scenes(kind)
    opt = abi.make_options(**{**dict(max_iterations=30), **kw})

    def both():
        plan = gba.Plan(ss, opt)
        out = []
        for _ in range(2):   # a replay counts and ends as the first run
            plan.run()
            plan.synchronize()
            xs, reps = plan.get_all()
            out.append((xs, reps, plan.launches()))
        plan.close()
        xs, reps = gba.solve_batch(ss, opt)
        return out + [(xs, reps, None)]

    loop = both()
    monkeypatch.setenv("GBA_UNROLLED", "1")
    flat = both()
    for (xa, ra, la), (xb, rb, lb) in zip(loop, flat):
        for a, b in zip(xa, xb):
            assert np.array_equal(a, b)
        for a, b in zip(ra, rb):
            assert [getattr(a, f) for f in FIELDS] == [getattr(b, f) for f in FIELDS]
        if la is not None and max(r.iterations for r in ra) + 3 < opt.max_iterations:
            assert 0 < la < lb
    assert loop[0][2] == loop[1][2]


def test_loop_from_threads(monkeypatch):
    """Plans looping on their own streams at the same time give the bits they
    give alone."""
    import threading
    from hs_sfm_gb300 import gba
    ss = [synthetic.ring_scene(num_images=8 + q, num_points=500, seed=20 + q) for q in range(4)]
    opt = abi.make_options(max_iterations=30, shared_device=1)
    alone = [gba.solve(s, opt)[0] for s in ss]
    got = [None] * len(ss)

    def work(q):
        for _ in range(3):
            got[q] = gba.solve(ss[q], opt)[0]

    ts = [threading.Thread(target=work, args=(q,)) for q in range(len(ss))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for a, b in zip(alone, got):
        assert np.array_equal(a, b)
