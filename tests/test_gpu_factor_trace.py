"""GBA_FACTOR_TRACE writes the factorization's timeline for every kind of run:
resident plans and one-shot solves, with and without stopping tests."""
import pytest

from hs_sfm_gb300 import abi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, dict(eps1=0.0, eps2=0.0)])
@pytest.mark.parametrize("resident", [False, True])
def test_trace_is_written(kw, resident, tmp_path, monkeypatch):
    from hs_sfm_gb300 import gba
    s = synthetic.ring_scene(num_images=64, num_points=2500, obs_per_point=4, seed=3)
    opt = abi.make_options(max_iterations=6, precision=abi.PRECISION_FP64, **kw)
    path = tmp_path / "trace.csv"
    monkeypatch.setenv("GBA_FACTOR_TRACE", str(path))
    if resident:
        plan = gba.Plan(s, opt)
        plan.run()
        plan.synchronize()
        plan.close()
    else:
        gba.solve(s, opt)
    lines = path.read_text().splitlines()
    assert lines[0].startswith("cta,mode,i,j") and len(lines) > 12
