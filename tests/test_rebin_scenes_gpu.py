"""The rebin's scene grids at the edges of its paths: one scene, a block's
worth of scenes (256), one either side of it, and more; scenes of one particle
among them.  Every scene steps like an engine of its own."""
import numpy as np
import pytest

from pysph_b200 import workloads as W
from pysph_b200.engine import Engine, fluid_scheme

pytestmark = pytest.mark.gpu


def _scene(s):
    arrays, _, params = W.elliptical_drop(dx=0.3 if s % 3 else 0.2, vel_scale=50.0 + s)
    a = {k: np.array(v, copy=True) for k, v in arrays[0].items()}
    if s % 5 == 4:
        a = {k: v[:1] for k, v in a.items()}
    a["x"] = a["x"] + 3.0 * (s % 7) - 10.0     # grids away from the origin too
    a["y"] = a["y"] - 2.0 * (s % 4)
    return [a], dict(params, dt=1e-4)


@pytest.mark.parametrize("num", [1, 2, 255, 256, 257, 600])
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_scenes_step_alone(num, precision):
    specs = [_scene(s) for s in range(num)]
    eng = Engine(specs, fluid_scheme(1), dim=2, precision=precision)
    checked = sorted({0, 1, 4, num // 2, num - 1} & set(range(num)))
    for s in checked:
        one = Engine([specs[s]], fluid_scheme(1), dim=2, precision=precision)
        np.testing.assert_array_equal(eng.cell_coords(s), one.cell_coords(0))
    eng.reset_pair_counts()
    for _ in range(12):       # the skin is crossed several times
        eng.pc_step()
    eng.check_status()
    assert eng.device_rebins() >= 2
    tol = 1e-12 if precision == "fp64" else 1e-5
    for s in checked:
        one = Engine([specs[s]], fluid_scheme(1), dim=2, precision=precision)
        for _ in range(12):
            one.pc_step()
        one.check_status()
        for n in ("x", "y", "u", "v", "rho"):
            got = eng.get(0, n, scene=s).cpu().numpy()
            ref = one.get(0, n).cpu().numpy()
            scale = max(np.max(np.abs(ref)), 1.0)
            assert np.max(np.abs(got - ref)) <= tol * scale, (s, n)
