"""The integrator stage in the FP64 force pass's epilogue against the stage
as its own pass: the same state bit for bit, for every integrator, with walls,
in 3D and with the integrated density, over rebins, host writes of fluid and
walls between steps, and replayed from a graph."""
import numpy as np
import pytest
import torch

from pysph_b200 import workloads as W
from pysph_b200.engine import Engine, continuity_scheme, fluid_scheme

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("thread_rule")]


def _case(name):
    if name == "lattice3d":
        arrays, _, params = W.lattice3d(n=8)
        rng = np.random.default_rng(2)
        for c in "uvw":
            arrays[0][c] = rng.normal(0.0, 1.0, len(arrays[0]["x"]))
        return arrays, dict(params, dt=5e-4, alpha=0.1), fluid_scheme(1), 3
    arrays, _, params = W.dam_break(dx=0.05)
    rng = np.random.default_rng(3)
    n = len(arrays[0]["x"])
    arrays[0]["u"], arrays[0]["v"] = rng.normal(0.0, 1.0, (2, n))
    scheme = continuity_scheme(2) if name == "continuity" else fluid_scheme(2)
    return arrays, dict(params, dt=2e-4, cfl=0.0 if name == "continuity" else 0.3), scheme, 2


@pytest.mark.parametrize("integrator", ["pc", "euler", "rk2", "rk4"])
@pytest.mark.parametrize("name", ["dam", "continuity", "lattice3d"])
def test_matches_the_separate_stage(name, integrator):
    arrays, params, scheme, dim = _case(name)
    engs = [Engine([(arrays, params)], scheme, dim=dim, precision="fp64", fuse_stage=f)
            for f in (True, False)]
    assert engs[0].fuses_stage and not engs[1].fuses_stage
    names = ["x", "y", "u", "v", "rho", "p"] + (["z", "w"] if dim == 3 else [])

    def same(when):
        for a in range(engs[0].A):
            for n in names:
                assert torch.equal(engs[0].get(a, n), engs[1].get(a, n)), (when, a, n)
        s0, s1 = (e.scene_state()[0] for e in engs)
        assert (s0.dt, s0.t, s0.count) == (s1.dt, s1.t, s1.count)
    for e in engs:
        e.reset_pair_counts()
        for _ in range(7):
            e.step(integrator)
        e.check_status()
    same("steps")
    for e in engs:     # the host moves fluid and walls
        for a in range(e.A):
            e.exchange_in(a, "x", e.get(a, "x") + 0.012)
            e.exchange_in(a, "v", e.get(a, "v") * 0.5)
        for _ in range(3):
            e.step(integrator)
        for _ in range(5):
            e.step_graphed(integrator)
        e.check_status()
        assert e.device_rebins() >= 1
    same("host writes and graph replays")


@pytest.mark.parametrize("integrator", ["pc", "euler", "rk2", "rk4"])
def test_a_callers_graph_outlives_other_steps(integrator):
    """A graph that a program captured itself holds the buffers' addresses, so
    every step leaves the state where it found it: a captured PC step, then one
    step of each integrator, then the graph again."""
    arrays, params, scheme, dim = _case("dam")
    engs = [Engine([(arrays, params)], scheme, dim=dim, precision="fp64", fuse_stage=f)
            for f in (True, False)]
    for e in engs:
        for _ in range(2):
            e.pc_step()
        if integrator == "rk4":
            e.step("rk4")       # makes its sums
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            e.pc_step()
        g.replay()
        e.step(integrator)
        g.replay()
        e.check_status()
    for n in ("x", "y", "u", "v", "rho", "p"):
        assert torch.equal(engs[0].get(0, n), engs[1].get(0, n)), n


def test_needs_the_second_copy():
    arrays, params, scheme, dim = _case("dam")
    eng = Engine([(arrays, params)], scheme, dim=dim, precision="fp64", step_lists=False)
    assert not eng.fuses_stage          # every rebin swaps the state buffers
    eng.pc_step()
    eng.check_status()
    with pytest.raises(RuntimeError):   # refused on the host
        eng.call("sphb_momentum", eng.cur, 1, 1, 16 | (1 << 8))
