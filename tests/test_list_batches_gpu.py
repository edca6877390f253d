"""The pair passes over neighbour lists whose lengths are the edges of their
batches: sets of 1 .. 9 (and 33) particles within one another's supports, so
every list holds the whole set and the last batch holds 1 .. 4 entries, then
pads.  Against the oracle, and the list form against the cell search."""
import numpy as np
import pytest

from helpers import oracle_density_eos, oracle_from, oracle_momentum, rel_err
from pysph_b200 import _native as nat
from pysph_b200 import engine
from pysph_b200.engine import Engine, fluid_scheme

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("thread_rule")]

USE_LIST = 16
# sums of at most 33 terms: FP64 a few ulp of the largest term, times the
# cancellation of opposite forces; FP32C the bars of the FP32 path
TOL = {"fp64": (1e-13, 1e-11), "fp32c": (1e-5, 1e-4)}


def _cluster(n, dim, varying):
    rng = np.random.default_rng(n)
    h = 0.1
    pos = rng.uniform(-0.4 * h, 0.4 * h, (3, n))
    vel = rng.normal(0, 1.0, (3, n))
    if dim == 2:
        pos[2] = vel[2] = 0.0
    hs = np.full(n, h) * (1.0 + (0.05 * rng.uniform(-1, 1, n) if varying else 0.0))
    return dict(x=pos[0], y=pos[1], z=pos[2], u=vel[0], v=vel[1], w=vel[2],
                m=rng.uniform(0.5, 1.0, n), h=hs, rho=np.full(n, 1000.0), p=np.zeros(n),
                cs=np.full(n, 10.0))


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 33])
@pytest.mark.parametrize("lanes", [1, 2, 8])
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_lists_of_every_length(n, lanes, precision):
    for dim, varying in ((2, False), (3, False), (2, True)):
        params = dict(dim=dim, c0=10.0, rho0=100.0, gamma=1.0, alpha=0.1, beta=0.2, eta=0.1,
                      gravity=(0.0, -9.81, 0.0), dt=1e-5)
        arr = _cluster(n, dim, varying)
        scheme = fluid_scheme(1)
        eng = Engine([([arr], params)], scheme, dim=dim, precision=precision, lanes=lanes,
                     exact_lanes=True)
        assert eng.desc.cfg.lanes == lanes
        osys = oracle_from([arr], params, scheme, dim)
        osys.update()
        oracle_density_eos(osys, scheme)
        oracle_momentum(osys, scheme)
        O = osys.arrays[0]
        rtol, atol = TOL[precision]
        names = ("au", "av", "aw")[:dim]
        eng.density()          # records the lists
        rho = eng.get(0, "rho").cpu().numpy()
        assert np.max(np.abs(rho - O.rho) / O.rho) <= rtol
        assert eng.pair_counts()[0] == n * n
        for mode in (0, 1, 2):
            eng.momentum(mode=mode | USE_LIST)
            listed = [eng.get(0, c).cpu().numpy() for c in names]
            eng.momentum(mode=mode)
            searched = [eng.get(0, c).cpu().numpy() for c in names]
            scale = max(np.max(np.abs(s)) for s in searched)
            for a, b in zip(listed, searched):
                assert rel_err(a, b, scale) <= atol, (dim, mode)
            if mode == 0:
                for a, c in zip(listed, names):
                    assert rel_err(a, getattr(O, c), scale) <= atol, (dim, c)
        # the same lists read back by a second density pass
        eng.call("sphb_density", eng.cur, 1, nat.DENSITY_EOS | nat.DENSITY_USE_LIST)
        again = eng.get(0, "rho").cpu().numpy()
        assert np.max(np.abs(again - O.rho) / O.rho) <= rtol
        eng.check_status()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
def test_lists_as_long_as_the_capacity(lanes, dim, precision):
    """Every slot of a list can hold an entry: a clump with as many particles
    as there are slots keeps its lists, one more overflows them all (and the
    passes search the cells).  The capacity covers h = 2 dx (66 entries in
    2D with the skin)."""
    params = dict(dim=dim, c0=10.0, rho0=100.0, gamma=1.0, alpha=0.1, beta=0.2, eta=0.1, dt=1e-5)
    cap = Engine([([_cluster(1, dim, False)], params)], fluid_scheme(1), dim=dim,
                 precision=precision).list_cap
    assert cap >= (88 if dim == 2 else 248)
    for n in (cap, cap + 1):
        arr = _cluster(n, dim, False)
        scheme = fluid_scheme(1)
        eng = Engine([([arr], params)], scheme, dim=dim, precision=precision, lanes=lanes,
                     exact_lanes=True)
        osys = oracle_from([arr], params, scheme, dim)
        osys.update()
        oracle_density_eos(osys, scheme)
        O = osys.arrays[0]
        eng.density()
        rho = eng.get(0, "rho").cpu().numpy()
        assert np.max(np.abs(rho - O.rho) / O.rho) <= TOL[precision][0]
        assert bool((eng.fields["nbr_cnt"][:eng.N] == (n if n == cap else -1)).all())
        listed = {}
        for mode in (USE_LIST, 0):
            eng.momentum(mode=mode)
            listed[mode] = [eng.get(0, c).cpu().numpy() for c in ("au", "av", "aw")[:dim]]
        scale = max(np.max(np.abs(s)) for s in listed[0])
        for a, b in zip(listed[USE_LIST], listed[0]):
            assert rel_err(a, b, scale) <= TOL[precision][1]
        eng.check_status()


def test_threads_per_dest():
    """At least the lanes asked for, more for small engines; exactly as many
    where the caller says so, for the engine or for one launch shape."""
    params = dict(dt=1e-5)
    scenes = [([_cluster(33, 2, False)], params)]
    kw = dict(dim=2, precision="fp64")
    for lanes in (1, 2, 4, 8):
        eng = Engine(scenes, fluid_scheme(1), lanes=lanes, **kw)
        assert eng.desc.cfg.lanes == engine.lanes_for(33, lanes)
        eng.set_launch(lanes, 64, exact=True)
        assert eng.desc.cfg.lanes == eng.lanes == lanes
        eng.set_launch(lanes, 128)         # as the last call said
        assert eng.desc.cfg.lanes == lanes
        eng = Engine(scenes, fluid_scheme(1), lanes=lanes, exact_lanes=True, **kw)
        assert eng.desc.cfg.lanes == lanes
        eng.set_launch(lanes, 128, exact=False)
        assert eng.desc.cfg.lanes == engine.lanes_for(33, lanes)
    for n, want in ((1, 8), (12500, 8), (12501, 4), (25000, 4), (25001, 2), (50000, 2),
                    (50001, 1)):
        if engine.FILL_THREADS:
            assert engine.lanes_for(n, 1) == want
        else:
            assert engine.lanes_for(n, 1) == 1
