"""Parity of the sm_100a engine (through the C ABI) with the oracle.

Integer work is compared bit for bit: cell coordinates floor(x / cs) and
neighbour sets (sorted index lists) against the reference algorithm.
Floating point: FP64 against the oracle to 1e-12 (densities) / 1e-10
(accelerations, relative to the largest); FP32C (FP32 pair sums with Kahan
compensation) to 1e-5 relative density error, the accuracy bar of the FP32
path, and 1e-4 for accelerations relative to the largest.
"""
import numpy as np
import pytest
import torch

from helpers import (oracle_from, oracle_density_eos, oracle_momentum, rel_err,
                     pairs_from_oracle)
from pysph_b200 import workloads as W
from pysph_b200.engine import Engine, SceneParams, continuity_scheme, fluid_scheme, lanes_for
from pysph_b200 import _native as nat

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("thread_rule")]

RHO_TOL = {"fp64": 1e-12, "fp32c": 1e-5}
ACC_TOL = {"fp64": 1e-10, "fp32c": 1e-4}
# trajectories over <= 10 steps: position error in units of the particle
# spacing dx, max|x - x_ref| / dx.  FP64 to round-off; FP32C accelerations
# carry ~1e-7..1e-6 relative error (the Tait EOS amplifies a density error
# by 7 B / rho0), which moves particles by ~1e-9 of a unit per step.
TRAJ_TOL = {"fp64": 1e-10, "fp32c": 2e-6}


def traj_err(got, ref, h):
    dx = float(np.max(h)) / 1.3
    return float(np.max(np.abs(got - ref)) / dx)


def drop(dx=0.025):
    arrays, types, params = W.elliptical_drop(dx=dx)
    return arrays, params, fluid_scheme(1), 2


def small_dam(dx=0.02):
    arrays, types, params = W.dam_break(dx=dx)
    return arrays, params, fluid_scheme(2), 2


def lattice(n=20):
    arrays, types, params = W.lattice3d(n=n)
    return arrays, params, fluid_scheme(1), 3


CASES = {"drop": drop, "dam": small_dam, "lattice3d": lattice}


def engine_for(case, precision, **kw):
    arrays, params, scheme, dim = CASES[case]()
    eng = Engine([(arrays, params)], scheme, dim=dim, precision=precision, **kw)
    return eng, arrays, params, scheme, dim


@pytest.mark.parametrize("case", list(CASES))
def test_cell_coords_bit_exact(case):
    # step_lists=False: the cell size is exactly the reference's 2 * max h
    eng, arrays, params, scheme, dim = engine_for(case, "fp64", step_lists=False)
    cs = eng.cell_size()
    # CellManager cell size = 2 * max h over all arrays (S/base/cell.pyx:911-941)
    max_h = max(float(np.max(a["h"])) for a in arrays)
    assert cs == 2.0 * max_h
    import oracle
    for a, arr in enumerate(arrays):
        got = eng.cell_coords(0, a)
        ref = oracle.cell_ids(arr["x"], arr["y"], arr["z"], cs)
        if dim == 2:
            ref[:, 2] = 0
        np.testing.assert_array_equal(got, ref)
    eng.check_status()


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("stencil", [1, 2])
def test_neighbor_sets_bit_exact(case, stencil):
    eng, arrays, params, scheme, dim = engine_for(case, "fp64", stencil=stencil)
    osys = oracle_from(arrays, params, scheme, dim)
    A = len(arrays)
    osys.update_pairs([(d, s) for d in range(A) for s in range(A)])
    for d in range(A):
        for s in range(A):
            di, sa, sj = eng.neighbors(d, 1 << s)
            assert np.all(sa == s)
            odi, osj = pairs_from_oracle(osys, d, s)
            np.testing.assert_array_equal(di, odi)
            np.testing.assert_array_equal(sj, osj)


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("lanes", [1, 4])
def test_density_eos(case, precision, lanes):
    eng, arrays, params, scheme, dim = engine_for(case, precision, lanes=lanes, exact_lanes=True)
    assert eng.desc.cfg.lanes == lanes
    osys = oracle_from(arrays, params, scheme, dim)
    osys.update()
    oracle_density_eos(osys, scheme)
    eng.density()
    eng.check_status()
    for a in range(len(arrays)):
        rho = eng.get(a, "rho").cpu().numpy()
        ref = osys.arrays[a].rho
        err = np.max(np.abs(rho - ref) / np.abs(ref))
        assert err <= RHO_TOL[precision], (a, err)
        p = eng.get(a, "p").cpu().numpy()
        B = params["c0"] ** 2 * params["rho0"] / params["gamma"]
        assert rel_err(p, osys.arrays[a].p, scale=B) <= 10 * RHO_TOL[precision]
    npairs, _ = eng.pair_counts()
    total = sum(len(osys.neighbors(d, s)[1]) for d, srcs in scheme.rho_src.items()
                for s in srcs)
    if precision == "fp64":
        assert npairs == total
    else:
        assert abs(npairs - total) <= max(2, total * 1e-5)


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("lanes", [1, 8])
def test_momentum(case, precision, lanes):
    eng, arrays, params, scheme, dim = engine_for(case, precision, lanes=lanes, exact_lanes=True)
    assert eng.desc.cfg.lanes == lanes
    osys = oracle_from(arrays, params, scheme, dim)
    osys.update()
    oracle_density_eos(osys, scheme)
    oracle_momentum(osys, scheme)
    eng.density()
    eng.momentum()
    eng.check_status()
    for d in scheme.mom_src:
        O = osys.arrays[d]
        names = ("au", "av", "aw")[:dim]
        refs = [O.au, O.av, O.aw][:dim]
        scale = max(np.max(np.abs(r)) for r in refs)
        for nm, ref in zip(names, refs):
            got = eng.get(d, nm).cpu().numpy()
            assert rel_err(got, ref, scale) <= ACC_TOL[precision], nm
        dtf = eng.get(d, "dt_fac").cpu().numpy()
        assert rel_err(dtf, O.dt_fac) <= ACC_TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_drop_trajectory(precision):
    arrays, params, scheme, dim = drop()
    params = dict(params, dt=1e-5)
    eng = Engine([(arrays, params)], scheme, dim=2, precision=precision)
    osys = oracle_from(arrays, params, scheme, dim)
    for _ in range(10):
        eng.pc_step()
        osys.pc_step(1e-5)
    eng.check_status()
    O = osys.arrays[0]
    x = eng.get(0, "x").cpu().numpy()
    y = eng.get(0, "y").cpu().numpy()
    u = eng.get(0, "u").cpu().numpy()
    assert traj_err(x, O.x, arrays[0]["h"]) <= TRAJ_TOL[precision]
    assert traj_err(y, O.y, arrays[0]["h"]) <= TRAJ_TOL[precision]
    # FP32C: velocities integrate accelerations whose relative error is
    # ~1e-7..1e-6 (the Tait EOS amplifies density round-off by ~7 B / rho0)
    assert rel_err(u, O.u) <= (1e-12 if precision == "fp64" else 2e-6)
    rho = eng.get(0, "rho").cpu().numpy()
    assert np.max(np.abs(rho - O.rho) / O.rho) <= RHO_TOL[precision]
    st = eng.scene_state()[0]
    assert st.count == 10
    assert st.t == pytest.approx(1e-4)


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_dam_break_cfl(precision):
    arrays, params, scheme, dim = small_dam()
    eng = Engine([(arrays, params)], scheme, dim=2, precision=precision)
    osys = oracle_from(arrays, params, scheme, dim)
    dts = []
    for _ in range(6):
        dt = osys.cfl_time_step(params["cfl"], params["c0"], params["dt_initial"])
        osys.pc_step(dt)
        dts.append(dt)
        eng.pc_step()
        st = eng.scene_state()[0]
        if precision == "fp64":
            assert st.dt == pytest.approx(dt, rel=1e-12)
        else:
            assert st.dt == pytest.approx(dt, rel=1e-5)
    eng.check_status()
    O = osys.arrays[0]
    for nm in ("x", "y"):
        got = eng.get(0, nm).cpu().numpy()
        assert traj_err(got, getattr(O, nm), arrays[0]["h"]) <= TRAJ_TOL[precision]
    rho = eng.get(1, "rho").cpu().numpy()
    assert np.max(np.abs(rho - osys.arrays[1].rho) / osys.arrays[1].rho) <= RHO_TOL[precision]


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_batched_scenes_match_single(precision):
    scenes = W.batched_drops(num_scenes=5, seed=1, n_lo=300, n_hi=1500)
    specs = [(arrs, p) for arrs, _, p in scenes]
    eng = Engine(specs, fluid_scheme(1), dim=2, precision=precision, lanes=4)
    for _ in range(4):
        eng.pc_step()
    eng.check_status()
    for s, (arrs, p) in enumerate(specs):
        osys = oracle_from(arrs, p, fluid_scheme(1), 2)
        for _ in range(4):
            osys.pc_step(p["dt"])
        x = eng.get(0, "x", scene=s).cpu().numpy()
        rho = eng.get(0, "rho", scene=s).cpu().numpy()
        assert traj_err(x, osys.arrays[0].x, arrs[0]["h"]) <= TRAJ_TOL[precision]
        assert np.max(np.abs(rho - osys.arrays[0].rho) / osys.arrays[0].rho) <= RHO_TOL[precision]


def test_free_fall_closed_form():
    n = 6
    arr = dict(x=np.arange(n) * 10.0, y=np.zeros(n), z=np.zeros(n),
               u=np.linspace(-1, 1, n), v=np.zeros(n), w=np.zeros(n),
               m=np.ones(n), h=np.full(n, 0.1), rho=np.ones(n), p=np.zeros(n),
               cs=np.ones(n))
    params = dict(c0=1.0, rho0=1.0, alpha=0.1, beta=0.0, gravity=(0.0, -9.81, 0.0),
                  dt=1e-3)
    eng = Engine([([arr], params)], fluid_scheme(1), dim=2, precision="fp64")
    for _ in range(100):
        eng.pc_step()
    t = 0.1
    np.testing.assert_allclose(eng.get(0, "x").cpu().numpy(), arr["x"] + arr["u"] * t,
                               rtol=0, atol=1e-12)
    np.testing.assert_allclose(eng.get(0, "y").cpu().numpy(), -0.5 * 9.81 * t * t, rtol=1e-10)


def test_nonfinite_position_reported_not_faulted():
    """A NaN position planted on the host is caught by the binning bounds
    checks and reported through the status word; nothing is written out of
    bounds and the context stays usable."""
    arrays, params, scheme, dim = drop(dx=0.1)
    arrays[0]["x"] = arrays[0]["x"].copy()
    arrays[0]["x"][3] = np.nan
    eng = Engine([(arrays, params)], scheme, dim=2, precision="fp64")
    st = eng.status()
    assert st & nat.ST_NONFINITE_POS
    eng.clear_status()
    assert eng.status() == 0
    torch.cuda.synchronize()


def _decisions(eng, steps):
    """Run pc_steps; per step the device's rebin decisions (start, mid)."""
    out = []
    for _ in range(steps):
        rec = {}
        eng.pc_step(on_half=lambda: rec.__setitem__("start", eng.rebin_count()))
        out.append((rec["start"], eng.rebin_count()))
    return out


def _assert_same_state(a, b, names=("x", "y", "u", "v", "rho"), tol=1e-10):
    for n in names:
        ga, gb = a.get(0, n).cpu().numpy(), b.get(0, n).cpu().numpy()
        assert np.max(np.abs(ga - gb)) <= tol * max(1.0, np.max(np.abs(gb))), n


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("case,margin,steps", [("dam", None, 60), ("drop", 0.02, 20)])
def test_list_reuse_matches_rebinning_pipeline(precision, case, margin, steps):
    """Lists kept across stages and steps (the device rebins once a particle
    has moved half the skin) evaluate the same pairs as rebinning every
    stage: trajectories agree to round-off (FP64) or to the FP32C
    trajectory bar, and both device decisions (keep, rebin) occur; the
    drop with a thin skin rebins on displacement mid-run."""
    arrays, params, scheme, dim = small_dam() if case == "dam" else drop(dx=0.1)
    if case == "drop":
        params = dict(params, dt=1e-5)   # c0 dt / h = 0.11
    a = Engine([(arrays, params)], scheme, dim=2, precision=precision, step_lists=True,
               skin_margin=margin)
    b = Engine([(arrays, params)], scheme, dim=2, precision=precision, step_lists=False)
    dec = _decisions(a, steps)
    for _ in range(steps):
        b.pc_step()
    a.check_status()
    b.check_status()
    flat = [d for pair in dec for d in pair]
    assert 0 in flat and 1 in flat, dec
    if case == "drop":
        assert 1 in flat[2:], dec   # a rebin after the first one
    # FP32C: the two pipelines sum in different orders, and the FP32 round-off
    # they differ by grows over the run; 1e-5 of the largest magnitude
    tol = 1e-10 if precision == "fp64" else 1e-5
    _assert_same_state(a, b, tol=tol)


def test_fast_motion_rebins_every_stage():
    """Particles that cross half the skin in one stage force a rebin at
    every decision, and the result still matches the rebinning pipeline."""
    arrays, params, scheme, dim = drop(dx=0.1)
    arrays[0]["u"] = arrays[0]["u"] * 20.0
    arrays[0]["v"] = arrays[0]["v"] * 20.0
    p = dict(params, dt=1e-5)
    a = Engine([(arrays, p)], scheme, dim=2, precision="fp64", step_lists=True,
               skin_margin=0.02)
    b = Engine([(arrays, p)], scheme, dim=2, precision="fp64", step_lists=False)
    dec = _decisions(a, 5)
    for _ in range(5):
        b.pc_step()
    a.check_status()
    # the first step starts where the engine's initial bin put the particles
    assert dec[0] == (0, 1) and all(d == (1, 1) for d in dec[1:]), dec
    _assert_same_state(a, b)


def test_state_written_from_host_forces_rebin():
    """exchange_in of positions between steps withdraws the lists: the next
    step rebins at its start, and the result matches the rebinning
    pipeline given the same write."""
    arrays, params, scheme, dim = small_dam()
    a = Engine([(arrays, params)], scheme, dim=2, precision="fp64", step_lists=True)
    b = Engine([(arrays, params)], scheme, dim=2, precision="fp64", step_lists=False)
    for e in (a, b):
        for _ in range(3):
            e.pc_step()
    x = a.get(0, "x").clone()
    x[:50] += 0.3 * 0.02
    for e in (a, b):
        e.exchange_in(0, "x", x)
    dec = _decisions(a, 2)
    for _ in range(2):
        b.pc_step()
    assert dec[0][0] == 1, dec
    _assert_same_state(a, b)


@pytest.mark.parametrize("case", ["dam", "drop"])
def test_graph_replay_matches_eager_steps(case):
    """One captured pc_step replayed N times equals N eager steps bit for
    bit: with list reuse the state never changes buffers, and inside the
    graph the rebin is a conditional node the device's decision opens or
    skips (the drop with a thin skin rebins every few stages, the dam keeps
    its lists)."""
    if case == "dam":
        arrays, params, scheme, dim = small_dam()
        kw = {}
    else:
        arrays, params, scheme, dim = drop(dx=0.1)
        params = dict(params, dt=1e-5)
        kw = dict(skin_margin=0.02)
    a = Engine([(arrays, params)], scheme, dim=2, precision="fp32c", **kw)
    b = Engine([(arrays, params)], scheme, dim=2, precision="fp32c", **kw)
    for e in (a, b):
        for _ in range(3):
            e.pc_step()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        a.pc_step()
        b.pc_step()
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.pc_step()
    rebins = 0
    for _ in range(20):
        g.replay()
        b.pc_step()
        rebins += b.rebin_count()
    torch.cuda.synchronize()
    a.check_status()
    b.check_status()
    if case == "drop":
        assert rebins > 0   # the replays took the rebin branch too
    # the capture itself runs nothing: both did 4 + 20 steps
    for n in ("x", "y", "u", "v", "rho", "p"):
        assert torch.equal(a.get(0, n), b.get(0, n)), n
    del g


def test_grid_overflow_reported():
    arrays, params, scheme, dim = drop(dx=0.1)
    eng = Engine([(arrays, params)], scheme, dim=2, precision="fp64",
                 cell_capacity=16)
    assert eng.status() & nat.ST_GRID_OVERFLOW
    torch.cuda.synchronize()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_continuity_list_reuse_matches_rebinning(precision):
    """The continuity scheme (lists recorded by a lists-only density pass,
    one pair pass for SPHDensityRate + momentum + XSPH) with kept lists
    against rebinning every stage."""
    from pysph_b200.engine import continuity_scheme
    arrays, params, _, dim = small_dam()
    sch = continuity_scheme(2, 0.5)
    a = Engine([(arrays, params)], sch, dim=2, precision=precision, step_lists=True)
    b = Engine([(arrays, params)], sch, dim=2, precision=precision, step_lists=False)
    dec = _decisions(a, 40)
    for _ in range(40):
        b.pc_step()
    a.check_status()
    b.check_status()
    flat = [d for pair in dec for d in pair]
    assert 0 in flat, dec
    tol = 1e-10 if precision == "fp64" else 1e-5
    _assert_same_state(a, b, tol=tol)
    for i in range(2):
        ra, rb = a.get(i, "rho").cpu().numpy(), b.get(i, "rho").cpu().numpy()
        assert np.max(np.abs(ra - rb)) <= tol * np.max(np.abs(rb)), i


def test_continuity_against_oracle_with_walls_and_ghosts():
    """FP64 engine against the oracle on the small dam break with the
    continuity scheme, one ghost particle (tag != 0) in the fluid."""
    from pysph_b200.engine import continuity_scheme
    from oracle import OracleArray, OracleSystem
    arrays, params, _, dim = small_dam()
    arrays[0]["tag"] = np.zeros(len(arrays[0]["x"]), np.int32)
    arrays[0]["tag"][7] = 1
    sch = continuity_scheme(2, 0.5)
    p = dict(params, cfl=0.0, dt=5e-5)
    eng = Engine([(arrays, p)], sch, dim=2, precision="fp64")
    oarrs = [OracleArray(f"a{i}", **{k: np.array(v, np.float64) for k, v in arr.items()
                                     if k != "tag"}, tag=arr.get("tag", np.zeros(len(arr["x"]))))
             for i, arr in enumerate(arrays)]
    osys = OracleSystem(oarrs, dim=2, rho_src={}, tait_on=sch.tait_on, mom_src=sch.mom_src,
                        step_on=sch.step_on, rate_src=sch.rate_src, xsph_src=sch.xsph_src,
                        xsph_eps=0.5, c0=params["c0"], rho0=params["rho0"],
                        alpha=params["alpha"], beta=params["beta"], eta=params["eta"],
                        gravity=tuple(params["gravity"]))
    for _ in range(5):
        eng.pc_step()
        osys.pc_step(5e-5)
    eng.check_status()
    for i in range(2):
        O = osys.arrays[i]
        for n in ("x", "y", "u", "v", "rho"):
            got = eng.get(i, n).cpu().numpy()
            ref = getattr(O, n)
            assert np.max(np.abs(got - ref)) <= 1e-10 * max(1.0, np.max(np.abs(ref))), (i, n)


@pytest.mark.parametrize("case,cont,integ", [("dam", False, "pc"), ("dam", True, "pc"),
                                             ("drop", False, "euler"), ("drop", True, "rk2")])
def test_fused_stage_matches_separate_pass(case, cont, integ):
    """The integrator stage in the force pass's epilogue (FP32C) against the
    same stage as its own pass: the same rates in the same arithmetic, so
    the states, the CFL time steps and the rebin decisions agree bit for
    bit."""
    from pysph_b200.engine import continuity_scheme
    arrays, params, scheme, dim = CASES[case]()
    if case == "drop":
        params = dict(params, dt=1e-5)   # the fixed dt the drop is stable at
    if cont:
        scheme = continuity_scheme(len(arrays), 0.5)
    a = Engine([(arrays, params)], scheme, dim=dim, precision="fp32c")
    b = Engine([(arrays, params)], scheme, dim=dim, precision="fp32c", fuse_stage=False)
    assert a.fuses_stage and not b.fuses_stage
    dts, rebins = [], 0
    for _ in range(30):
        a.step(integ)
        b.step(integ)
        rebins += a.rebin_count()
        assert a.rebin_count() == b.rebin_count()
        dts.append((a.scene_state()[0].dt, b.scene_state()[0].dt))
    a.check_status()
    b.check_status()
    assert all(x == y for x, y in dts)
    for i in range(len(arrays)):
        for n in ("x", "y", "u", "v", "rho", "p"):
            assert torch.equal(a.get(i, n), b.get(i, n)), (i, n)
    if case == "dam" and not cont:
        assert rebins > 0   # the rebin path ran too


def test_autotune_returns_a_timed_shape(tmp_path, monkeypatch):
    """The autotuner times the candidate shapes, then the skin on the best
    one, and caches the result per workload bucket (in a file when asked)."""
    from pysph_b200 import autotune as T
    monkeypatch.setenv("PYSPH_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    T._cache.clear()
    arrays, params, scheme, dim = drop(dx=0.05)
    scenes = [(arrays, dict(params, dt=1e-5))]
    kw = dict(lanes=(1, 2), blocks=(128,), stencils=(1,), steps=2, tiled=False)
    res = T.autotune(scenes, scheme, dim, "fp32c", **kw)
    assert res["lanes"] in (1, 2) and res["pair_block"] == 128 and res["stencil"] == 1
    assert res["skin_margin"] in T.SKINS and res["ms_per_step"] > 0
    assert len(res["table"]) == 2 + 1 + len(T.SKINS)
    assert (tmp_path / "tune.json").exists()
    again = T.autotune(scenes, scheme, dim, "fp32c", **kw)   # from the cache file
    assert {k: again[k] for k in ("lanes", "pair_block", "stencil", "skin_margin")} == \
        {k: res[k] for k in ("lanes", "pair_block", "stencil", "skin_margin")}
    T._cache.clear()


def test_autotune_times_the_shapes_that_it_reports(monkeypatch):
    """Every candidate runs as many threads per dest as its row says, and no
    two candidates but the repeated winner are the same program."""
    from pysph_b200 import autotune as T
    monkeypatch.delenv("PYSPH_B200_TUNE_CACHE", raising=False)
    T._cache.clear()
    ran = []
    time_steps = T.time_steps

    def spy(eng, *a, **k):
        ran.append((eng.pairs, eng._stencil, eng.desc.cfg.lanes, eng.pair_block, eng.skin_margin))
        return time_steps(eng, *a, **k)
    monkeypatch.setattr(T, "time_steps", spy)
    arrays, params, scheme, dim = drop(dx=0.05)
    res = T.autotune([(arrays, dict(params, dt=1e-5))], scheme, dim, "fp32c", blocks=(64, 128),
                     stencils=(1,), steps=2)
    T._cache.clear()
    rows = [(r["pairs"], r["stencil"], r["lanes"], r["pair_block"],
             r.get("skin_margin", 0.15)) for r in res["table"]]
    assert ran == rows and all(r["exact_lanes"] for r in res["table"])
    shapes = [r for r in rows[:-len(T.SKINS)]]
    assert len(shapes) - len(set(shapes)) <= 1
    assert {r[2] for r in shapes if r[0] == "lists"} == set(T.LANES)


def test_euler_step_graph_replays_like_eager_steps():
    """A captured Euler step (one stage) keeps the record copies in place, so
    its replays match eager steps."""
    arrays, params, scheme, dim = drop(dx=0.05)
    params = dict(params, dt=1e-5)
    a = Engine([(arrays, params)], scheme, dim=2, precision="fp32c")
    b = Engine([(arrays, params)], scheme, dim=2, precision="fp32c")
    for e in (a, b):
        e.step("euler")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.step("euler")
    for _ in range(5):
        g.replay()
        b.step("euler")
    torch.cuda.synchronize()
    a.check_status()
    b.check_status()
    for n in ("x", "y", "u", "v", "rho"):
        assert torch.equal(a.get(0, n), b.get(0, n)), n
    del g


def test_rk4_step_graph_replays_like_eager_steps():
    """A captured RK4 step (four fused stages, the record copies swapped
    four times) replays like eager steps, rebins and running sums
    included."""
    arrays, params, scheme, dim = drop(dx=0.05)
    params = dict(params, dt=1e-5)
    a = Engine([(arrays, params)], scheme, dim=2, precision="fp32c")
    b = Engine([(arrays, params)], scheme, dim=2, precision="fp32c")
    for e in (a, b):
        e.step("rk4")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.step("rk4")
    for _ in range(5):
        g.replay()
        b.step("rk4")
    torch.cuda.synchronize()
    a.check_status()
    b.check_status()
    for n in ("x", "y", "u", "v", "rho"):
        assert torch.equal(a.get(0, n), b.get(0, n)), n
    del g


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("cont", [False, True])
@pytest.mark.parametrize("lists", [True, False])
def test_rk4_against_oracle_with_walls(precision, cont, lists):
    """RK4 fused on the engine (stage kinds 4-7) on the dam break with walls,
    summation density or the continuity scheme with XSPH, 3 steps of fixed
    dt against the oracle's RK4Integrator.  Without list reuse every stage
    rebins, so the running sums ride through a rebin between every two
    stages."""
    arrays, _, params = W.dam_break(dx=0.05)
    params = dict(params, dt=1e-5, cfl=0.0)
    scheme = continuity_scheme(2, 0.5) if cont else fluid_scheme(2)
    eng = Engine([(arrays, params)], scheme, dim=2, precision=precision, step_lists=lists)
    osys = oracle_from(arrays, params, scheme, 2)
    for _ in range(3):
        eng.step("rk4")
        osys.step(1e-5, "rk4")
    eng.check_status()
    O = osys.arrays[0]
    tol = 1e-10 if precision == "fp64" else 2e-6
    for n in ("x", "y"):
        err = float(np.max(np.abs(eng.get(0, n).cpu().numpy() - getattr(O, n)))) / 0.05
        assert err <= tol, n
    for n in ("u", "v"):
        assert rel_err(eng.get(0, n).cpu().numpy(), getattr(O, n)) <= (
            1e-10 if precision == "fp64" else 2e-5), n
    for d in range(2):
        rho = eng.get(d, "rho").cpu().numpy()
        ref = osys.arrays[d].rho
        assert float(np.max(np.abs(rho - ref) / ref)) <= (
            1e-12 if precision == "fp64" else 1e-5), d


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_host_written_state_within_the_skin_keeps_the_lists(precision):
    """Positions and velocities written from the host: the engine refreshes
    the records and measures every displacement before its next decision,
    which keeps the lists while no particle has left half the skin (and
    rebins otherwise), with results matching the rebinning pipeline."""
    arrays, params, scheme, dim = small_dam()
    a = Engine([(arrays, params)], scheme, dim=2, precision=precision, step_lists=True)
    b = Engine([(arrays, params)], scheme, dim=2, precision=precision, step_lists=False)
    for e in (a, b):
        for _ in range(3):
            e.pc_step()
    skin = a._scene_host[0].skin_max
    x = a.get(0, "x").clone()
    u = a.get(0, "u").clone()
    x[:50] += 0.1 * skin
    u[:50] += 0.5
    for e in (a, b):
        e.exchange_in(0, "x", x)
        e.exchange_in(0, "u", u)
    dec = _decisions(a, 2)
    for _ in range(2):
        b.pc_step()
    assert dec[0][0] == 0, dec   # kept: nobody left half the skin
    tol = 1e-10 if precision == "fp64" else 1e-5
    _assert_same_state(a, b, tol=tol)
    # three skins: the measured displacement forces the rebin
    x = a.get(0, "x").clone()
    x[:5] += 3.0 * skin
    a.exchange_in(0, "x", x)
    assert _decisions(a, 1)[0][0] == 1


@pytest.mark.parametrize("case", ["dam", "lattice3d"])
@pytest.mark.parametrize("lists", [True, False])
def test_common_case_loops_match_the_general_loops(case, lists):
    """The pair passes compile the common case (one h in the scene, every
    source summed; the force pass per mode) apart from the general loops.
    Writing the same h back from the host marks the scene as having several
    h, which sends every pass through the general loops with arithmetic that
    is the same for equal h: three FP32C steps (lists kept, or the cells
    searched every stage) must agree bit for bit."""
    a, arrays, params, scheme, dim = engine_for(case, "fp32c", step_lists=lists)
    b, _, _, _, _ = engine_for(case, "fp32c", step_lists=lists)
    assert a.desc.cfg.lanes == b.desc.cfg.lanes == lanes_for(a.N, 1)
    for arr in range(b.A):
        b.exchange_in(arr, "h", torch.as_tensor(arrays[arr]["h"], dtype=torch.float64))
    assert not any(t.uniform_h for t in b._scene_host)
    for e in (a, b):
        e.rebin_now()
        for _ in range(3):
            e.pc_step()
        e.check_status()
    for arr in range(a.A):
        for n in ("x", "y", "u", "v", "rho", "p"):
            assert torch.equal(a.get(arr, n), b.get(arr, n)), (arr, n)
    assert a.pair_counts() == b.pair_counts()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_exchange_many_matches_single_exchanges(precision):
    """sphb_exchange_many (several properties of one array in one launch)
    moves the same values as one sphb_exchange per property, both ways, and
    leaves the engine in the same state: the imports of positions,
    velocities, rho and p followed by a PC step agree bit for bit."""
    engs = [engine_for("dam", precision)[0] for _ in range(2)]
    assert engs[0].user_n[0] > 0
    for eng in engs:
        for _ in range(3):
            eng.pc_step()
    names = ["x", "y", "u", "v", "rho", "p"]
    a = 0
    n = engs[0].user_n[a]
    outs1 = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in names]
    engs[0].exchange_out_many(a, names, outs1)
    outs2 = [engs[1].exchange_out(a, k) for k in names]
    for k, t1, t2 in zip(names, outs1, outs2):
        assert torch.equal(t1, t2), k
    # host-style edits imported back: all at once into one engine, one by
    # one into the other
    new = [t * (1.0 + 1e-4) if k in ("u", "v") else t.clone() for k, t in zip(names, outs1)]
    engs[0]._exchange_many(a, 0, list(zip(names, new)))
    for k, t in zip(names, new):
        engs[1].exchange_in(a, k, t)
    for eng in engs:
        eng.invalidate_box()
        eng._host_state = True
        eng.pc_step()
        eng.check_status()
    for k in names:
        assert torch.equal(engs[0].exchange_out(a, k), engs[1].exchange_out(a, k)), k
