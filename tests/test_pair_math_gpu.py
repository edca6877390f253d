"""The FP64 pair arithmetic (seeded reciprocals and reciprocal square roots
in place of divisions): the functions themselves against 80-bit arithmetic, to
units in the last place; and scenes of one pair each, over six orders of
magnitude of h and every distance within the support, densities and
accelerations against numpy."""
import ctypes
import math

import numpy as np
import pytest
import torch

from pysph_b200 import _native as nat
from pysph_b200 import build
from pysph_b200.engine import Engine, fluid_scheme

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("thread_rule")]


@pytest.mark.parametrize("lists", [True, False])
def test_one_pair_per_scene(lists):
    rng = np.random.default_rng(11)
    S = 400
    h = 10.0 ** rng.uniform(-3, 3, S)
    q = rng.uniform(0.001, 1.9, S)   # (2 - q amplifies the last bits beyond)
    t = rng.uniform(0, 2 * math.pi, S)
    m = rng.uniform(0.5, 2.0, (S, 2))
    p = rng.uniform(1.0, 2.0, (S, 2))
    vel = rng.normal(0, 1, (S, 2, 2))
    scenes = []
    for s in range(S):
        x = np.array([0.0, q[s] * h[s] * math.cos(t[s])])
        y = np.array([0.0, q[s] * h[s] * math.sin(t[s])])
        z = np.zeros(2)
        scenes.append(([dict(x=x, y=y, z=z, u=vel[s, :, 0], v=vel[s, :, 1], w=z, m=m[s],
                             h=np.full(2, h[s]), rho=np.ones(2), p=p[s], cs=np.full(2, 3.0))],
                       dict(c0=3.0, rho0=1.0, gamma=7.0, alpha=0.1, beta=0.2, eta=0.1)))
    eng = Engine(scenes, fluid_scheme(1), dim=2, precision="fp64", use_lists=lists)
    dx = np.stack([-np.array([sc[0][0]["x"][1], sc[0][0]["y"][1]]) for sc in scenes])
    r = np.hypot(dx[:, 0], dx[:, 1])
    qq = r / h
    fac = 10.0 / (7.0 * math.pi) / h ** 2
    w = fac * np.where(qq <= 1, 1 - 1.5 * qq ** 2 * (1 - 0.5 * qq), 0.25 * (2 - qq) ** 3)
    g = fac * np.where(qq < 1, 3 * (0.75 * qq - 1) / h ** 2, -0.75 * (2 - qq) ** 2 / (h * r))
    mode = nat.FORCE_USE_LIST if lists else 0
    # the pressures given, unit densities: accelerations first
    eng.exchange_in(0, "rho", eng.get(0, "rho") * 0 + 1.0)
    eng.exchange_in(0, "p", eng.get(0, "p") * 0 + 1.0)
    eng.density(eos=False)
    rho = eng.get(0, "rho").view(S, 2).cpu().numpy()
    ref = fac[:, None] * m + w[:, None] * m[:, ::-1]
    assert np.max(np.abs(rho / ref - 1)) < 2e-15 * 4
    eng.momentum(gravity=False, mode=mode)
    acc = np.stack([eng.get(0, c).view(S, 2).cpu().numpy() for c in ("au", "av")], -1)
    dv = vel[:, 0] - vel[:, 1]
    dot = (dv * dx).sum(1)
    mu = h * dot / (r ** 2 + 0.01 * h ** 2)
    pi = np.where(dot < 0, (-0.1 * 3.0 * mu + 0.2 * mu ** 2) / (0.5 * rho.sum(1)), 0.0)
    tmp = (1.0 / rho ** 2).sum(1) + pi
    for a, sign in ((0, 1.0), (1, -1.0)):
        want = -(m[:, 1 - a] * tmp * g * sign)[:, None] * dx
        scale = np.abs(want).max(1, keepdims=True)
        # dot cancels where the velocity is nearly across the pair
        cond = 1 + np.linalg.norm(dv, axis=1) * r / np.maximum(np.abs(dot), 1e-300)
        cond = np.where(dot < 0, np.minimum(cond, 1e3), 1)[:, None]
        assert np.max(np.abs(acc[:, a] - want) / (scale * cond)) < 2e-14
    eng.check_status()


def _probe(which, a, b=None):
    fn = ctypes.CDLL(build.PROBE_LIB).sphb_math_probe
    p = ctypes.c_void_p
    fn.argtypes = [ctypes.c_int, ctypes.c_int, p, p, p, p, p]
    dev = torch.device("cuda", torch.cuda.current_device())
    a = torch.as_tensor(a, device=dev)
    b = None if b is None else torch.as_tensor(b, device=dev)
    out, out2 = torch.empty_like(a), torch.empty_like(a)
    assert fn(which, a.numel(), a.data_ptr(), None if b is None else b.data_ptr(),
              out.data_ptr(), out2.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    return out.cpu().numpy(), out2.cpu().numpy()


def _ulps(got, want):
    """Largest error in units in the last place (want: 80 bits, 11 more than
    the unit; its own rounding is 2^-12 of one)."""
    return float(np.max(np.abs(got.astype(np.longdouble) - want)
                        / np.spacing(np.abs(want.astype(np.float64)))))


def _numbers(rng, n, lo, hi):
    """Random mantissas and the ends of the mantissa's range, exponents of
    lo .. hi."""
    m = np.concatenate([rng.uniform(1, 2, n - 64), 1 + np.spacing(1.0) * np.arange(32),
                        2 - np.spacing(1.0) * np.arange(1, 33)])
    return np.ldexp(m, rng.integers(lo, hi, n))


def test_reciprocals_distances_and_quotients():
    """The seeds are within 2^-19 of the result (e below 2^-19, 2^-18 for the
    square root).  Reciprocal: half a unit of the last FMA and e^3 < 2^-57.
    Distance and its reciprocal: half a unit, half the rounding of t (at most
    half a unit more) and 5/16 e^3 < 2^-55.  Quotient: half a unit, the residual
    being exact and its own factor off by 2^-52 of it."""
    L = np.longdouble
    rng = np.random.default_rng(5)
    n = 1 << 20
    a = _numbers(rng, n, -300, 300)
    assert _ulps(_probe(0, a)[0], 1 / a.astype(L)) <= 0.5 + 2.0 ** -4 + 2.0 ** -10
    assert _ulps(_probe(0, -a)[0], -1 / a.astype(L)) <= 0.5 + 2.0 ** -4 + 2.0 ** -10
    r2 = _numbers(rng, n, -600, 600)
    r, ir = _probe(1, r2)
    s = np.sqrt(r2.astype(L))
    assert _ulps(r, s) <= 1.0 + 2.0 ** -2 + 2.0 ** -10
    assert _ulps(ir, 1 / s) <= 1.0 + 2.0 ** -2 + 2.0 ** -10
    h = _numbers(rng, n, -40, 40)
    x = h * rng.uniform(0.0, 3.0, n)
    assert _ulps(_probe(2, x, h)[0], x.astype(L) / h) <= 0.5 + 2.0 ** -10
    # a particle with itself: a finite reciprocal, a distance far below any h
    r, ir = _probe(1, np.zeros(1))
    assert 0 <= r[0] <= 1e-99 and np.isfinite(ir[0])


@pytest.mark.parametrize("hks", [False, True])
@pytest.mark.parametrize("lists", [True, False])
def test_one_pair_per_scene_of_two_smoothing_lengths(lists, hks):
    """The general pair loops: a reciprocal of h per pair.  About a dozen
    roundings stand in a density, here and in numpy's (36 units in the last
    place allowed); the accelerations (no viscosity) are those of the densities
    read back."""
    rng = np.random.default_rng(12)
    S = 400
    h = 10.0 ** rng.uniform(-3, 3, S)[:, None] * rng.uniform(0.8, 1.2, (S, 2))
    q = rng.uniform(0.001, 1.8, S)
    t = rng.uniform(0, 2 * math.pi, S)
    m = rng.uniform(0.5, 2.0, (S, 2))
    p = rng.uniform(1.0, 2.0, (S, 2))
    d = q * h.min(1)
    scenes = []
    for s in range(S):
        x = np.array([0.0, d[s] * math.cos(t[s])])
        y = np.array([0.0, d[s] * math.sin(t[s])])
        z = np.zeros(2)
        scenes.append(([dict(x=x, y=y, z=z, u=z, v=z, w=z, m=m[s], h=h[s], rho=np.ones(2),
                             p=p[s], cs=np.full(2, 3.0))],
                       dict(c0=3.0, rho0=1.0, gamma=7.0, alpha=0.0, beta=0.0, eta=0.1)))
    scheme = fluid_scheme(1)
    scheme.hks = hks
    eng = Engine(scenes, scheme, dim=2, precision="fp64", use_lists=lists, variable_h=True)
    dx = np.stack([-np.array([sc[0][0]["x"][1], sc[0][0]["y"][1]]) for sc in scenes])
    r = np.hypot(dx[:, 0], dx[:, 1])

    def kernel(hh, rr):
        qq, fac = rr / hh, 10.0 / (7.0 * math.pi) / hh ** 2
        w = fac * np.where(qq <= 1, 1 - 1.5 * qq ** 2 * (1 - 0.5 * qq),
                           0.25 * np.maximum(2 - qq, 0) ** 3)
        g = fac * np.where(qq < 1, 3 * (0.75 * qq - 1) / hh ** 2,
                           -0.75 * np.maximum(2 - qq, 0) ** 2 / (hh * np.maximum(rr, 1e-300)))
        return w, g
    if hks:
        (wa, ga), (wb, gb) = kernel(h[:, 0], r), kernel(h[:, 1], r)
        w, g = 0.5 * (wa + wb), 0.5 * (ga + gb)
    else:
        w, g = kernel(h.mean(1), r)
    own = kernel(h, np.zeros_like(h))[0]
    eng.density(eos=False)
    rho = eng.get(0, "rho").view(S, 2).cpu().numpy()
    ref = own * m + w[:, None] * m[:, ::-1]
    assert np.max(np.abs(rho / ref - 1)) < 2e-15 * 4
    eng.momentum(gravity=False, mode=1 | (nat.FORCE_USE_LIST if lists else 0))
    acc = np.stack([eng.get(0, c).view(S, 2).cpu().numpy() for c in ("au", "av")], -1)
    tmp = (p / rho ** 2).sum(1)
    # (2 - q amplifies the last bits near the edge of the support)
    cond = 1 + 2 / np.maximum(2 - r / h.mean(1), 0.05)
    for a, sign in ((0, 1.0), (1, -1.0)):
        want = -(m[:, 1 - a] * tmp * g * sign)[:, None] * dx
        scale = np.abs(want).max(1, keepdims=True)
        assert np.max(np.abs(acc[:, a] - want) / (scale * cond[:, None])) < 8e-15
    eng.check_status()
