"""The FP64 pair arithmetic (seeded reciprocals and reciprocal square roots
in place of divisions) to a few units in the last place: scenes of one pair
each, over six orders of magnitude of h and every distance within the
support, densities and accelerations against numpy."""
import math

import numpy as np
import pytest

from pysph_b200 import _native as nat
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
