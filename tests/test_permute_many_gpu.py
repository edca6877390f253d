"""sphb_permute_many and Engine.exchange_in_many against one call per buffer:
1 .. 8 buffers (and 9, two launches), both ways, two arrays."""
import pytest
import torch

from pysph_b200 import workloads as W
from pysph_b200.engine import Engine, fluid_scheme

pytestmark = pytest.mark.gpu


def _engine():
    arrays, _, params = W.dam_break(dx=0.1)
    return Engine([(arrays, params)], fluid_scheme(2), dim=2, precision="fp64")


@pytest.mark.parametrize("count", [1, 2, 7, 8, 9])
@pytest.mark.parametrize("array", [0, 1])
def test_permute_many(count, array):
    eng = _engine()
    eng.pc_step()
    n = eng.user_n[array]
    dev = eng.device
    g = torch.Generator(device=dev).manual_seed(count)
    user = torch.rand(count, n, dtype=torch.float64, device=dev, generator=g)
    inside = torch.zeros(count, eng.N, dtype=torch.float64, device=dev)
    eng.permute_many(array, 0, list(user), list(inside))
    one = torch.zeros(eng.N, dtype=torch.float64, device=dev)
    for i in range(count):
        one.zero_()
        eng.call("sphb_permute", eng.cur, array, 0, user[i].data_ptr(), one.data_ptr(),
                 eng.user_offset[array].data_ptr())
        assert torch.equal(one, inside[i])
    back = torch.zeros_like(user)
    eng.permute_many(array, 1, list(back), list(inside))
    assert torch.equal(back, user)


def test_exchange_in_many():
    a, b = _engine(), _engine()
    vals = {c: a.get(0, c) * 1.001 for c in ("x", "y", "u", "v")}
    a.exchange_in_many(0, list(vals.items()))
    # not contiguous: one exchange each
    b.exchange_in_many(0, [(c, torch.stack([v, v], 1)[:, 0]) for c, v in vals.items()])
    for e in (a, b):
        e.invalidate_box()
        e.pc_step()
        e.check_status()
    for c in ("x", "y", "u", "v", "rho"):
        assert torch.equal(a.get(0, c), b.get(0, c)), c
