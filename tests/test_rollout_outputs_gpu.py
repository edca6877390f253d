"""A rollout's outputs are tensors of their own: a program may change them in
place, under autograd too, without touching another output."""
import numpy as np
import pytest
import torch

from pysph_b200 import workloads as W
from pysph_b200.adjoint import Rollout, RolloutFunction
from pysph_b200.engine import fluid_scheme

pytestmark = pytest.mark.gpu


def _rollout():
    arrays, _, params = W.elliptical_drop(dx=0.1)
    r = Rollout(arrays, params, fluid_scheme(1), dim=2, dt=1e-5, steps=4, checkpoint_every=2)
    v0 = torch.tensor(np.stack([arrays[0]["u"], arrays[0]["v"]]), device="cuda")
    return r, v0


def test_positions_can_be_modified_in_place_under_autograd():
    r, v0 = _rollout()
    grads = []
    for inplace in (False, True):
        v = v0.clone().requires_grad_(True)
        x = RolloutFunction.apply(v, r)
        if inplace:
            x -= 0.5
            x.mul_(2.0)
        else:
            x = (x - 0.5) * 2.0
        (x ** 2).sum().backward()
        grads.append(v.grad)
    assert torch.equal(grads[0], grads[1])


def test_states_and_gradients_do_not_share_memory():
    r, v0 = _rollout()
    X, V = r.forward({0: v0})[0]
    lX, lV = r.vjp_F({0: (X, V)}, {0: torch.ones_like(X)})[0]
    r.adj.check_status()
    for a, b in ((X, V), (lX, lV)):
        assert a.untyped_storage().data_ptr() != b.untyped_storage().data_ptr()
        before = b.clone()
        a.zero_()
        assert torch.equal(b, before)
