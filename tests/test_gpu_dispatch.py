"""Every device call of a checkpointed gradient goes through the dispatcher as an
operator of the aeolus namespace, kept stage inputs included, so that dispatch-level
tools see the whole path: forward steps, kept steps and step adjoints."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import aeolus_gb300 as ae
from aeolus_gb300 import workloads as W
from aeolus_gb300.adjoint import swe_rk4_checkpointed
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu


class Calls(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if func.namespace == "aeolus":
            self.names.append(func._opname)
        return func(*args, **(kwargs or {}))


def test_checkpointed_gradient():
    s0, depth = W.member_states(15, 2, seed=1)
    m = ShallowWaterModel(ae.make_planet("latlon", nlat=24, nlon=48, l_max=15), gravity=W.GRAVITY, mean_depth=depth)
    y = torch.as_tensor(s0, device="cuda").requires_grad_(True)
    with Calls() as calls:
        out = swe_rk4_checkpointed(m, y, 120.0, 5, every=3)
        forward = list(calls.names)
        out.backward(torch.ones_like(out))  # the mode is this thread's: the backward runs on the device's own
    assert forward == ["swe_rk4"] * 3 + ["swe_rk4_stages"] * 2
    for op in ("swe_rk4_stages", "swe_rk4_adjoint_stages"):
        assert getattr(torch.ops.aeolus, op).default._schema.is_mutable is False
