"""A model whose tendency or step is its own (a subclass's, or one set on the
instance, as a forcing is added) is stepped with it, also on the way of a
checkpointed gradient."""
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import workloads as W
from aeolus_gb300.adjoint import swe_rk4_checkpointed
from aeolus_gb300.engine import rk4_step_device
from aeolus_gb300.primitive_equations import PrimitiveEquationsModel, SigmaGrid, isothermal_rest_state
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu
L, K = 9, 3


class Relaxed(PrimitiveEquationsModel):
    def tendency(self, coeffs):
        return super().tendency(coeffs) - 1e-4 * coeffs


@pytest.mark.parametrize("kind", ["subclass", "instance"])
def test_primitive_equations_rk4(kind):
    planet = ae.make_planet("latlon", nlat=16, nlon=32, l_max=L)
    m = (Relaxed if kind == "subclass" else PrimitiveEquationsModel)(planet, SigmaGrid.uniform(K))
    plain = PrimitiveEquationsModel(planet, SigmaGrid.uniform(K))
    if kind == "instance":
        m.tendency = lambda c: plain.tendency(c) - 1e-4 * c
    y = isothermal_rest_state(L, K, temperature=260.0, surface_pressure=101325.0).coeffs
    want = y
    for _ in range(2):
        want = rk4_step_device(lambda c: plain.tendency(c) - 1e-4 * c, want, 0.0, 300.0)
    got = m.rk4(y, 300.0, 2)
    assert torch.equal(got, want)
    assert not torch.equal(got, plain.rk4(y, 300.0, 2))


class Damped(ShallowWaterModel):
    def rk4(self, coeffs, dt, nsteps=1, check=True):
        return 0.75 * super().rk4(coeffs, dt, nsteps, check)


@pytest.mark.parametrize("kind", ["subclass", "instance"])
@pytest.mark.parametrize("nsteps,every", [(1, 1), (3, 8), (5, 2)])
def test_checkpointed_shallow_water(kind, nsteps, every):
    s0, depth = W.member_states(15, 2, seed=1)
    planet = ae.make_planet("latlon", nlat=24, nlon=48, l_max=15)
    m = (Damped if kind == "subclass" else ShallowWaterModel)(planet, gravity=W.GRAVITY, mean_depth=depth)
    plain = ShallowWaterModel(planet, gravity=W.GRAVITY, mean_depth=depth)
    if kind == "instance":
        m.rk4 = lambda c, dt, nsteps=1, check=True: 0.75 * plain.rk4(c, dt, nsteps, check)
    y = torch.as_tensor(s0, device="cuda").requires_grad_(True)
    want = y.detach()
    for _ in range(nsteps):
        want = 0.75 * plain.rk4(want, 120.0, 1)
    out = swe_rk4_checkpointed(m, y, 120.0, nsteps, every=every)
    assert torch.equal(out.detach(), want)
    (g,) = torch.autograd.grad((torch.view_as_real(out) ** 2).sum(), y)
    assert torch.isfinite(torch.view_as_real(g)).all()
