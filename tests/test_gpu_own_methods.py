"""A model whose tendency is its own (a subclass's, or one set on the instance,
as a forcing is added) is stepped with it."""
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300.engine import rk4_step_device
from aeolus_gb300.primitive_equations import PrimitiveEquationsModel, SigmaGrid, isothermal_rest_state

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
