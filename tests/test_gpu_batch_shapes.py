"""Launch shapes that depend on the batch: threads per latitude row (rows that
leave SMs idle take more), members per slicing CTA, and columns that pad the
last data tile, which nothing writes (the scratch is filled with NaN first).
Every sum is exact integers or one fixed order, so a member of a batch has to
equal the same member alone bit for bit."""
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import _lib, workloads as W
from aeolus_gb300.barotropic import BarotropicState, BarotropicVorticity
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu


def _poison():
    x = torch.full((1 << 25,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    del x


@pytest.mark.parametrize("nlat,nlon,L", [(20, 36, 11), (32, 64, 21), (64, 128, 42), (90, 192, 63), (128, 256, 85),
                                         (150, 320, 100), (192, 384, 127)])
@pytest.mark.parametrize("split", [False, True])
def test_members_alone_and_in_batches(nlat, nlon, L, split):
    planet = ae.make_planet("latlon", nlat=nlat, nlon=nlon, l_max=L, product_quadrature="coarse")
    if split:
        planet.sh.plan.set_precision(_lib.PREC_SPLIT_BF16)
    s0, depth = W.member_states(L, 23, seed=11)
    s0 = torch.as_tensor(s0, device="cuda")
    swe = ShallowWaterModel(planet, gravity=W.GRAVITY, mean_depth=depth)
    bve = BarotropicVorticity(planet, viscosity=1e5)

    def run(lo, hi):
        _poison()
        y = swe.rk4(s0[lo:hi].clone(), 60.0, 1)
        return swe.tendency(y), y, bve.tendency(BarotropicState(s0[lo:hi, 0].contiguous()))

    alone = [run(b, b + 1) for b in (0, 1, 6, 22)]
    for lo, hi in [(0, 2), (0, 3), (1, 7), (0, 11), (0, 23)]:
        got = run(lo, hi)
        assert all(torch.isfinite(torch.view_as_real(g)).all() for g in got)
        for b, one in zip((0, 1, 6, 22), alone):
            if lo <= b < hi:
                for g, o in zip(got, one):
                    assert torch.equal(g[b - lo], o[0])
