"""Row stages of FP64 plans whose dynamic shared memory alone fits the 48 KB that
need no attribute, but not together with the kernel's static per-CTA scalars:
direct sums of 4 fields on 614 points (49,120 + 48 bytes) and 5 on 511 (49,096 +
60), lengths next to them, and the grouped row kernel, which holds the scalars of
several bodies, around 450 points (9 fields: 48,816 bytes).  The products are alias-free on each grid, so
another row length gives the same result up to rounding: 1e-13 relative L2."""
import numpy as np
import pytest
import torch

from helpers import rel_l2, tri

import aeolus_gb300 as ae
from aeolus_gb300 import workloads as W
from aeolus_gb300.ensemble import ShallowWaterEnsemble
from aeolus_gb300.ops import Plan, bve_tendency, bve_tendency_adjoint
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu
L, NLAT = 7, 12


def _spectra(seed):
    rng = np.random.default_rng(seed)
    a = tri(rng.standard_normal((2, L + 1, L + 1)) + 1j * rng.standard_normal((2, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    a[:, 0] = 0.0
    return torch.as_tensor(a, device="cuda")


@pytest.mark.parametrize("nlon", [610, 612, 614, 616, 618])
def test_direct_sums_of_a_tendency(nlon):
    z, out = _spectra(1), []
    for n in (nlon, 640):
        plan = Plan.gauss(NLAT, n, L)
        out.append(bve_tendency(plan.id, 1.0, 0.5, 0.0, z, None).cpu().numpy())
        plan.close()
    assert rel_l2(*out) < 1e-13


@pytest.mark.parametrize("nlon", [509, 511, 513])
def test_direct_sums_of_an_adjoint(nlon):
    z, q, out = _spectra(1), _spectra(2), []
    for n in (nlon, 512):
        plan = Plan.gauss(NLAT, n, L)
        out.append(bve_tendency_adjoint(plan.id, 1.0, 0.5, 0.0, z, q).cpu().numpy())
        plan.close()
    assert rel_l2(*out) < 1e-13


@pytest.mark.parametrize("nlon", [432, 450, 480])
def test_grouped_rows(nlon):
    s0, depth = W.member_states(L, 3, seed=3)
    y = torch.as_tensor(s0, device="cuda")
    models = [ShallowWaterModel(ae.make_planet("latlon", nlat=NLAT, nlon=n, l_max=L), gravity=W.GRAVITY, mean_depth=depth)
              for n in (nlon, 64)]
    assert models[0]._plan.nlon == nlon
    want = [m.rk4(y, 300.0, 1) for m in models]
    states = [y.clone(), y.clone()]
    ShallowWaterEnsemble(models, [3, 3]).rk4(states, 300.0, 1)
    for a, b in zip(states, want):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-13
