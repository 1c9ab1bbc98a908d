"""Analyses of which only the 2/3-rule triangle is kept: tendencies whose cut
leaves one or two degrees, one order pair without a partner, odd row counts and both
the FFT and the direct-DFT row lengths, against the oracle, on FP64 and split
plans; and the slots above the cut, which no contraction visits.  Tolerances:
the FP64 bound of the parity tests (1e-12) and the split bound (1e-10)."""
import numpy as np
import pytest
import torch

import oracle
from oracle import models as om

import aeolus_gb300 as ae
from aeolus_gb300 import _lib, workloads as W
from aeolus_gb300.barotropic import BarotropicState, BarotropicVorticity
from aeolus_gb300.shallow_water import ShallowWaterModel
from helpers import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlat,nlon,L", [(4, 8, 2), (6, 10, 3), (9, 16, 5), (17, 36, 11), (33, 64, 21), (64, 128, 42)])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("members", [1, 5])
def test_cut_tendencies(nlat, nlon, L, split, members):
    planet = ae.make_planet("latlon", nlat=nlat, nlon=nlon, l_max=L, product_quadrature="coarse")
    if split:
        planet.sh.plan.set_precision(_lib.PREC_SPLIT_BF16)
    tol = 1e-10 if split else 1e-12
    ops = oracle.Operators(oracle.GaussSH(nlat, nlon, L), W.EARTH_RADIUS)
    s0, depth = W.member_states(L, members, seed=3)
    swe = ShallowWaterModel(planet, gravity=W.GRAVITY, mean_depth=depth)
    ref = om.SWE(ops, W.EARTH_OMEGA, W.GRAVITY, depth)
    got = swe.tendency(torch.as_tensor(s0, device="cuda")).cpu().numpy()
    bve = BarotropicVorticity(planet, viscosity=1e5)
    zeta = bve.tendency(BarotropicState(torch.as_tensor(s0[:, 0].copy(), device="cuda"))).cpu().numpy()
    cut = (2 * L) // 3
    for b in range(members):
        want = ref.tendency(s0[b])
        for f in range(3):
            assert np.linalg.norm(got[b, f] - want[f]) <= tol * max(np.linalg.norm(want[f]), 1e-30)
        wz = om.bve_tendency(ops, s0[b, 0], W.EARTH_OMEGA, 1e5)
        assert rel_l2(zeta[b], wz) < tol
        # above the cut only the linear terms are left: d(delta)/dt = -lap phi, d(zeta)/dt = 0
        assert not got[b, 0, cut + 1:].any() and not got[b, 0, :, cut + 1:].any()
