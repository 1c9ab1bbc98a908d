"""Launch shapes and dispatch branches of FP64 plans that small batches and short
rows do not reach:

* several member rows per CTA of the row stage (8 of one field, 4 of two, 2 of four)
  with a last CTA that is not full, for every radix, and with a NaN, an infinity,
  zeros and far magnitudes among the grouped rows;
* direct sums that stage fewer fields than the functor has, and ones that read
  their twiddles from global memory;
* several members per CTA of the Legendre stage, and analyses of one order per CTA
  (rows too many for two orders' shared memory), with and without the 2/3 cut.

Transforms of one member do not depend on the shape (equal bit for bit); products
are alias-free in longitude on every grid used here, so another row length gives
the same tendency up to rounding (1e-13 relative L2, 1e-12 for the divergence,
whose largest term the Laplacian amplifies)."""
import math

import numpy as np
import pytest
import torch

import oracle
from helpers import rel_l2, tri
from oracle import models

from aeolus_gb300 import workloads as W
from aeolus_gb300.ops import Plan, analyze, bve_tendency, swe_tendency, synthesize, winds

pytestmark = pytest.mark.gpu
FFT = [(8, 3), (12, 5), (16, 7), (20, 8), (24, 11), (32, 10), (40, 13), (48, 15), (60, 9), (64, 21), (90, 12), (128, 20),
       (160, 18), (250, 14), (384, 21)]


def _rows_for(per_cta, members):
    """Latitude rows with which the row stage groups `per_cta` member rows."""
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    groups = -(-members // per_cta)
    nlat = -(-4 * sm // groups) + 1
    assert nlat * groups >= 4 * sm and members % per_cta
    return nlat


def _spectra(L, members, seed):
    rng = np.random.default_rng(seed)
    a = tri(rng.standard_normal((members, L + 1, L + 1)) + 1j * rng.standard_normal((members, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    return torch.as_tensor(a, device="cuda"), rng


@pytest.mark.parametrize("nlon,L", FFT)
def test_grouped_rows_of_one_field(nlon, L):
    members = 61
    plan = Plan.gauss(max(_rows_for(8, members), L + 1), nlon, L)
    a, rng = _spectra(L, members, nlon)
    f = torch.as_tensor(rng.standard_normal((members, plan.n_points)), device="cuda")
    g, c = synthesize(plan.id, a), analyze(plan.id, f)
    for i in (0, 1, 7, 8, 55, 56, 60):
        assert torch.equal(g[i], synthesize(plan.id, a[i:i + 1])[0])
        assert torch.equal(c[i], analyze(plan.id, f[i:i + 1])[0])
    plan.close()


@pytest.mark.parametrize("nlon,L", [(48, 15), (64, 21), (250, 14)])
def test_grouped_rows_keep_to_themselves(nlon, L):
    members = 61
    plan = Plan.gauss(max(_rows_for(8, members), L + 1), nlon, L)
    a, rng = _spectra(L, members, nlon)
    f = torch.as_tensor(rng.standard_normal((members, plan.n_points)), device="cuda")
    good = (synthesize(plan.id, a), analyze(plan.id, f))
    scale = {2: 1e-250, 3: 0.0, 5: 1e250, 57: 1e-250, 59: 0.0}
    for i, s in scale.items():
        a[i] *= s
        f[i] *= s
    a[4, 3, 2] = a[60, 5, 1] = complex(math.nan, 0.0)
    f[4, 5 * nlon + 3], f[60, 7 * nlon] = math.nan, math.inf
    g, c = synthesize(plan.id, a), analyze(plan.id, f)
    low = torch.ones((L + 1, L + 1), device="cuda").tril() > 0
    for i in range(members):
        if i in (4, 60):
            assert torch.isnan(g[i]).all() and not torch.isfinite(torch.view_as_real(c[i])[low]).any()
        elif i not in scale:
            assert torch.equal(g[i], good[0][i]) and torch.equal(c[i], good[1][i])
        elif scale[i] == 0.0:
            assert not g[i].any() and not c[i].any()
        else:
            assert rel_l2((g[i] / scale[i]).cpu(), good[0][i].cpu()) < 1e-13
            assert rel_l2((c[i] / scale[i]).cpu(), good[1][i].cpu()) < 1e-13
    plan.close()


@pytest.mark.parametrize("nlon,L", [(16, 5), (40, 13), (64, 21), (90, 12)])
def test_grouped_rows_of_two_and_four_fields(nlon, L):
    members = 29
    a, _ = _spectra(L, members, nlon)
    a[:, 0] = 0.0
    plan = Plan.gauss(max(_rows_for(4, members), (3 * L) // 2 + 1), nlon, L)
    uv = winds(plan.id, 1.0, a, None)
    for i in (0, 3, 4, 27, 28):
        assert rel_l2(uv[:, i].cpu(), winds(plan.id, 1.0, a[i:i + 1], None)[:, 0].cpu()) < 1e-13
    plan.close()
    plan = Plan.gauss(max(_rows_for(2, members), (3 * L) // 2 + 1), nlon, L)
    t = bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None)
    for i in (0, 1, 2, 27, 28):
        assert rel_l2(t[i].cpu(), bve_tendency(plan.id, 1.0, 0.5, 0.0, a[i:i + 1], None)[0].cpu()) < 1e-13
    plan.close()


def _swe(plan, y, depth):
    return swe_tendency(plan.id, W.EARTH_RADIUS, W.EARTH_OMEGA, W.GRAVITY, depth, 0.0, y, None).cpu().numpy()


def _close(got, want):
    for f, tol in enumerate((1e-13, 1e-12, 1e-13)):
        assert rel_l2(got[:, f], want[:, f]) < tol


@pytest.mark.parametrize("nlon", [614, 662, 661, 1618, 1814, 1813])
def test_long_direct_sums(nlon):
    L, nlat = 5, 8
    s0, depth = W.member_states(L, 2, seed=4)
    y = torch.as_tensor(s0, device="cuda")
    long, short = Plan.gauss(nlat, nlon, L, W.EARTH_RADIUS), Plan.gauss(nlat, 64, L, W.EARTH_RADIUS)
    _close(_swe(long, y, depth), _swe(short, y, depth))
    long.close()
    short.close()


@pytest.mark.parametrize("nlon", [1226, 1262, 3502, 3538])
def test_long_direct_sums_of_four_fields(nlon):
    L, nlat = 5, 8
    a, _ = _spectra(L, 2, 7)
    a[:, 0] = 0.0
    out = []
    for n in (nlon, 64):
        plan = Plan.gauss(nlat, n, L)
        out.append(bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None).cpu().numpy())
        plan.close()
    assert rel_l2(*out) < 1e-13


@pytest.mark.parametrize("nlat,nlon,L", [(9, 8, 3), (24, 48, 15), (65, 24, 11), (36, 72, 23)])
def test_members_per_legendre_cta(nlat, nlon, L):
    plan, members = Plan.gauss(nlat, nlon, L), 7
    a, rng = _spectra(L, members, nlat)
    f = torch.as_tensor(rng.standard_normal((members, plan.n_points)), device="cuda")
    g, c = synthesize(plan.id, a), analyze(plan.id, f)
    t = bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None)
    for bc in (1, 2, 3, 4, 7):
        plan.set_tuning((bc, bc, 0, 0, 0))
        assert torch.equal(synthesize(plan.id, a), g) and torch.equal(analyze(plan.id, f), c)
        assert torch.equal(bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None), t)
    plan.close()


@pytest.mark.parametrize("nlat", [7264, 7301])
def test_one_order_per_analysis_cta(nlat):
    L, nlon = 3, 12
    plan = Plan.gauss(nlat, nlon, L)
    a, _ = _spectra(L, 2, nlat)
    assert rel_l2(analyze(plan.id, synthesize(plan.id, a)).cpu(), a.cpu()) < 1e-12
    a[:, 0] = 0.0
    few = Plan.gauss(8, nlon, L)
    assert rel_l2(bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None).cpu(), bve_tendency(few.id, 1.0, 0.5, 0.0, a, None).cpu()) < 1e-12
    few.close()
    plan.close()


@pytest.mark.parametrize("nlat", [1818, 1901])
def test_one_order_per_analysis_cta_of_four_fields(nlat):
    L, nlon = 5, 16
    s0, depth = W.member_states(L, 2, seed=4)
    plan = Plan.gauss(nlat, nlon, L, W.EARTH_RADIUS)
    got = _swe(plan, torch.as_tensor(s0, device="cuda"), depth)
    # the quotients by cos^2 of truncated fields are no polynomials: the same rows
    # (and the plan's nodes: numpy's weights of so many are 5e-8 off next to a pole)
    lat, w = plan.nodes()
    sh = oracle.PointSetSH(np.repeat(lat, nlon), np.tile(np.arange(nlon) * (2.0 * np.pi / nlon), nlat), L,
                           weights=np.repeat(w, nlon) * (2.0 * np.pi / nlon))
    ref = models.SWE(oracle.Operators(sh, W.EARTH_RADIUS), W.EARTH_OMEGA, W.GRAVITY, depth)
    for b in range(2):
        want = ref.tendency(s0[b])
        for f in range(3):
            assert rel_l2(got[b, f], want[f]) < 1e-11
    plan.close()


def test_each_order_at_its_own_magnitude():
    L = 15
    plan = Plan.gauss(24, 48, L)
    a, _ = _spectra(L, L + 1, 5)
    scale = 10.0 ** np.linspace(-200, 200, L + 1)
    for m in range(L + 1):  # member m: order m alone
        a[m, :, :m] = 0.0
        a[m, :, m + 1:] = 0.0
    back = analyze(plan.id, synthesize(plan.id, a * torch.as_tensor(scale, device="cuda")[:, None, None]))
    for m in range(L + 1):
        assert rel_l2((back[m] / scale[m]).cpu(), a[m].cpu()) < 1e-13
    plan.close()
