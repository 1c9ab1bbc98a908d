"""Legendre sums of FP64 plans where their launch shape or arithmetic changes:
rows per warp 8, 16 and 32 with rows left over, one and two columns per thread
with a column left over, one to many lanes per analysed degree, sums across a
flush of the 64-bit totals, a middle row, one order per CTA (more rows than two
orders' shared memory holds); then columns far from 1, zero columns and a NaN,
which stays in its order and member.  Against the reference's dense basis; the
tolerance is 1e-13 relative L2 (sums of at most 500 terms in 64 bits)."""
import numpy as np
import pytest
import torch

import oracle
from aeolus_gb300.ops import Plan, analyze, synthesize
from helpers import rel_l2, tri

pytestmark = pytest.mark.gpu


def T(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda")


def _setup(nlat, nlon, L, members, seed):
    plan = Plan.gauss(nlat, nlon, L)
    lat, w = plan.nodes()
    pl, po = np.repeat(lat, nlon), np.tile(np.arange(nlon) * (2.0 * np.pi / nlon), nlat)
    ref = oracle.PointSetSH(pl, po, L, weights=np.repeat(w, nlon) * (2.0 * np.pi / nlon))
    rng = np.random.default_rng(seed)
    a = tri(rng.standard_normal((members, L + 1, L + 1)) + 1j * rng.standard_normal((members, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    return plan, ref, a, rng.standard_normal((members, nlat * nlon))


@pytest.mark.parametrize("nlat,nlon,L,members", [
    (2, 4, 1, 3), (3, 4, 1, 1), (9, 8, 3, 5), (16, 16, 7, 1), (17, 16, 7, 4), (31, 16, 7, 3), (34, 16, 7, 40),
    (63, 16, 5, 7), (65, 24, 11, 130), (35, 72, 33, 2), (36, 72, 31, 2), (66, 136, 65, 1), (97, 24, 8, 33),
    (300, 12, 5, 2), (1001, 8, 3, 1), (2600, 8, 3, 1), (5001, 8, 2, 2)])
def test_shapes(nlat, nlon, L, members):
    plan, ref, a, f = _setup(nlat, nlon, L, members, 3 * nlat + L)
    g = synthesize(plan.id, T(a)).cpu().numpy()
    c = analyze(plan.id, T(f)).cpu().numpy()
    for i in {0, members // 2, members - 1}:
        assert rel_l2(g[i], ref.inv_transform(a[i])) < 1e-13
        assert rel_l2(c[i], ref.transform(f[i])) < 1e-13
    plan.close()


def test_magnitudes_zeros_and_nan():
    nlat, nlon, L = 24, 48, 15
    plan, ref, a, f = _setup(nlat, nlon, L, 6, 5)
    cols = 10.0 ** np.linspace(-200, 200, L + 1)  # one magnitude per order
    a[1] *= cols[None, :]
    a[2, :, 4] = 0.0
    a[3, 9, 6] = np.nan
    a[4] *= 1e-300  # partly subnormal
    a[5, :, ::2] = 0.0
    back = analyze(plan.id, synthesize(plan.id, T(a[[0, 2, 4, 5]])))
    for i, k in enumerate((0, 2, 4, 5)):
        unit = 1e-300 if k == 4 else 1.0
        assert rel_l2(back[i].cpu().numpy() / unit, a[k] / unit) < 1e-13
    g = synthesize(plan.id, T(a)).cpu().numpy()
    assert rel_l2(g[1] / 1e200, ref.inv_transform(a[1] / 1e200)) < 1e-13
    assert np.isnan(g[3]).all()
    for i in (0, 2, 5):
        assert rel_l2(g[i], ref.inv_transform(a[i])) < 1e-13
    plan.close()
