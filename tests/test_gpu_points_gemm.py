"""FP64 basis products of point-set plans at the edges of their tiles: one to
a few more columns than one pass takes, point counts around the 16-row CTA,
basis sizes around the staged chunk and both analysis tilings, against the
oracle's dense basis.  Tolerance 1e-13 relative L2: sums of at most 2,562
terms in 64 bits (2^-53 sqrt(n) of normally distributed terms, the basis
recurrences' own 1e-14 included)."""
import numpy as np
import pytest
import torch

import oracle
from aeolus_gb300.ops import Plan, analyze, synthesize
from helpers import rel_l2, tri

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,L", [(15, 0), (16, 3), (17, 15), (162, 16), (401, 50), (2562, 20)])
@pytest.mark.parametrize("fields", [1, 2, 7, 8, 9, 17])
def test_fp64_basis_products(npts, L, fields):
    rng = np.random.default_rng(100 * npts + fields)
    lat = np.arcsin(rng.uniform(-1.0, 1.0, npts))
    lon = rng.uniform(-np.pi, np.pi, npts)
    w = rng.uniform(0.5, 1.5, npts) * (4.0 * np.pi / npts)
    ref = oracle.PointSetSH(lat, lon, L, weights=w)
    plan = Plan.points(lat, lon, w, L)
    a = tri(rng.standard_normal((fields, L + 1, L + 1)) + 1j * rng.standard_normal((fields, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    g = synthesize(plan.id, torch.as_tensor(a, device="cuda")).cpu().numpy()
    f = rng.standard_normal((fields, npts))
    c = analyze(plan.id, torch.as_tensor(f, device="cuda")).cpu().numpy()
    for i in range(fields):
        assert rel_l2(g[i], ref.inv_transform(a[i])) < 1e-13
        assert rel_l2(c[i], ref.transform(f[i])) < 1e-13
    plan.close()
