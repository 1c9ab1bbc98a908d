"""Direct sums of FP64 rows (lengths without a 2/3/5 transform) add the many small
values of a row without a bias: one value of size 1 and all others near 2^-20 of
it, of one sign, whose low bits a sum that cuts them loses N times over.  Errors
in units of the large value:

* c2r, order 0 of 0.28 and 95 orders of 2^-20 of it: each order is rounded to
  2^-61 and counts twice (2^-53.4 in all at worst), the constant in the table may be
  off by 2^-54 and the result rounds by 2^-55: below 2^-52.
* r2c, a row of one 1 and N - 1 values near 2^-20: each is rounded to 2^-58 (2^-50.4
  in all), eight FP64 roundings of weights and table: below 2^-49."""
import math

import numpy as np
import pytest
import torch

from aeolus_gb300.ops import Plan, analyze, synthesize

pytestmark = pytest.mark.gpu
NLAT, L, ROW = 97, 95, 48  # row 48 is the equator: the basis there is known in closed form


def _pmm():
    p = [np.sqrt(np.longdouble(1) / (4 * np.arccos(np.longdouble(-1))))]
    for k in range(1, L + 1):
        p.append(-np.sqrt(np.longdouble(2 * k + 1) / np.longdouble(2 * k)) * p[-1])
    return np.array(p)


@pytest.mark.parametrize("nlon", [194, 191])
def test_small_orders_beside_a_large_one(nlon):
    plan, p, rng = Plan.gauss(NLAT, nlon, L), _pmm(), np.random.default_rng(nlon)
    t = 2.0 ** -20 * float(p[0]) * rng.uniform(0.5, 1.0, L)
    a = np.zeros((1, L + 1, L + 1), dtype=np.complex128)
    a[0, 0, 0] = 1.0
    for m in range(1, L + 1):
        a[0, m, m] = t[m - 1] / float(p[m])
    g = synthesize(plan.id, torch.as_tensor(a, device="cuda")).cpu().numpy().reshape(NLAT, nlon)[ROW]
    m = np.arange(1, L + 1)
    ang = (np.arange(nlon)[:, None] * m % nlon) * (2 * np.arccos(np.longdouble(-1)) / nlon)
    want = p[0] + 2 * (np.cos(ang) * (a[0, m, m].real * p[1:])).sum(-1)
    assert float(np.abs(g - want).max()) < 2.0 ** -52
    plan.close()


@pytest.mark.parametrize("nlon", [194, 191])
def test_small_points_beside_a_large_one(nlon):
    plan, rng = Plan.gauss(NLAT, nlon, L), np.random.default_rng(nlon)
    f = np.zeros((1, NLAT, nlon))
    f[0, ROW] = 2.0 ** -20 * rng.uniform(0.5, 1.0, nlon)
    f[0, ROW, 0] = 1.0
    a = analyze(plan.id, torch.as_tensor(f.reshape(1, -1), device="cuda"))[0].cpu().numpy()
    _, w = plan.nodes()
    want = float(_pmm()[0]) * w[ROW] * (2.0 * math.pi / nlon) * math.fsum(f[0, ROW])
    assert abs(a[0, 0].real / want - 1.0) < 2.0 ** -49
    plan.close()
