"""FP64 Legendre sums keep FP64's accuracy row by row and degree by degree, not
only in the norm of a field.

* A field of one coefficient a_mm: every row is sin^m(colatitude) times a cosine,
  down to 1e-70 of the equator's value next to the poles.  The table forms P_mm as m
  factors of four roundings each, from a sine that next to a pole may lose
  2^-53 / sin^2 by its square-root form; a twentieth of that is allowed (320
  roundings per factor at the row nearest the pole, sin = 0.0125).  A row's
  relative error against nodes and products in extended precision stays below
  (m + 2) 2^-53 (8 + 0.05 / sin^2).
* The transpose: an analysis of data in one row gives a_lm = P_lm G, to the same
  relative bound for l = m.
* Coefficients that fall by 25 decades in degree within one order: the rows see
  their largest coefficients, so the field is as accurate as one of those alone."""
import math

import numpy as np
import pytest
import torch

from aeolus_gb300.ops import Plan, analyze, synthesize

pytestmark = pytest.mark.gpu
NLAT, NLON, L = 192, 384, 127
EPS = 2.0 ** -53


def _nodes():
    """cos and sin of the colatitudes, north to south, in extended precision."""
    t = np.longdouble
    x = np.cos((np.arange(NLAT, dtype=t) + t(0.75)) / (t(NLAT) + t(0.5)) * np.arccos(t(-1)))
    for _ in range(10):
        p0, p1 = np.ones_like(x), x
        for l in range(2, NLAT + 1):
            p0, p1 = p1, ((2 * l - 1) * x * p1 - (l - 1) * p0) / t(l)
        x = x - p1 * (x * x - 1) / (NLAT * (x * p1 - p0))
    return x, np.sqrt((1 - x) * (1 + x))


X, S = _nodes()


def _pmm(m):
    t = np.longdouble
    p = np.full(NLAT, np.sqrt(1 / (4 * np.arccos(t(-1)))))
    for k in range(1, m + 1):
        p = -np.sqrt(t(2 * k + 1) / t(2 * k)) * S * p
    return p


def _bound(m):
    return EPS * (m + 2) * (8.0 + 0.05 / S.astype(np.float64) ** 2)


@pytest.fixture(scope="module")
def plan():
    p = Plan.gauss(NLAT, NLON, L)
    yield p
    p.close()


@pytest.mark.parametrize("m", [1, 5, 20, 40])
@pytest.mark.parametrize("members", [1, 9])
def test_rows_of_one_coefficient(plan, m, members):
    a = torch.zeros((members, L + 1, L + 1), dtype=torch.complex128, device="cuda")
    a[:, m, m] = 1.0
    g = synthesize(plan.id, a).cpu().numpy().reshape(members, NLAT, NLON)
    want = 2.0 * _pmm(m).astype(np.float64)[:, None] * np.cos((m * np.arange(NLON) % NLON) * (2.0 * np.pi / NLON))
    err = np.linalg.norm(g - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert (err < _bound(m)).all()


@pytest.mark.parametrize("m", [1, 5, 20, 40])
@pytest.mark.parametrize("row", [0, 12, 95])
def test_coefficients_of_one_row(plan, m, row):
    _, w = plan.nodes()
    f = torch.zeros((1, NLAT, NLON), dtype=torch.float64, device="cuda")
    f[0, row] = torch.as_tensor(np.cos((m * np.arange(NLON) % NLON) * (2.0 * np.pi / NLON)))
    a = analyze(plan.id, f.reshape(1, -1))[0].cpu().numpy()
    want = float(_pmm(m)[row]) * w[row] * math.pi
    assert abs(a[m, m] - want) < _bound(m)[row] * abs(want) + 8 * EPS * abs(want)


def test_coefficients_that_fall_with_degree(plan):
    m = 12
    a = torch.zeros((1, L + 1, L + 1), dtype=torch.complex128, device="cuda")
    fall = torch.pow(10.0, -0.25 * torch.arange(L + 1 - m, dtype=torch.float64, device="cuda"))
    a[0, m:, m] = fall * (1.0 + 0.5j)
    g = synthesize(plan.id, a).cpu().numpy().reshape(NLAT, NLON)
    # the same sums from a table formed by the recurrence in extended precision
    total, p2, p1, h = np.zeros(NLAT, np.longdouble), np.zeros(NLAT, np.longdouble), _pmm(m), fall.cpu().numpy()
    size = np.zeros(NLAT)
    for l in range(m, L + 1):
        if l > m:
            n = np.longdouble(l)
            ca = np.sqrt((4 * n * n - 1) / (n * n - m * m))
            cb = np.sqrt(((n - 1) ** 2 - m * m) / (4 * (n - 1) ** 2 - 1))
            p2, p1 = p1, ca * (X * p1 - cb * p2)
        total += h[l - m] * p1
        size += np.abs((h[l - m] * p1).astype(np.float64))
    ang = (m * np.arange(NLON) % NLON) * (2.0 * np.pi / NLON)
    want = 2.0 * total.astype(np.float64)[:, None] * (np.cos(ang) - 0.5 * np.sin(ang))
    err = np.abs(g - want).max(-1) / (2.0 * size * math.hypot(1.0, 0.5))
    assert (err < 4.0 * _bound(m)).all()
