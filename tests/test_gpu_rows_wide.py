"""Row stage of FP64 plans at the row lengths where it changes: every radix of
the 96-bit transforms, one and several member rows per CTA with a last CTA that
is not full, and direct sums (odd, prime and twice-prime lengths, a length
whose even middle point stands alone, orders at and above half the length),
against the reference's dense basis on the same points; rows far from 1 in
magnitude, a row of zeros, and a NaN, which stays in its row and member.
Tolerance 1e-13 relative L2 (sums of at most 8,000 terms in 64 bits)."""
import numpy as np
import pytest
import torch

import oracle
from aeolus_gb300.ops import Plan, analyze, synthesize
from helpers import rel_l2, tri

pytestmark = pytest.mark.gpu
FFT = [(8, 3), (12, 5), (16, 7), (20, 8), (24, 11), (32, 10), (40, 13), (48, 15), (60, 9), (64, 21), (90, 12), (128, 20),
       (160, 18), (250, 14), (384, 21)]
DFT = [(5, 2), (7, 3), (14, 4), (23, 7), (22, 10), (31, 15), (46, 15), (61, 20), (94, 21), (190, 16), (382, 12),
       (12, 6), (10, 9), (9, 12)]


def _setup(nlat, nlon, L, members, seed):
    plan = Plan.gauss(nlat, nlon, L)
    lat, w = plan.nodes()
    pl, po = np.repeat(lat, nlon), np.tile(np.arange(nlon) * (2.0 * np.pi / nlon), nlat)
    ref = oracle.PointSetSH(pl, po, L, weights=np.repeat(w, nlon) * (2.0 * np.pi / nlon))
    rng = np.random.default_rng(seed)
    a = tri(rng.standard_normal((members, L + 1, L + 1)) + 1j * rng.standard_normal((members, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    return plan, ref, a, rng.standard_normal((members, nlat * nlon))


def T(x):
    return torch.as_tensor(np.ascontiguousarray(x), device="cuda")


@pytest.mark.parametrize("nlon,L", FFT + DFT)
@pytest.mark.parametrize("members", [1, 13])
def test_rows(nlon, L, members):
    nlat = max(5, L + 1) if members == 1 else 97  # 13 members on 97 rows: eight member rows per CTA
    if members > 1 and nlon > 64:
        nlat = 50
    plan, ref, a, f = _setup(nlat, nlon, L, members, 7 * nlon + L)
    g = synthesize(plan.id, T(a)).cpu().numpy()
    c = analyze(plan.id, T(f)).cpu().numpy()
    for i in (0, members // 2, members - 1):
        assert rel_l2(g[i], ref.inv_transform(a[i])) < 1e-13
        assert rel_l2(c[i], ref.transform(f[i])) < 1e-13
    plan.close()


@pytest.mark.parametrize("nlon,L", [(48, 15), (64, 21), (46, 15), (61, 20)])
def test_magnitudes_zeros_and_nan(nlon, L):
    nlat, members = 24, 9
    plan, ref, a, f = _setup(nlat, nlon, L, members, nlon)
    scale = np.array([1e-250, 1e-30, 1.0, 1e30, 1e250, 0.0, 1.0, 1.0, 1.0])
    a *= scale[:, None, None]
    f *= scale[:, None]
    a[7, 3, 2] = np.nan
    f[7, 5 * nlon + 3] = np.nan
    f[8, 5 * nlon + 3] = np.inf
    g = synthesize(plan.id, T(a)).cpu().numpy()
    c = analyze(plan.id, T(f)).cpu().numpy()
    for i in range(members):
        if i == 7:
            assert np.isnan(g[i]).all()
        elif scale[i] == 0.0:
            assert not g[i].any() and not c[i].any()
        else:
            assert rel_l2(g[i] / scale[i], ref.inv_transform(a[i] / scale[i])) < 1e-13
        if i in (7, 8):
            low = np.tril(np.ones((L + 1, L + 1), bool))
            assert not np.isfinite(c[i][low]).any()
        elif scale[i] != 0.0:
            assert rel_l2(c[i] / scale[i], ref.transform(f[i] / scale[i])) < 1e-13
    plan.close()
