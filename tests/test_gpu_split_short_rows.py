"""Split-precision plans whose rows have fewer points than orders (half the row
below l_max): the direct DFT stages every order of a field.  Such rows alias the same
way in either precision, so transforms and the tendency agree with the FP64 plan's
within the split path's 1e-10."""
import numpy as np
import pytest
import torch

from helpers import rel_l2, tri

from aeolus_gb300 import _lib
from aeolus_gb300.ops import Plan, analyze, bve_tendency, synthesize

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlat,nlon,L", [(12, 10, 9), (16, 9, 12), (24, 12, 6), (20, 15, 18), (40, 5, 39), (12, 16, 8),
                                         (12, 16, 9), (130, 31, 120)])
@pytest.mark.parametrize("members", [1, 5])
def test_transforms_and_tendency(nlat, nlon, L, members):
    rng = np.random.default_rng(L)
    a = tri(rng.standard_normal((members, L + 1, L + 1)) + 1j * rng.standard_normal((members, L + 1, L + 1)))
    a[..., 0] = a[..., 0].real
    a[:, 0] = 0.0
    a, out = torch.as_tensor(a, device="cuda"), []
    f = torch.as_tensor(rng.standard_normal((members, nlat * nlon)), device="cuda")
    for split in (False, True):
        plan = Plan.gauss(nlat, nlon, L)
        if split:
            plan.set_precision(_lib.PREC_SPLIT_BF16)
        out.append([x.cpu().numpy() for x in (synthesize(plan.id, a), analyze(plan.id, f),
                                              bve_tendency(plan.id, 1.0, 0.5, 0.0, a, None))])
        plan.close()
    for x, y in zip(*out):
        assert rel_l2(y, x) < 1e-10
