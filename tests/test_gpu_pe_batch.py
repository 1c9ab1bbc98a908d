"""Batch limits of the one-call primitive-equation tendency: a point-set plan takes
every batch up to 65535 whatever its levels, a Gauss plan batch (K + 1) <= 65535,
as its grid rows do.  Members of a large batch equal those of a small one (1e-13
relative L2: the same sums)."""
from ctypes import byref, c_size_t, c_void_p

import numpy as np
import pytest
import torch

from aeolus_gb300 import _lib
from aeolus_gb300.ops import Plan

pytestmark = pytest.mark.gpu
L, K = 2, 1


def _points():
    rng = np.random.default_rng(3)
    lat, lon, w = np.arcsin(rng.uniform(-1, 1, 16)), rng.uniform(-np.pi, np.pi, 16), np.full(16, 4 * np.pi / 16)
    return Plan.points(lat, lon, w, L, 6.371e6)


def _tendency(plan, x):
    lib, B = _lib.load(), x.shape[0]
    nb, out = c_size_t(), torch.zeros_like(x)
    sig = np.array([0.0, 1.0])
    phis = torch.zeros((L + 1, L + 1), dtype=torch.complex128, device="cuda")
    prm = _lib.PeParams(6.371e6, 7.292e-5, 287.04, 1004.64)
    _lib.check(lib.aeolus_pe_workspace_bytes(plan.handle, K, B, byref(nb), None))
    w = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    p = lambda t: c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(lib.aeolus_pe_tendency(plan.handle, byref(prm), K, sig.ctypes.data_as(c_void_p), p(x), p(phis), p(out), B,
                                      p(w), w.numel(), None))
    torch.cuda.synchronize()
    return out


def _states(B):
    g = torch.Generator("cuda").manual_seed(1)
    x = torch.randn((B, 3 * K + 1, L + 1, L + 1), dtype=torch.complex128, device="cuda", generator=g).tril()
    x[..., 0] = x[..., 0].real.to(x.dtype)
    x[:, :2] *= 2e-6
    x[:, 2] *= 0.5
    x[:, 3] *= 1e-3
    x[:, 2, 0, 0] += 260.0
    return x


def test_point_set_takes_a_large_batch():
    plan, B = _points(), 33000
    x = _states(B)
    got = _tendency(plan, x)
    for lo in (0, B // 2, B - 3):
        want = _tendency(plan, x[lo:lo + 3].contiguous())
        for f in range(3 * K + 1):
            a, b = got[lo:lo + 3, f], want[:, f]
            assert float(torch.linalg.vector_norm(a - b)) <= 1e-13 * float(torch.linalg.vector_norm(b))
    plan.close()


def test_gauss_plan_refuses_one():
    plan = Plan.gauss(4, 8, L, 6.371e6)
    with pytest.raises(ValueError):
        _tendency(plan, _states(33000))
    assert torch.isfinite(torch.view_as_real(_tendency(plan, _states(32767)))).all()
    plan.close()
