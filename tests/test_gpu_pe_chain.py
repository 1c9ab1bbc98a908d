"""The one-call primitive-equation tendency and RK4 (aeolus_pe_tendency,
aeolus_pe_rk4) against the composition of the single calls it fuses
(aeolus_pe_derive, synthesis, aeolus_pe_columns, analysis, weak-form curl/div on
the extended plan, aeolus_pe_spectral): one level, level counts around the
eight warps of a column CTA, the largest, point counts that leave the last CTA
part empty, ragged rows, point sets, one degree left by the 2/3 cut; FP64 and
split precision.  Tolerance per prognostic block: 1e-12 relative L2 in FP64
(the same sums in another order), 1e-10 split."""
from ctypes import byref, c_void_p

import numpy as np
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import _lib
from aeolus_gb300._lib import check
from aeolus_gb300.engine import rk4_step_device
from aeolus_gb300.ops import analyze, synthesize, vector_curl_div
from aeolus_gb300.primitive_equations import PrimitiveEquationsModel, SigmaGrid, isothermal_rest_state

pytestmark = pytest.mark.gpu


def _composed(m, x):
    K, n, B = m.nlev, m.l_max + 1, x.shape[0]
    lib, st, plan = _lib.load(), c_void_p(torch.cuda.current_stream().cuda_stream), m._plan
    p = lambda t: c_void_p(t.data_ptr())  # noqa: E731
    sig = m._sigma_host.ctypes.data_as(c_void_p)
    f = torch.empty((B, 10 * K + 2, n, n), dtype=torch.complex128, device="cuda")
    check(lib.aeolus_pe_derive(plan.handle, byref(m._params), K, p(x), p(f), B, st))
    g = synthesize(plan.id, f)
    npts = g.shape[-1]
    prod = torch.empty((B, 4 * K + 1, npts), dtype=torch.float64, device="cuda")
    fen = torch.empty((B * K, 2, npts), dtype=torch.float64, device="cuda")
    check(lib.aeolus_pe_columns(plan.handle, byref(m._params), K, sig, p(g), p(prod), p(fen), B, st))
    an = analyze(plan.id, prod)
    cd = vector_curl_div(m._ext_plan().id, m.R, fen[:, 0], fen[:, 1], False)
    cz, dz = cd[0].contiguous(), cd[1].contiguous()
    out = torch.empty_like(x)
    check(lib.aeolus_pe_spectral(m.l_max, byref(m._params), K, sig, p(x), p(an), p(cz), p(dz), p(m.phi_surface_lm),
                                 p(out), B, st))
    return out


def _state(L, K, B, seed, phis=False):
    rng = np.random.default_rng(seed)
    n, cut = L + 1, (2 * L) // 3
    x = torch.stack([isothermal_rest_state(L, K, temperature=260.0, surface_pressure=101325.0).coeffs for _ in range(B)])
    a = rng.standard_normal((B, 3 * K + 1, n, n)) + 1j * rng.standard_normal((B, 3 * K + 1, n, n))
    a[..., 0] = a[..., 0].real
    a = np.tril(a)
    a[..., cut + 1:, :] = 0
    a[:, :2 * K] *= 2e-6
    a[:, 2 * K:3 * K] *= 0.5
    a[:, 3 * K] *= 1e-3
    a[:, :2 * K, 0, 0] = 0
    return x + torch.as_tensor(a, device="cuda")


@pytest.mark.parametrize("grid,L,K,B", [((6, 10), 2, 1, 1), ((8, 14), 3, 2, 2), ((16, 32), 10, 7, 1), ((16, 33), 10, 8, 3),
                                        ((23, 46), 15, 9, 1), ((32, 64), 21, 17, 2), ((12, 24), 7, 64, 1),
                                        ((64, 128), 42, 5, 1), (2, 5, 4, 2), (3, 10, 9, 1)])
@pytest.mark.parametrize("split", [False, True])
def test_chain_equals_the_composed_calls(grid, L, K, B, split):
    if isinstance(grid, tuple):
        planet = ae.make_planet("latlon", nlat=grid[0], nlon=grid[1], l_max=L, product_quadrature="coarse")
    else:
        planet = ae.make_planet("geodesic", resolution=grid, l_max=L, product_quadrature="coarse")
    rng = np.random.default_rng(K)
    s = np.concatenate([[0.0], np.sort(rng.uniform(0.05, 0.95, K - 1)), [1.0]])
    n, cut = L + 1, (2 * L) // 3
    phis = np.zeros((n, n), complex)
    phis[1:cut + 1, 0] = rng.standard_normal(cut)
    m = PrimitiveEquationsModel(planet, SigmaGrid(tuple(s)), surface_geopotential_lm=phis)
    if split:
        m._plan.set_precision(_lib.PREC_SPLIT_BF16)
    x = _state(L, K, B, 10 * L + K)
    got, want = m.tendency(x), _composed(m, x)
    tol = 1e-10 if split else 1e-12
    for lo, hi in ((0, K), (K, 2 * K), (2 * K, 3 * K), (3 * K, 3 * K + 1)):
        a, b = got[:, lo:hi], want[:, lo:hi]
        assert float(torch.linalg.vector_norm(a - b)) <= tol * float(torch.linalg.vector_norm(b))
    # the fused steps are the generic engine's, bit for bit
    y = m.rk4(x, 30.0, 2)
    z = x
    for _ in range(2):
        z = rk4_step_device(m.tendency, z, 0.0, 30.0)
    assert torch.equal(y, z)
