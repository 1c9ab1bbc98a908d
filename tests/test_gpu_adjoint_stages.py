"""Gradients through RK4 steps whose stage inputs are kept: the kept step is
the step, its adjoint with kept stages is the adjoint that recomputes them, and
the checkpointed gradient does not depend on how many steps keep them (bit for
bit: the same kernels run on the same numbers).  Single steps, a short last
segment, one segment longer than the run, several and no lead dimensions,
topography, a second backward through a retained graph, scratch limits."""
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import _lib, adjoint, workloads as W
from aeolus_gb300.adjoint import swe_rk4_checkpointed
from aeolus_gb300.ops import _swe_params, swe_rk4, swe_rk4_adjoint, swe_rk4_adjoint_stages, swe_rk4_stages
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu


def _model(L, split, nlat=32, nlon=64, members=3):
    planet = ae.make_planet("latlon", nlat=nlat, nlon=nlon, l_max=L, product_quadrature="coarse")
    if split:
        planet.sh.plan.set_precision(_lib.PREC_SPLIT_BF16)
    s0, depth = W.member_states(L, members, seed=5)
    return ShallowWaterModel(planet, gravity=W.GRAVITY, mean_depth=depth), torch.as_tensor(s0, device="cuda")


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("lead", [(), (3,), (1, 3)])
def test_step_and_adjoint(split, lead):
    m, s0 = _model(21, split)
    y = s0[0] if lead == () else s0.reshape(lead + s0.shape[1:])
    args = adjoint._swe_args(m)
    nxt, stages = swe_rk4_stages(*args, y, 120.0, m.forcing)
    none, again = swe_rk4_stages(*args, y, 120.0, m.forcing, False)
    assert none is None and torch.equal(stages, again)
    assert torch.equal(nxt, m.rk4(y, 120.0, 1))
    yb = torch.flip(y, dims=(-3,)).contiguous()
    want = swe_rk4_adjoint(*args, y, yb, 120.0, m.forcing)
    assert torch.equal(swe_rk4_adjoint_stages(*args, y, stages, yb, 120.0, m.forcing), want)
    with pytest.raises(ValueError):
        swe_rk4_adjoint_stages(*args, y, stages[:2], yb, 120.0, m.forcing)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nsteps,every", [(1, 1), (4, 1), (7, 3), (6, 3), (5, 9), (0, 2)])
def test_gradient_does_not_depend_on_kept_steps(split, nsteps, every, monkeypatch):
    m, s0 = _model(21, split)
    grads = []
    for keep in (None, 0, 1):
        if keep is not None:
            monkeypatch.setattr(adjoint, "_stage_steps", lambda *_: keep)
        y = s0.clone().requires_grad_(True)
        out = swe_rk4_checkpointed(m, y, 120.0, nsteps, every=every)
        assert torch.equal(out.detach(), m.rk4(s0, 120.0, nsteps) if nsteps else s0)
        J = (torch.view_as_real(out) ** 2).sum()
        (a,) = torch.autograd.grad(J, y, retain_graph=True)
        (b,) = torch.autograd.grad(J, y)
        assert torch.equal(a, b)
        grads.append(a)
    assert all(torch.equal(g, grads[0]) for g in grads)


def test_argument_errors():
    m, s0 = _model(21, True)
    p, lib = m._plan, _lib.load()
    prm = _swe_params(m.R, m.Omega, m.gravity, m.mean_depth, m.nu4)
    stages, nxt = torch.empty((3,) + tuple(s0.shape), dtype=s0.dtype, device="cuda"), torch.empty_like(s0)
    w = p.workspace(_lib.OP_SWE_RK4, 3)
    call = lambda s, n, g, size, dt=1.0: lib.aeolus_swe_rk4_stages(p.handle, prm, s, n, g, 3, dt, w.data_ptr(), size, None)
    ok = (s0.data_ptr(), nxt.data_ptr(), stages.data_ptr())
    assert call(*ok, w.numel()) == _lib.OK
    assert call(*ok, 1024) not in (_lib.OK, _lib.ERR_ARG)
    assert call(*ok, w.numel(), float("nan")) == _lib.ERR_ARG
    assert call(ok[0], ok[0], ok[2], w.numel()) == _lib.ERR_ARG
    assert call(ok[0], ok[1], None, w.numel()) == _lib.ERR_ARG
    torch.cuda.synchronize()


def test_split_point_sets():
    """The step refuses a split point-set plan and so do kept stages; the step
    adjoint takes one."""
    from test_gpu_adjoint import points_plan

    p = points_plan(8)
    p.set_precision(_lib.PREC_SPLIT_BF16)
    s0, depth = W.member_states(8, 2, seed=9)
    y = torch.as_tensor(s0, device="cuda")
    args = (p.id, W.EARTH_RADIUS, W.EARTH_OMEGA, W.GRAVITY, depth, 0.0)
    with pytest.raises(ValueError):
        swe_rk4(*args, y, 60.0, 1)
    with pytest.raises(ValueError):
        swe_rk4_stages(*args, y, 60.0)
    g = swe_rk4_adjoint(*args, y, torch.ones_like(y).tril(), 60.0)
    assert torch.isfinite(torch.view_as_real(g)).all() and g.abs().max() > 0
    p.close()
