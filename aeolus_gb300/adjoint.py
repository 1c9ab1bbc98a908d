"""Differentiation through the spectral models: hand-written adjoints behind
``torch.autograd.Function``.

The reference has no gradients; this module adds them on top of the GB300
kernels.  Every backward is a call into ``libaeolus_gb300.so``:

* ``synthesize`` / ``analyze`` (``aeolus_gb300.ops``) carry registered
  autograd formulas whose backward is the transposed transform
  (``aeolus_synthesize_adjoint`` = unit-weight analysis with the m > 0
  factor 2, ``aeolus_analyze_adjoint`` = weighted synthesis of the halved
  m > 0 slots).
* :func:`swe_rk4_checkpointed` / :func:`bve_rk4_checkpointed` advance
  ``nsteps`` RK4 steps and keep the step input every ``every`` steps; their
  backward re-runs each segment forward from its checkpoint (holding the
  ``every`` step inputs of one segment) and applies the per-step adjoint,
  which runs the four tendency VJPs on the device.  The shallow-water path
  keeps the stage inputs of a segment too, as long as they fit into the size
  of one step adjoint's workspace (``aeolus_swe_rk4_adjoint_stages``; beyond
  that the step adjoint recomputes them), and the last segment, with which the
  backward starts, from the forward pass until the backward has used it.
  ``keep_stages=False`` keeps neither, and neither is kept where the device's
  memory does not hold them; the gradient is the same bit for bit.

Peak device memory is therefore (checkpoints + one segment) states plus two
RK4-adjoint workspaces, of which the graph holds one segment and at most one
workspace until its backward, independent of ``nsteps``; without kept stages
(checkpoints + one segment) states plus one workspace, and the graph holds the
checkpoints alone.
"""
from __future__ import annotations

import torch

from . import _lib
from .ops import bve_rk4_adjoint, swe_rk4_adjoint, swe_rk4_adjoint_stages, swe_rk4_stages


def _swe_args(m):
    return m._plan.id, m.R, m.Omega, m.gravity, m.mean_depth, m.nu4


def _stage_steps(m, y, every):
    """Steps of a segment whose stage inputs (three states each) are kept: as
    many as fit into the size of one step adjoint's workspace."""
    L = m._plan.lmax
    members = y.numel() // (3 * (L + 1) * (L + 1))
    if members == 0:
        return 0
    return min(every, m._plan.workspace_bytes(_lib.OP_SWE_RK4_ADJOINT, members) // (3 * 16 * y.numel()))


def _keeps_stages(model):
    """Whether the model's steps are the library's: a model that steps by a
    method of its own keeps nothing, every step goes through that method."""
    from .shallow_water import ShallowWaterModel

    return getattr(type(model), "rk4", None) is ShallowWaterModel.rk4 and "rk4" not in vars(model)


def _swe_segment(m, y, dt, n, keep, last):
    """[(input, stage inputs or None)] of n steps from y, and with `last` the
    state after them."""
    steps = []
    for i in range(n):
        step = last or i < n - 1
        nxt, stages = None, None
        if i < keep:
            nxt, stages = swe_rk4_stages(*_swe_args(m), y, dt, m.forcing, step)
        elif step:
            nxt = m.rk4(y, dt, 1, check=False)
        steps.append((y, stages))
        y = nxt
    return steps, y


class _SweRk4Checkpointed(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y0, model, dt, nsteps, every, keep):
        every = max(1, int(every))
        nsteps = int(nsteps)
        ckpts = []
        y = y0.detach()
        # the backward starts with the last segment: its steps keep their
        # inputs from here on instead of being run again
        head = (nsteps - 1) // every * every if keep and nsteps > 0 else nsteps
        tail, keep = None, 0
        for i in range(nsteps):
            if i % every == 0:
                ckpts.append(y.clone())
            if i == head:
                keep = _stage_steps(model, y, every)
                try:
                    tail, out = _swe_segment(model, ckpts[-1], float(dt), nsteps - head, keep, True)
                    break
                except torch.cuda.OutOfMemoryError:
                    keep = 0
            y = out = model.rk4(y, dt, 1, check=False)
        ctx.model, ctx.dt, ctx.nsteps, ctx.every, ctx.ckpts = model, float(dt), nsteps, every, ckpts
        ctx.keep, ctx.tail = keep, tail
        return out if nsteps > 0 else y

    @staticmethod
    def backward(ctx, ybar):
        m = ctx.model
        yb = ybar.contiguous()
        for seg in range(len(ctx.ckpts) - 1, -1, -1):
            n = min(ctx.every, ctx.nsteps - seg * ctx.every)
            steps = None
            if seg == len(ctx.ckpts) - 1:  # kept once: a second backward runs the segment again
                steps, ctx.tail = ctx.tail, None
            if steps is None:
                steps = _rerun(ctx, seg, n)
            while steps:
                y, stages = steps.pop()
                if stages is not None:
                    try:
                        yb = swe_rk4_adjoint_stages(*_swe_args(m), y, stages, yb, ctx.dt, m.forcing)
                        continue
                    except torch.cuda.OutOfMemoryError:
                        ctx.keep, stages = 0, None
                    steps = [(x, None) for x, _ in steps]  # the adjoints do not fit beside the stages
                yb = swe_rk4_adjoint(*_swe_args(m), y, yb, ctx.dt, m.forcing)
        return yb, None, None, None, None, None


def _rerun(ctx, seg, n):
    """The steps of segment `seg` from its checkpoint."""
    try:
        return _swe_segment(ctx.model, ctx.ckpts[seg], ctx.dt, n, ctx.keep, False)[0]
    except torch.cuda.OutOfMemoryError:
        if ctx.keep == 0:
            raise
        ctx.keep = 0
    return _swe_segment(ctx.model, ctx.ckpts[seg], ctx.dt, n, 0, False)[0]


class _BveRk4Checkpointed(torch.autograd.Function):
    @staticmethod
    def forward(ctx, z0, model, dt, nsteps, every):
        every = max(1, int(every))
        ckpts = []
        z = z0.detach()
        for i in range(nsteps):
            if i % every == 0:
                ckpts.append(z.clone())
            z = model.rk4(z, dt, 1)
        ctx.model, ctx.dt, ctx.nsteps, ctx.every, ctx.ckpts = model, float(dt), int(nsteps), every, ckpts
        return z

    @staticmethod
    def backward(ctx, zbar):
        m = ctx.model
        zb = zbar.contiguous()
        for seg in range(len(ctx.ckpts) - 1, -1, -1):
            start = seg * ctx.every
            n = min(ctx.every, ctx.nsteps - start)
            states = [ctx.ckpts[seg]]
            for _ in range(n - 1):
                states.append(m.rk4(states[-1], ctx.dt, 1))
            for i in range(n - 1, -1, -1):
                zb = bve_rk4_adjoint(m._plan.id, m.R, m.Omega, m.nu, states[i], zb, ctx.dt)
        return zb, None, None, None, None


def swe_rk4_checkpointed(model, y0: torch.Tensor, dt: float, nsteps: int, every: int = 8, *,
                         keep_stages: bool = True) -> torch.Tensor:
    """``nsteps`` SWE RK4 steps of ``[..., 3, L+1, L+1]`` states, differentiable
    in ``y0`` through the hand-written adjoint with checkpoints every
    ``every`` steps (run/engine.py:406-431 differentiated).  ``keep_stages``
    trades memory for time (module docstring); without a gradient to come
    nothing is kept."""
    keep = bool(keep_stages) and torch.is_grad_enabled() and y0.requires_grad and _keeps_stages(model)
    return _SweRk4Checkpointed.apply(y0, model, float(dt), int(nsteps), int(every), keep)


def bve_rk4_checkpointed(model, z0: torch.Tensor, dt: float, nsteps: int, every: int = 8) -> torch.Tensor:
    """``nsteps`` BVE RK4 steps, differentiable in ``z0`` (run/bve/runner.py:211-216)."""
    return _BveRk4Checkpointed.apply(z0, model, float(dt), int(nsteps), int(every))


def weighted_phi_misfit(model, y: torch.Tensor, target_grid: torch.Tensor) -> torch.Tensor:
    """Area-weighted squared error of the final geopotential on the state
    grid: sum_points w (phi(y) - target)^2 per member (w = the quadrature
    weights, summing to 4 pi).  Differentiable through ``synthesize``."""
    from .ops import synthesize
    plan = model._state_plan
    g = synthesize(plan.id, y[..., 2, :, :])
    w = model.sh.weights.reshape(-1).to(g)
    return ((g - target_grid) ** 2 * w).sum(dim=-1)
