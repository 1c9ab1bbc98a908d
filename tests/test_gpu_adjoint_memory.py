"""What a checkpointed shallow-water gradient keeps: nothing but checkpoints when no
gradient is to come or the caller asks for it, the last segment until a backward has
used it, and nothing where the memory does not hold it; the gradient stays the same
bit for bit."""
import pytest
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import adjoint, workloads as W
from aeolus_gb300.adjoint import swe_rk4_checkpointed
from aeolus_gb300.shallow_water import ShallowWaterModel

pytestmark = pytest.mark.gpu
NSTEPS, EVERY = 7, 4


@pytest.fixture(scope="module")
def problem():
    s0, depth = W.member_states(21, 4, seed=1)
    m = ShallowWaterModel(ae.make_planet("latlon", nlat=32, nlon=64, l_max=21), gravity=W.GRAVITY, mean_depth=depth)
    y = torch.as_tensor(s0, device="cuda")
    return m, y, _gradient(m, y, keep_stages=False)


def _gradient(m, y0, **kw):
    y = y0.clone().requires_grad_(True)
    out = swe_rk4_checkpointed(m, y, 120.0, NSTEPS, every=EVERY, **kw)
    return torch.autograd.grad((torch.view_as_real(out) ** 2).sum(), y)[0]


def _never(*_):
    raise AssertionError("stage inputs kept")


def test_nothing_kept_without_a_gradient(problem, monkeypatch):
    m, y0, want = problem
    monkeypatch.setattr(adjoint, "swe_rk4_stages", _never)
    y = y0.clone().requires_grad_(True)
    with torch.no_grad():
        swe_rk4_checkpointed(m, y, 120.0, NSTEPS, every=EVERY)
    swe_rk4_checkpointed(m, y0, 120.0, NSTEPS, every=EVERY)
    assert torch.equal(_gradient(m, y0, keep_stages=False), want)


@pytest.mark.parametrize("keep", [False, True])
def test_memory_of_the_graph(problem, keep):
    m, y0, want = problem
    size = 512 * -(-y0.numel() * 16 // 512)  # the allocator's blocks
    y = y0.clone().requires_grad_(True)
    held = torch.cuda.memory_allocated()
    out = swe_rk4_checkpointed(m, y, 120.0, NSTEPS, every=EVERY, keep_stages=keep)
    lasting = 2 * size + size  # two checkpoints and the output
    tail = (NSTEPS - EVERY) * (size + 512 * -(-3 * y0.numel() * 16 // 512)) - size  # less its first input, a checkpoint
    assert torch.cuda.memory_allocated() - held <= lasting + (tail if keep else 0)
    (g,) = torch.autograd.grad(out, y, 2.0 * out.detach(), retain_graph=True)
    assert torch.equal(g, want)
    del g
    assert torch.cuda.memory_allocated() - held <= lasting
    assert torch.equal(torch.autograd.grad(out, y, 2.0 * out.detach())[0], want)


@pytest.mark.parametrize("name", ["swe_rk4_stages", "swe_rk4_adjoint_stages"])
@pytest.mark.parametrize("call", [0, 1, 2, 3, 5])
def test_out_of_memory(problem, monkeypatch, name, call):
    m, y0, want = problem
    inner, calls = getattr(adjoint, name), []

    def fails(*args):
        calls.append(1)
        if len(calls) == call + 1:
            raise torch.cuda.OutOfMemoryError("no room for the stage inputs")
        return inner(*args)

    monkeypatch.setattr(adjoint, name, fails)
    assert torch.equal(_gradient(m, y0), want)
