"""A differentiable problem's step captured into a CUDA graph by its caller: accepted before any
other call on the problem, and the graph keeps the step it was captured with when the schedule
changes and other steps run."""
import pytest
import torch

from gemini_b200 import adjoint as AD
from gemini_b200 import grid as G
from gemini_b200 import state as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("used", [False, True])
def test_captured_step(used):
    g = G.cartesian_grid(24, 8, 6)
    P = AD.DiffProblem(g, S.init_state(g, seed=2, perturb=0.1), 2, checkpoint_every=1)
    start = P.ds.fluidvars.clone()
    faces = P.v1i.clone()
    if used:
        P.dt_tensor(0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        P.cuda_step(0)

    def run(f):
        P.ds.fluidvars.copy_(start)
        P.v1i.copy_(faces)
        f()
        return P.ds.fluidvars.clone()

    want = run(lambda: P.cuda_step(0))
    assert torch.equal(run(graph.replay), want)
    P.dts = [0.5 * x for x in P.dts]
    other = run(lambda: P.cuda_step(0))
    assert not torch.equal(other, want)
    hold = [torch.full((2,), 1e3, dtype=torch.float64, device="cuda") for _ in range(64)]  # reuse of freed blocks
    assert torch.equal(run(graph.replay), want)
    assert torch.equal(run(lambda: P.cuda_step(0)), other)
    del hold


@pytest.mark.parametrize("k", [1, 2])
def test_captured_gradient(k):
    """Forward and backward in one captured graph, replayed after the schedule has changed."""
    g = G.cartesian_grid(24, 8, 6)
    P = AD.DiffProblem(g, S.init_state(g, seed=2, perturb=0.1), 4, checkpoint_every=k)
    x = P.base[(slice(0, 6), slice(2, -2), slice(2, -2), slice(2, -2))].clone().requires_grad_(True)

    def grad():
        ns, Ts = AD.FluidAdvance.apply(x, None, P)
        return torch.autograd.grad(ns.sum() * 1e-11 + (Ts * Ts).sum() * 1e-6, [x])[0]

    want = grad().clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        grad()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = grad()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    P.dts = [0.5 * d for d in P.dts]
    assert not torch.equal(grad(), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
