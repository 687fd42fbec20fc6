"""The step VJP on grids one cell wide along x2, x3 or both: a single-cell line passes through the
sweeps (advec.f90:384-435), so its cotangent passes through too.  Against autograd of the
pure-tensor transcription, on random cotangents, with the tolerance of
test_gpu_adjoint.py::test_cuda_step_vjp_matches_autograd; the replay gives the forward step's bits."""
import numpy as np
import pytest
import torch

from gemini_b200 import adjoint as AD
from gemini_b200 import grid as G
from gemini_b200 import state as S

pytestmark = pytest.mark.gpu

GRIDS = {
    "x3": lambda: G.cartesian_grid(24, 6, 1),
    "x2": lambda: G.cartesian_grid(24, 1, 9),
    "x2_periodic": lambda: G.cartesian_grid(20, 1, 6, flagper=1),
    "both": lambda: G.cartesian_grid(22, 1, 1, inverted=True),
}


@pytest.mark.parametrize("name", GRIDS)
def test_step_vjp(name):
    g = GRIDS[name]()
    st = S.init_state(g, seed=2, perturb=0.1)
    P = AD.DiffProblem(g, st, 2, checkpoint_every=1)
    rng = np.random.default_rng(7)
    I = (slice(None), slice(2, g.lx3 + 2), slice(2, g.lx2 + 2), slice(2, g.lx1 + 2))
    Ttop = torch.from_numpy(st.Teinf * (1 + 0.05 * rng.uniform(-1, 1, (g.lx3, g.lx2)))).cuda()
    fin, ck = P.run(P.base[0:6][I].clone(), Ttop, keep=True)
    cot = []
    for t in ck[1][:3]:
        c = torch.zeros_like(t)
        c[I] = torch.from_numpy(rng.standard_normal(c[I].shape)).cuda()
        cot.append(c)
    cot += [torch.from_numpy(rng.standard_normal(t.shape)).cuda() for t in ck[1][3:]]
    got, gtop = P.step_vjp_cuda(ck[1], Ttop, 1, cot)
    P.cuda_sweep_adjoint = False
    inp = [t.detach().clone().requires_grad_(True) for t in ck[1]]
    tt = Ttop.clone().requires_grad_(True)
    exp, etop = P._vjp_body(inp, tt, P.dt_tensor(1), cot, use_cuda_diffusion_adjoint=False)
    for nm, x, y in zip(("ns", "vs1", "Ts", "lo", "hi", "Ttop"), list(got) + [gtop], list(exp) + [etop]):
        assert float((x - y).abs().max()) <= 1e-9 * float(y.abs().max()), (name, nm)  # both zero: equal
    P._set_top(Ttop)
    P._replay(0, ck[1], 1)
    for x, y in zip(P._finish(0, 1), fin):
        assert torch.equal(x, y)
    P.close()
