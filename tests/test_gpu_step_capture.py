"""The step captured into a CUDA graph (its kernels are launched with programmatic stream
serialization, which the capture turns into graph edges): replays equal plain calls bit for bit.
"""
import pytest
import torch

from gemini_b200 import _lib
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

from helpers import assert_identical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mk", [lambda: G.cartesian_grid(40, 16, 9, flagper=1), lambda: G.dipole_grid(48, 33, 40, q_extent=0.5)],
                         ids=["cart", "dipole"])
def test_captured_step(mk):
    g = mk()
    st = S.init_state(g, seed=3, perturb=0.2)
    dg = F.DeviceGrid(g)
    a, b = (F.DeviceState.from_host(dg, st.copy()) for _ in range(2))
    cfg = F.FluidCfg(st.Teinf)
    out = torch.empty(1, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().gem_work_prepare(b.work, dg.handle))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        F.fluid_adv(cfg, b, F.dt_calc(b, 0.5, out=out))
    for _ in range(3):
        F.fluid_adv(cfg, a, F.dt_calc(a, 0.5))
        graph.replay()
    assert_identical(b.to_host(st), a.to_host(st), "captured step")
