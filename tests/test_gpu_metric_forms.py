"""Tabulated metrics that vary along x3, and periodic grids with tabulated metrics: a dipole whose
metric factors are scaled by smooth functions of x3, open and periodic, and the plain dipole
periodic.  The x3 sweep reads a line's metrics at every cell there, the diffusion takes its
columns x2 fastest, the ghost passes wrap.  Lines cut into parts and lines in place; step and
time step bit for bit against the oracle, the step with compression against the routines in the
reference's order bit for bit and the oracle to 1e-12, the batch against plain steps, the replay
of a step against the step."""
import dataclasses

import numpy as np
import pytest
import torch

import oracle as O
from gemini_b200 import adjoint as AD
from gemini_b200 import batch as BT
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

from helpers import assert_identical, state_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _device_semantics():
    O.set_device_semantics(True)
    yield
    O.set_device_semantics(False)


def _grid(lx, vary, flagper, **kw):
    g = G.dipole_grid(*lx, **kw)
    g.flagper = flagper
    if not vary:
        return g
    new = {}
    for n in ("1", "2", "3"):
        # cells -1 .. lx3+2, and the x3 faces 1 .. lx3+1 half a cell below
        def f(pos, a=0.02 + 0.01 * int(n), w=0.9 + 0.2 * int(n)):
            return 1.0 + a * np.sin(w * pos + int(n))
        new["h" + n] = getattr(g, "h" + n) * f(np.arange(-1, lx[2] + 3))
        new[f"h{n}x1i"] = getattr(g, f"h{n}x1i") * f(np.arange(1, lx[2] + 1))
        new[f"h{n}x2i"] = getattr(g, f"h{n}x2i") * f(np.arange(1, lx[2] + 1))
        new[f"h{n}x3i"] = getattr(g, f"h{n}x3i") * f(np.arange(1, lx[2] + 2) - 0.5)
    return dataclasses.replace(g, **{k: np.asfortranarray(v) for k, v in new.items()})


FORMS = {"vary": (True, 0), "vary_periodic": (True, 1), "periodic": (False, 1)}
SIZES = [(35, 17, 23), (40, 9, 6), (34, 75, 77)]  # lines in parts; few cells; lines in place


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("lx", SIZES, ids=str)
def test_step(form, lx):
    g = _grid(lx, *FORMS[form], q_extent=0.5 if lx[0] == 40 else None)
    st = S.init_state(g, seed=lx[1], perturb=0.2)
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    cfg, ref = F.FluidCfg(st.Teinf), st.copy()
    for _ in range(2):
        dt = F.dt_calc(ds, 0.5)
        F.fluid_adv(cfg, ds, dt)
        want, _ = O.dt_calc(g, ref, 0.5)
        assert float(dt.item()) == want
        O.fluid_adv(g, ref, want)
    assert_identical(ds.to_host(st), ref, form)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("lx", SIZES, ids=str)
def test_step_with_compression(form, lx):
    g = _grid(lx, *FORMS[form])
    st = S.init_state(g, seed=3, perturb=0.2)
    dg = F.DeviceGrid(g)
    a, b = (F.DeviceState.from_host(dg, st.copy()) for _ in range(2))
    cfg, ref = F.FluidCfg(st.Teinf), st.copy()
    dt = F.dt_calc(a, 0.5)
    Qa = F.fluid_adv_compression(cfg, a, dt)
    Qb = F.fluid_adv_compression_reference_order(cfg, b, dt)
    assert torch.equal(Qa, Qb)
    assert_identical(a.to_host(st), b.to_host(st), form)
    O.fluid_adv_compression(g, ref, float(dt.item()))
    err = state_err(a.to_host(st), ref)
    assert max(err.values()) <= 1e-12, err


def test_batch():
    """Every form with an invariant open dipole beside it, so that both x3 sweeps run."""
    both = []
    for k, (vary, per) in enumerate(list(FORMS.values()) + [(False, 0)]):
        g = _grid((33, 11 + k, 9), vary, per)
        st = S.init_state(g, seed=k, perturb=0.2)
        dg = F.DeviceGrid(g)
        both.append((st, [(dg, F.DeviceState.from_host(dg, st.copy()), F.FluidCfg(st.Teinf)) for _ in range(2)]))
    for sel in ([0], [1], [2], [0, 3], [0, 1, 2, 3]):
        b = BT.Batch([both[k][1][0] for k in sel])
        b.step()
        for k in sel:
            BT.plain_step(*both[k][1][1])
        torch.cuda.synchronize()
        for k in sel:
            st, (p, q) = both[k]
            assert_identical(p[1].to_host(st), q[1].to_host(st), f"{sel} {k}")
        b.close()


@pytest.mark.parametrize("form", FORMS)
def test_replay(form):
    g = _grid((28, 9, 10), *FORMS[form])
    P = AD.DiffProblem(g, S.init_state(g, seed=5, perturb=0.2), 2, checkpoint_every=1)
    I = (slice(0, 6), slice(2, g.lx3 + 2), slice(2, g.lx2 + 2), slice(2, g.lx1 + 2))
    fin, ck = P.run(P.base[I].clone(), None, keep=True)
    P._set_top(None)
    P._replay(0, ck[1], 1)
    for x, y in zip(P._finish(0, 1), fin):
        assert torch.equal(x, y), form
    P.close()
