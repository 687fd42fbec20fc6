"""Grids one cell wide along x2: advec1D_MC_curv passes a single-cell line through
(advec.f90:384-435), and the step still ends with rhov12v1, clean_param and rhoe2T.  The step
bit for bit against the oracle, the step with compression and the batched step against their
plain forms, x3 lines whole and in parts (lx3 >= 8 on these grids).
"""
import pytest
import torch

import oracle as O
from gemini_b200 import batch as BT
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

from helpers import assert_identical

pytestmark = pytest.mark.gpu

GRIDS = {
    "parts": lambda: G.cartesian_grid(24, 1, 9),
    "whole": lambda: G.cartesian_grid(24, 1, 5, inverted=True),
    "column": lambda: G.cartesian_grid(40, 1, 1),
    "periodic": lambda: G.cartesian_grid(33, 1, 13, flagper=1),
    "dipole": lambda: G.dipole_grid(35, 1, 17),
    "dipole_nulls": lambda: G.dipole_grid(40, 1, 9, q_extent=0.5),
}


@pytest.fixture(scope="module", autouse=True)
def _device_semantics():
    O.set_device_semantics(True)
    yield
    O.set_device_semantics(False)


def _device(g, st):
    return F.DeviceState.from_host(F.DeviceGrid(g), st.copy())


@pytest.mark.parametrize("name", GRIDS)
def test_step(name):
    g = GRIDS[name]()
    st = S.init_state(g, seed=3, perturb=0.2)
    ds, cfg, ref = _device(g, st), F.FluidCfg(st.Teinf), st.copy()
    for _ in range(2):
        dt = F.dt_calc(ds, 0.5)
        F.fluid_adv(cfg, ds, dt)
        want, _ = O.dt_calc(g, ref, 0.5)
        assert float(dt.item()) == want
        O.fluid_adv(g, ref, want)
    assert_identical(ds.to_host(st), ref, name)


@pytest.mark.parametrize("name", GRIDS)
def test_step_with_compression(name):
    g = GRIDS[name]()
    st = S.init_state(g, seed=3, perturb=0.2)
    a, b = _device(g, st), _device(g, st)
    cfg = F.FluidCfg(st.Teinf)
    for _ in range(2):
        dt = F.dt_calc(a, 0.5)
        Qa = F.fluid_adv_compression(cfg, a, dt)
        Qb = F.fluid_adv_compression_reference_order(cfg, b, dt)
        assert bool((Qa == Qb).all())
    assert_identical(a.to_host(st), b.to_host(st), name)


def test_batch():
    insts = []
    for k, mk in enumerate(GRIDS.values()):
        g = mk()
        st = S.init_state(g, seed=k, perturb=0.2)
        dg = F.DeviceGrid(g)
        insts.append((st, [(dg, F.DeviceState.from_host(dg, st.copy()), F.FluidCfg(st.Teinf)) for _ in range(2)]))
    b = BT.Batch([i[0] for _, i in insts])
    for _ in range(2):
        b.step()
        for _, i in insts:
            BT.plain_step(*i[1])
    torch.cuda.synchronize()
    for (st, i), name in zip(insts, GRIDS):
        assert_identical(i[0][1].to_host(st), i[1][1].to_host(st), name)
