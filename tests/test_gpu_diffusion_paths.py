"""The two forms of the energy diffusion, bit for bit against the oracle, where their shapes can
go wrong.  Many short columns run warp by warp through the scratch (tiles of 8 rows, chunks of
4): lengths around both sizes, a last warp that is not full.  Few columns run in shared
memory: several columns per block, a last block that is not full, more than one warp of rows.
"""
import pytest

import oracle as O
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

from helpers import assert_identical

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _device_semantics():
    O.set_device_semantics(True)
    yield
    O.set_device_semantics(False)


def _check(g, solver, **kw):
    st = S.init_state(g, perturb=0.2, **kw)
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    cfg = F.FluidCfg(st.Teinf, solver)
    dt, _ = O.dt_calc(g, st, 0.5)
    O.energy_diffusion(g, st, 5 * dt, solver)
    F.energy_diffusion(cfg, ds, 5 * dt)
    assert_identical(ds.to_host(st), st, "energy_diffusion")
    dt, _ = O.dt_calc(g, st, 0.5)
    O.fluid_adv(g, st, dt, solver)
    F.fluid_adv(cfg, ds, dt)
    assert_identical(ds.to_host(st), st, "step")


@pytest.mark.parametrize("solver", [2, 1])
@pytest.mark.parametrize("lx1", [4, 5, 6, 8, 9, 16, 17, 23])
def test_many_short_columns(lx1, solver):
    if lx1 < 16:
        _check(G.cartesian_grid(lx1, 61, 37, inverted=lx1 % 2 == 1), solver, seed=lx1, J1_amp=1e-5)
    else:
        _check(G.dipole_grid(lx1, 61, 37, q_extent=0.5 if lx1 == 17 else None), solver, seed=lx1)


@pytest.mark.parametrize("solver", [2, 1])
@pytest.mark.parametrize("lx", [(64, 25, 19), (33, 13, 41), (200, 21, 9)])
def test_few_columns(lx, solver):
    _check(G.dipole_grid(*lx, q_extent=0.5 if lx[0] == 64 else None), solver, seed=lx[0], J1_amp=1e-5)
