"""The fused advection bit for bit against the oracle where its paths can go wrong: lines cut
into parts (whole and ragged parts, periodic wraps, null cells, the step with compression),
lines in place on grids that fill the device, and values whose quotients leave the shared
range test (zero velocities, very small and very large densities and spacings).
"""
import numpy as np
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


def _steps(g, st, n=2):
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    cfg, ref = F.FluidCfg(st.Teinf), st.copy()
    for _ in range(n):
        dt = F.dt_calc(ds, 0.5)
        F.fluid_adv(cfg, ds, dt)
        want, _ = O.dt_calc(g, ref, 0.5)
        assert float(dt.item()) == want
        O.fluid_adv(g, ref, want)
    return ds.to_host(st), ref


CUT = [
    ("periodic_8", lambda: G.cartesian_grid(20, 5, 8, flagper=1)),
    ("periodic_ragged", lambda: G.cartesian_grid(33, 9, 13, flagper=1)),
    ("periodic_long", lambda: G.cartesian_grid(40, 6, 50, flagper=1)),
    ("dipole_ragged", lambda: G.dipole_grid(35, 17, 23)),
    ("dipole_nulls", lambda: G.dipole_grid(70, 31, 9, q_extent=0.5)),
    ("plane", lambda: G.cartesian_grid(65, 97, 1, inverted=True)),
    ("in_place", lambda: G.cartesian_grid(34, 76, 75)),
    ("in_place_periodic", lambda: G.cartesian_grid(34, 75, 77, flagper=1)),
]


@pytest.mark.parametrize("name,mk", CUT, ids=[c[0] for c in CUT])
def test_line_parts(name, mk):
    g = mk()
    got, ref = _steps(g, S.init_state(g, seed=len(name), perturb=0.2))
    assert_identical(got, ref, name)


@pytest.mark.parametrize("name,mk", CUT[:5], ids=[c[0] for c in CUT[:5]])
def test_line_parts_with_compression(name, mk):
    g = mk()
    st = S.init_state(g, seed=3, perturb=0.2)
    a = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    b = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    cfg = F.FluidCfg(st.Teinf)
    for _ in range(2):
        dt = F.dt_calc(a, 0.5)
        Qa = F.fluid_adv_compression(cfg, a, dt)
        Qb = F.fluid_adv_compression_reference_order(cfg, b, dt)
        assert bool((Qa == Qb).all())
    assert_identical(a.to_host(st), b.to_host(st), name)


@pytest.mark.parametrize("what", ["still", "tiny", "huge", "wide"])
@pytest.mark.parametrize("kind", ["cartesian", "dipole"])
def test_values_outside_the_shared_range(what, kind):
    g = G.cartesian_grid(37, 11, 9, x3span=1e70 if what == "wide" else 600e3) if kind == "cartesian" else G.dipole_grid(37, 11, 9)
    st = S.init_state(g, seed=5, perturb=0.2, vscale=0.0 if what == "still" else 1.0)
    rng = np.random.default_rng(1)
    if what in ("tiny", "huge"):  # one cell in twenty
        hit = rng.uniform(size=st.ns.shape) < 0.05
        st.ns[hit] = 1e-170 if what == "tiny" else 1e165
        st.vs1[rng.uniform(size=st.vs1.shape) < 0.05] = 1e-180
    with np.errstate(all="ignore"):
        got, ref = _steps(g, st, 1)
    for name in ("fluidvars", "fluidauxvars"):
        assert np.array_equal(getattr(got, name), getattr(ref, name), equal_nan=True), name
