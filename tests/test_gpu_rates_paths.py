"""The exchange rates where a block of 32 cells leaves the untested quotients: cells of very low
density, drifts far above the thermal speed (Psi underflows to zero), a vanishing neutral, and
the same with neighbours inside the range.  Tolerance as in test_gpu_rates.py, whose derivation
(the device's math functions, two ulp each, through sums of like and unlike signs) does not
depend on the inputs' range.
"""
import numpy as np
import pytest

import oracle as O
from gemini_b200 import fluid as F
from gemini_b200 import grid as G

from helpers import rate_inputs
from test_gpu_rates import _cmp, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["density", "drift", "neutral", "all_cells"])
@pytest.mark.parametrize("mk", [lambda: G.cartesian_grid(37, 5, 3), lambda: G.dipole_grid(40, 6, 5)], ids=["cart", "dipole"])
def test_outside_the_fast_range(mk, what):
    g = mk()
    st, nn, vn, Tn, E1, Q, g1, alt = rate_inputs(g, 7)
    st.electrovars[..., 0] = E1
    rng = np.random.default_rng(2)
    cells = np.ones(st.ns.shape[:3], bool) if what == "all_cells" else rng.uniform(size=st.ns.shape[:3]) < 0.03
    if what in ("density", "all_cells"):
        st.ns[cells, 1] = 1e-120
    if what == "drift":
        st.vs1[cells, 2] = 4e5
    if what == "neutral":
        nn[cells[2:-2, 2:-2, 2:-2], 1] = 0.0
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    d = [_dev(a) for a in (nn, vn[0], vn[1], vn[2], Tn)]
    _cmp("energy", F.srcs_energy(ds, *d), O.srcs_energy(g, st, nn, *vn, Tn))
    _cmp("momentum", F.srcs_momentum(ds, d[0], d[1], d[4], _dev(Q), _dev(alt), _dev(g1)),
         O.srcs_momentum(g, st, nn, vn[0], Tn, E1, Q, g1))
