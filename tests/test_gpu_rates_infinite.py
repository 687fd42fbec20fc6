"""Infinite neutral temperatures in some cells: the exchange rates are infinite or NaN exactly where
the oracle's are, and the other cells of the same blocks agree with it to the tolerance of
test_gpu_rates.py.  (An infinite collision frequency divided through the untested quotients would
turn into NaN, so its block has to take the tested ones.)"""
import numpy as np
import pytest

import oracle as O
from gemini_b200 import fluid as F
from gemini_b200 import grid as G

from helpers import rate_inputs
from test_gpu_rates import RTOL, LSP, _dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mk", [lambda: G.cartesian_grid(37, 5, 3), lambda: G.dipole_grid(40, 6, 5)], ids=["cart", "dipole"])
def test_infinite_neutral_temperature(mk):
    g = mk()
    st, nn, vn, Tn, E1, Q, g1, alt = rate_inputs(g, 11)
    st.electrovars[..., 0] = E1
    Tn[np.random.default_rng(4).uniform(size=Tn.shape) < 0.03] = np.inf
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    d = [_dev(a) for a in (nn, vn[0], vn[1], vn[2], Tn)]
    with np.errstate(all="ignore"):
        pairs = {"energy": (F.srcs_energy(ds, *d), O.srcs_energy(g, st, nn, *vn, Tn)),
                 "momentum": (F.srcs_momentum(ds, d[0], d[1], d[4], _dev(Q), _dev(alt), _dev(g1)),
                              O.srcs_momentum(g, st, nn, vn[0], Tn, E1, Q, g1))}
    for what, (got, want) in pairs.items():
        for nm, a, b in zip(("Pr", "Lo"), got, want):
            a = a.cpu().numpy().reshape(b.shape, order="F")
            fin = np.isfinite(b)
            assert not fin.all(), (what, nm)
            assert np.array_equal(a[~fin], b[~fin], equal_nan=True), (what, nm)
            scale = np.where(fin, np.abs(b), 0.0).reshape(-1, LSP, order="F").max(axis=0)
            err = np.abs(np.where(fin, a, 0.0) - np.where(fin, b, 0.0))
            assert (err <= RTOL * (np.where(fin, np.abs(b), 0.0) + scale)).all(), (what, nm)
