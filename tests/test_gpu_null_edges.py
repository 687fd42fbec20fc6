"""clean_param(2)'s border fix at null points (a warp per column scans 32 cells at a time): null
runs that begin, end and cross at the scan's boundaries, against the oracle bit for bit."""
import numpy as np
import pytest

import oracle as O
from gemini_b200 import batch as BT
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

from helpers import assert_identical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gridflag", [0, 1])
@pytest.mark.parametrize("lx1", [5, 32, 33, 34, 65, 97])
def test_null_edges(lx1, gridflag):
    g = G.dipole_grid(lx1, 9, 7, q_extent=0.5)
    g.gridflag = gridflag
    rng = np.random.default_rng(lx1)
    edges = [e for e in (0, 1, 30, 31, 32, 33, 63, 64, lx1 - 2, lx1 - 1, lx1) if 0 <= e <= lx1]
    g.nullpts[...] = False
    for j in range(9):
        for k in range(7):  # some runs are empty, some a whole column
            a, b = sorted(rng.choice(edges, 2))
            g.nullpts[a:b, j, k] = True
    g.nullpts[:, 0, 0] = True
    g.nullpts[:, 1, 0] = False
    st = S.init_state(g, seed=lx1, perturb=0.2)
    ds = F.DeviceState.from_host(F.DeviceGrid(g), st.copy())
    O.clean_param(g, st, 2)
    F.clean_param(ds, 2)
    assert_identical(ds.to_host(st), st, "clean_param(2)")


def test_batched_work_items():
    """The batched fix gets a warp per column too: four columns per work item of 128 threads."""
    g = G.dipole_grid(40, 9, 7, q_extent=0.5)
    assert g.nullpts.any()
    items = []
    for nulls in (True, False):
        g.nullpts = g.nullpts & nulls
        st = S.init_state(g, seed=1)
        dg = F.DeviceGrid(g)
        b = BT.Batch([(dg, F.DeviceState.from_host(dg, st), F.FluidCfg(st.Teinf))])
        items.append(b.info()[1])
        b.close()
    assert items[0] - items[1] == (9 * 7 + 3) // 4
