"""The energy diffusion by warps of 32 columns (grids with too many columns for the shared-memory
form), bit for bit against the oracle on tabulated metrics: columns x3 fastest and x2 fastest,
null cells, both solvers, three and more tiles of 8 rows, a last warp that is not full, and the
instances for few blocks (at most three per SM) and for many.  The sizes keep clear of the line
between the two forms, and the form taken is asserted."""
import pytest

from gemini_b200 import _lib
from gemini_b200 import fluid as F
from gemini_b200 import grid as G

from test_gpu_diffusion_paths import _check, _device_semantics  # noqa: F401
from test_gpu_metric_forms import _grid

pytestmark = pytest.mark.gpu

FEW = [("two_tiles", lambda: G.dipole_grid(16, 61, 61)),
       ("nulls", lambda: G.dipole_grid(17, 61, 61, q_extent=0.5)),
       ("three_tiles", lambda: G.dipole_grid(23, 61, 77)),
       ("five_tiles", lambda: G.dipole_grid(33, 61, 61, q_extent=0.5)),
       ("x2_fastest", lambda: _grid((25, 61, 77), True, 0))]
MANY = [("nulls", lambda: G.dipole_grid(23, 129, 96, q_extent=0.5)),
        ("x2_fastest", lambda: _grid((21, 97, 129), True, 1)),
        ("unit", lambda: G.cartesian_grid(27, 129, 97, inverted=True))]


def _run(g, solver, few):
    import torch

    dg = F.DeviceGrid(g)
    assert _lib.lib().gem_diffusion_columns(dg.handle) == 0
    blocks = (((g.lx2 * g.lx3 + 31) // 32) * 7 + 3) // 4
    assert (blocks <= 3 * torch.cuda.get_device_properties(0).multi_processor_count) == few
    _check(g, solver, seed=g.lx1, J1_amp=1e-5)


@pytest.mark.parametrize("solver", [2, 1])
@pytest.mark.parametrize("name,mk", FEW, ids=[c[0] for c in FEW])
def test_few_blocks(name, mk, solver):
    _run(mk(), solver, True)


@pytest.mark.parametrize("solver", [2, 1])
@pytest.mark.parametrize("name,mk", MANY, ids=[c[0] for c in MANY])
def test_many_blocks(name, mk, solver):
    _run(mk(), solver, False)


@pytest.mark.parametrize("lx", [(64, 25, 19), (33, 13, 41), (200, 21, 9)], ids=str)
def test_short_side_of_the_line(lx):
    """The sizes of test_gpu_diffusion_paths.py::test_few_columns take the other form."""
    assert _lib.lib().gem_diffusion_columns(F.DeviceGrid(G.dipole_grid(*lx)).handle) > 0
