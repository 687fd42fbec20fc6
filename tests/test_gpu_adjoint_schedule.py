"""A changed dt schedule of a differentiable problem reaches the next pass."""
import pytest

from gemini_b200 import adjoint as AD
from gemini_b200 import grid as G
from gemini_b200 import state as S

pytestmark = pytest.mark.gpu


def test_schedule_changed_after_use():
    g = G.cartesian_grid(24, 8, 6)
    P = AD.DiffProblem(g, S.init_state(g, seed=2, perturb=0.1), 2, checkpoint_every=1)
    assert [P.dt_tensor(j).item() for j in range(2)] == P.dts
    P.dts[1] *= 0.5
    assert [P.dt_tensor(j).item() for j in range(2)] == P.dts
