"""The dt schedule of a differentiable problem as host logic (no GPU): a list, tuple or array, its
copy made again when it changes in value or length."""
import numpy as np
import pytest
import torch

from gemini_b200 import adjoint as AD


def _problem(dts):
    P = AD.DiffProblem.__new__(AD.DiffProblem)
    P.base = torch.zeros(1, dtype=torch.float64)
    P._dtt = P._dtt_of = None
    P._sa = None
    P.dts = dts
    return P


@pytest.mark.parametrize("kind", [list, tuple, np.array, torch.tensor])
def test_schedule_kinds(kind):
    v = [0.5, 0.25, 0.125]
    P = _problem(kind(v))
    for _ in range(2):
        assert [P.dt_tensor(j).item() for j in range(3)] == v
    first = P.dt_tensor(0).data_ptr()
    assert first == P.dt_tensor(0).data_ptr()  # one copy while nothing changes
    P.dts = kind([0.5, 0.75])
    assert [P.dt_tensor(j).item() for j in range(2)] == [0.5, 0.75]
    P.dts = kind(v)
    assert P.dt_tensor(2).item() == 0.125
