"""Work objects and batches on a device with little memory left: what fits without the optional
scratch still runs, with the same bits.  The memory is taken by plain torch tensors."""
import contextlib

import pytest
import torch

from gemini_b200 import _lib
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import workloads as WL

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _left(nbytes):
    """All but about nbytes of the device's memory in use."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def _run(g, dg, ds, compression):
    cfg = F.FluidCfg(ds.Teinf)
    dt = torch.full((1,), 0.2, dtype=torch.float64, device="cuda")
    if compression:
        F.fluid_adv_compression(cfg, ds, dt)
    else:
        F.fluid_adv(cfg, ds, dt)
    torch.cuda.synchronize()
    return ds.fluidvars.clone(), ds.fluidauxvars.clone()


@pytest.mark.parametrize("compression", [False, True])
def test_step_without_room_for_cut_lines(compression):
    """64x4x6000: 550 MB of blocks for the lines cut into parts, 200 MB for the diffusion."""
    g = G.cartesian_grid(64, 4, 6000)
    dg = F.DeviceGrid(g)
    a = WL.device_state(dg, g, 1)
    start, aux = a.fluidvars.clone(), a.fluidauxvars.clone()
    want = _run(g, dg, a, compression)
    a.close()
    b = WL.device_state(dg, g, 1)
    b.fluidvars.copy_(start)
    b.fluidauxvars.copy_(aux)
    with _left(450 * MB):
        _lib.check(_lib.lib().gem_work_prepare(b.work, dg.handle))
    got = _run(g, dg, b, compression)  # with the scratch it was left with
    b.close()
    for x, y in zip(got, want):
        assert torch.equal(x, y)
