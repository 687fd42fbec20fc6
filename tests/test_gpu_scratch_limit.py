"""Work objects and batches on a device with little memory left: what fits without the optional
scratch still runs, with the same bits.  The memory is taken by plain torch tensors."""
import contextlib

import pytest
import torch

from gemini_b200 import _lib
from gemini_b200 import batch as BT
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


def _mixed(lx1, lx23, n):
    """n Cartesian and n dipole instances of the same sizes, and their plain copies."""
    grids = [G.cartesian_grid(lx1, lx23, lx23) for _ in range(n)] + [G.dipole_grid(lx1, lx23, lx23) for _ in range(n)]
    out = []
    for k, g in enumerate(grids):
        dg = F.DeviceGrid(g)
        a, b = (WL.device_state(dg, g, k) for _ in range(2))
        b.fluidvars.copy_(a.fluidvars)
        b.fluidauxvars.copy_(a.fluidauxvars)
        out.append(((dg, a, F.FluidCfg(a.Teinf)), (dg, b, F.FluidCfg(b.Teinf))))
    return out


def _batch_bytes(insts):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    b = BT.Batch(insts)
    return b, before - torch.cuda.mem_get_info()[0]


def _check(b, insts):
    for _ in range(2):
        b.step()
        for _, p in insts:
            BT.plain_step(*p)
    torch.cuda.synchronize()
    for (_, x, _), (_, y, _) in insts:
        assert torch.equal(x.fluidvars, y.fluidvars) and torch.equal(x.fluidauxvars, y.fluidauxvars)


def test_batch_scratch_fits_its_instances():
    """Two instances of 40x8x8 are 14 warps of columns each: a few MB, not a slot for every warp
    that the device holds."""
    insts = _mixed(40, 8, 1)
    BT.Batch([i[0] for i in insts]).close()  # loads the kernels
    b, used = _batch_bytes([i[0] for i in insts])
    assert used < 16 * MB, used
    _check(b, insts)


def test_batch_without_room_for_two_chains():
    """Mixed instances that fill every slot of both variants: with room for one scratch only, the
    batch runs as one chain, with the same bits."""
    insts = _mixed(200, 80, 2)
    first = [i[0] for i in insts]
    b, both = _batch_bytes(first)
    b.close()
    with _left(both - both // 4):
        b, one = _batch_bytes(first)
    assert one < both - both // 4
    _check(b, insts)
