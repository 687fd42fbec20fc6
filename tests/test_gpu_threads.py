"""Host threads that work on grids of different sizes at the same time: each call asks for its own
size of dynamic shared memory, and none may take another's away between setting and launch.
The C entry points are called in tight loops (the calls run without Python's lock); results as
one thread alone, bit for bit."""
import ctypes
import threading

import pytest
import torch

from gemini_b200 import _lib
from gemini_b200 import fluid as F
from gemini_b200 import grid as G
from gemini_b200 import state as S

pytestmark = pytest.mark.gpu


def _in_threads(calls, rounds, n):
    """Each call(stream) rounds * n times in a thread of its own on a stream of its own; every call
    must return GEM_OK."""
    bad = []
    gate = threading.Barrier(len(calls))

    def body(call):
        stream = torch.cuda.Stream()
        s = ctypes.c_void_p(stream.cuda_stream)
        gate.wait(60)
        for _ in range(rounds):
            bad.extend(rc for rc in [call(s) for _ in range(n)] if rc)
            stream.synchronize()

    ts = [threading.Thread(target=body, args=(c,)) for c in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join(120)
    torch.cuda.synchronize()
    return bad


def _grids(sizes):
    for lx in sizes:
        g = G.cartesian_grid(*lx)
        st = S.init_state(g, seed=lx[0], perturb=0.1)
        yield F.DeviceGrid(g), st, ctypes.byref(F.FluidCfg(st.Teinf).c())


def test_diffusion_of_long_and_longer_columns():
    """1600 and 2800 rows: one column per block in 64 and 112 KB of shared memory."""
    L = _lib.lib()
    calls, states = [], []
    for dg, st, cfg in _grids([(1600, 2, 1), (2800, 2, 1)]):
        assert L.gem_diffusion_columns(dg.handle) == 1
        dt = torch.full((1,), 1e-3, dtype=torch.float64, device="cuda")
        pair = [F.DeviceState.from_host(dg, st.copy()) for _ in range(2)]
        for ds in pair:
            args = (cfg, dg.handle, F._ptr(ds.fluidvars), F._ptr(ds.electrovars), ds.work, F._ptr(dt))
            calls.append(lambda s, a=args: L.gem_energy_diffusion_dev(*a, s))
            assert L.gem_work_prepare(ds.work, dg.handle) == 0
        states.append((pair, dt))
    alone, together = calls[0::2], calls[1::2]
    for c in alone:
        for _ in range(600):
            assert c(None) == 0
    torch.cuda.synchronize()
    assert _in_threads(together, 6, 100) == []
    for (a, b), _ in states:
        assert torch.equal(a.fluidvars, b.fluidvars)


def test_diffusion_adjoint_of_short_and_long_columns():
    """40 and 500 rows: 57 and 229 KB of shared memory a block."""
    L = _lib.lib()
    calls, keep = [], []
    for dg, st, cfg in _grids([(40, 2, 2), (500, 2, 2)]):
        ds = F.DeviceState.from_host(dg, st.copy())
        ng = dg.ng
        n, T = ds.fluidvars[:7 * ng], ds.fluidvars[28 * ng:]
        dt = torch.full((1,), 1e-3, dtype=torch.float64, device="cuda")
        Y = torch.ones_like(T)
        outs = []
        for _ in range(2):
            o = [torch.zeros_like(T), torch.zeros_like(T), torch.zeros(28, dtype=torch.float64, device="cuda")]
            args = [cfg, dg.handle] + [F._ptr(x) for x in (T, n, ds.electrovars)] + [ds.work] + \
                [F._ptr(x) for x in [dt, Y] + o]
            calls.append(lambda s, a=args: L.gem_diffusion_vjp_dev(*a, s))
            outs.append(o)
        keep.append((ds, n, T, dt, Y, outs))
    for c in calls[0::2]:
        assert c(None) == 0
    torch.cuda.synchronize()
    assert _in_threads(calls[1::2], 6, 100) == []
    for k in keep:
        assert all(torch.equal(x, y) for x, y in zip(*k[-1]))
