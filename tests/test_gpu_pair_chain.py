"""Float-float increments call by call, with the coefficients written anew between the calls: the next
call's kernels read what the kernel just before it wrote, synchronised or not."""

import ctypes as C

import numpy as np
import pytest
import torch

import goosefem_gb300 as gf
from goosefem_gb300 import _dev, _lib
from goosefem_gb300.dynamics import VelocityVerlet, critical_dt

pytestmark = pytest.mark.gpu


def _steps(vv, K0, G0, state, sync):
    d, ws, st = C.addressof(vv.desc), vv.ws.data_ptr(), _dev.stream()
    s = [t.clone() for t in state]
    p = [t.data_ptr() for t in s]
    vv.K.copy_(K0)
    vv.G.copy_(G0)
    _lib.call("gfgpu_verlet_precompute_pair", d, vv.coef_pair.data_ptr(), st)
    _lib.call("gfgpu_verlet_pair_begin", d, *p, ws, st)
    n, at = (1, 2, 3, 1), 0
    for k, count in enumerate(n):
        last = k + 1 == len(n)
        vv.K.mul_(0.75)
        vv.G.mul_(0.5)
        _lib.call("gfgpu_verlet_precompute_pair", d, vv.coef_pair.data_ptr(), st)
        if sync:
            torch.cuda.synchronize()
        _lib.call("gfgpu_verlet_pair_increments", d, at, count, 0 if last else 1, ws, st)
        at += count
    _lib.call("gfgpu_verlet_pair_end", d, at - 1, *p, ws, st)
    torch.cuda.synchronize()
    return s


@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("nx,ny", [(9, 7), (300, 170)])
def test_coefficients_written_between_calls(mode, nx, ny):
    gf.set_strict(False)
    rng = np.random.default_rng(nx + mode)
    m = gf.Mesh.Quad4.Regular(nx, ny)
    K, G = rng.uniform(0.5, 1.5, nx * ny), rng.uniform(0.25, 0.75, nx * ny)
    coor = m.coor()
    if mode == 3:
        coor = coor + rng.uniform(-0.1, 0.1, coor.shape)
    vv = VelocityVerlet(coor, m.conn(), m.dofsPeriodic() if mode == 2 else m.dofs(), K, G,
                        dt=0.05 * critical_dt(K, G), eta=0.1, arithmetic="pair")
    assert vv.desc.pair_mode == mode
    state = [torch.tensor(rng.uniform(-1, 1, (m.nnode(), 2)), device="cuda") for _ in range(3)]
    K0, G0 = vv.K.clone(), vv.G.clone()
    want = _steps(vv, K0, G0, state, True)
    for _ in range(5):
        for g, w in zip(_steps(vv, K0, G0, state, False), want):
            assert torch.isfinite(g).all() and torch.equal(g, w)
