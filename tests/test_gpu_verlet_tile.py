"""The one-kernel increment of grid meshes against the element and node kernels: edges of the tiles
(15 and 7 nodes), open and periodic grids, many grids in one system, both arithmetics."""

import ctypes as C

import numpy as np
import pytest
import torch

import goosefem_gb300 as gf
from goosefem_gb300 import batch
from goosefem_gb300.dynamics import VelocityVerlet, critical_dt

pytestmark = pytest.mark.gpu

# Both run the same formulas and orders of sums; the compiler may place the fused multiply-adds of the
# closed form differently: about 40 roundings of 2^-53 per value and increment, 7 increments at most.
RTOL = 7 * 40 * 2.0**-53


def _close(got, want):
    for g, w in zip(got, want):
        assert torch.isfinite(g).all()
        scale = float(w.abs().max())
        assert float((g - w).abs().max()) <= RTOL * scale


def _state(n, rng):
    return [torch.tensor(rng.uniform(-1, 1, (n, 2)), device="cuda") for _ in range(3)]


@pytest.mark.parametrize("arithmetic", ["fp64", "mixed"])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nx,ny", [(2, 2), (3, 7), (6, 8), (14, 15), (15, 29), (300, 241)])
def test_single_grid(nx, ny, periodic, arithmetic):
    rng = np.random.default_rng(nx * 1000 + ny)
    m = gf.Mesh.Quad4.Regular(nx, ny)
    K, G = rng.uniform(0.5, 1.5, nx * ny), rng.uniform(0.25, 0.75, nx * ny)
    dofs = m.dofsPeriodic() if periodic else m.dofs()
    fext = rng.uniform(-1, 1, (m.nnode(), 2))
    iip = None if periodic else dofs[m.nodesBottomEdge()].ravel()
    vv = VelocityVerlet(m.coor(), m.conn(), dofs, K, G, dt=0.1 * critical_dt(K, G), eta=0.2, iip=iip,
                        fext=None if periodic else fext, arithmetic=arithmetic)
    assert bool(vv.desc.tiles) == periodic
    for nsteps in (1, 2, 7):
        s0 = _state(m.nnode(), rng)
        got = [t.clone() for t in s0]
        vv.step(*got, nsteps)
        tiles, reg = vv.desc.tiles, (vv.desc.reg_nx, vv.desc.reg_ny)
        vv.desc.tiles, vv.desc.reg_nx, vv.desc.reg_ny = None, 0, 0
        want = [t.clone() for t in s0]
        vv.step(*want, nsteps)
        vv.desc.tiles, (vv.desc.reg_nx, vv.desc.reg_ny) = tiles, reg
        _close(got, want)


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("nmax", [9, 90])
def test_many_grids(nmax, mode):
    inst = batch.seeded_instances(5, 3, nmin=2, nmax=nmax)
    bv = batch.BatchedVerlet(inst, eta=0.1)
    bv.mode = mode
    assert bv.vv.desc.tiles
    for nsteps in (1, 4):
        got, want = bv.state(), bv.state()
        bv.run_graph(*got, nsteps)
        bv.run_graph(*got, nsteps)
        bv.release()
        tiles, bv.vv.desc.tiles = bv.vv.desc.tiles, None
        bv.run_direct(*want, 2 * nsteps)
        bv.vv.desc.tiles = tiles
        _close(got[:1], want[:1])


def test_other_numbering_and_alignment():
    """A grid with two dofs exchanged is refused by the check; states off the 16-byte boundary run."""
    from goosefem_gb300 import _lib

    rng = np.random.default_rng(0)
    m = gf.Mesh.Quad4.Regular(9, 11)
    K, G = rng.uniform(0.5, 1.5, 99), rng.uniform(0.25, 0.75, 99)
    dofs = m.dofsPeriodic().copy()
    a, b = dofs == 4, dofs == 11
    dofs[a], dofs[b] = 11, 4
    vv = VelocityVerlet(m.coor(), m.conn(), dofs, K, G, dt=0.01)
    assert vv.desc.tiles  # a renumbering of the dofs alone leaves the sums as they are
    dofs = m.dofs().copy()
    dofs[5] = dofs[70]
    vv = VelocityVerlet(m.coor(), m.conn(), dofs, K, G, dt=0.01)
    assert not vv.desc.tiles and vv.desc.reg_nx == 0

    vv = VelocityVerlet(m.coor(), m.conn(), m.dofsPeriodic(), K, G, dt=0.01, arithmetic="mixed")
    s0 = _state(m.nnode(), rng)
    want = [t.clone() for t in s0]
    vv.step(*want, 3)
    n = m.nnode() * 2
    off = torch.empty(2 * n + 1, dtype=torch.float64, device="cuda")
    v, a = off[1:n + 1], off[n + 1:]
    v.copy_(s0[1].ravel())
    a.copy_(s0[2].ravel())
    u = s0[0].clone()
    st = torch.cuda.current_stream().cuda_stream
    _lib.call("gfgpu_verlet_step", C.addressof(vv.desc), u.data_ptr(), v.data_ptr(), a.data_ptr(), 3,
              vv.ws.data_ptr(), st)
    _close([u, v.view(-1, 2), a.view(-1, 2)], want)
