"""The explicit increment on both sides of the sizes at which its kernels change, bit for bit: FP64 takes
one kernel per increment (k_verlet_tile) up to 456 tiles of 7 x 7 nodes and an element and a node kernel
above; mixed arithmetic tiles of 7 x 7 nodes while those of 15 x 15 are fewer than 456."""

import numpy as np
import pytest
import torch

import goosefem_gb300 as gf
from goosefem_gb300.dynamics import VelocityVerlet, critical_dt

pytestmark = pytest.mark.gpu

FEW = 456


def tiles(nx, ny, edge):
    n = edge - 1
    return (nx + n) // n * ((ny + n) // n)


def _mesh(nx, ny, periodic, fext, arithmetic="fp64"):
    gf.set_strict(False)
    rng = np.random.default_rng(nx * 1000 + ny)
    m = gf.Mesh.Quad4.Regular(nx, ny)
    K, G = rng.uniform(0.5, 1.5, nx * ny), rng.uniform(0.25, 0.75, nx * ny)
    dofs = m.dofsPeriodic() if periodic else m.dofs()
    iip = None if periodic else dofs[m.nodesBottomEdge()].ravel()
    f = rng.uniform(-1, 1, (m.nnode(), 2)) if fext else None
    vv = VelocityVerlet(m.coor(), m.conn(), dofs, K, G, dt=0.1 * critical_dt(K, G), eta=0.2, iip=iip, fext=f,
                        arithmetic=arithmetic)
    return vv, [torch.tensor(rng.uniform(-1, 1, (m.nnode(), 2)), device="cuda") for _ in range(3)]


def _run(vv, state, nsteps):
    s = [t.clone() for t in state]
    vv.step(*s, nsteps)
    return s


@pytest.mark.parametrize("fext", [False, True])
def test_regular_node_kernel_gives_the_csr_bits(fext):
    """Above the limit of the one-kernel increment: element forces by index arithmetic against the CSR."""
    vv, s0 = _mesh(160, 153, False, fext)
    assert tiles(160, 153, 8) > FEW and vv.desc.reg_nx == 160
    got = _run(vv, s0, 9)
    vv.use_csr_gather()
    for g, w in zip(got, _run(vv, s0, 9)):
        assert torch.isfinite(g).all() and torch.equal(g, w)


def _without_tiles(vv, f):
    """f() on the element and node kernels."""
    d = vv.desc
    keep = d.tiles, d.reg_nx, d.reg_ny
    d.tiles, d.reg_nx, d.reg_ny = None, 0, 0
    out = f()
    d.tiles, d.reg_nx, d.reg_ny = keep
    return out


# (nx, ny), arithmetic, elements along a tile's edge
ONE_KERNEL = [((146, 139), "fp64", 8), ((2, 2), "fp64", 8), ((300, 241), "mixed", 8), ((331, 317), "mixed", 16)]


@pytest.mark.parametrize("fext", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("size,arithmetic,edge", ONE_KERNEL)
def test_one_kernel_gives_the_two_kernels_bits(size, arithmetic, edge, periodic, fext):
    nx, ny = size
    assert edge == (8 if tiles(nx, ny, 16) < FEW else 16) and (arithmetic == "mixed" or tiles(nx, ny, 8) <= FEW)
    vv, s0 = _mesh(nx, ny, periodic, fext and not periodic, arithmetic)
    if periodic:
        assert vv.desc.tiles and vv.desc.tile_edge == edge and vv.desc.ntiles == tiles(nx, ny, edge)
    else:
        assert (vv.desc.reg_nx, vv.desc.reg_ny) == size
    for nsteps in (1, 6):
        got = _run(vv, s0, nsteps)
        for g, w in zip(got, _without_tiles(vv, lambda: _run(vv, s0, nsteps))):
            assert torch.isfinite(g).all() and torch.equal(g, w)


@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("nmin,nmax,edge", [(2, 40, 8), (200, 300, 16)])
def test_many_grids_give_the_two_kernels_bits(nmin, nmax, edge, mode):
    """u, v and a of several grids in one table, from a random state."""
    from goosefem_gb300 import batch

    gf.set_strict(False)
    bv = batch.BatchedVerlet(batch.seeded_instances(5, 3, nmin=nmin, nmax=nmax), eta=0.1)
    bv.mode = mode
    assert bv.vv.desc.tiles and bv.vv.desc.tile_edge == edge
    rng = np.random.default_rng(nmax)
    s0 = [torch.tensor(rng.uniform(-1, 1, (bv.nnode, 2)), device="cuda") for _ in range(3)]

    def run():
        s = [t.clone() for t in s0]
        bv.run_direct(*s, 5)
        return s

    got = run()
    for g, w in zip(got, _without_tiles(bv.vv, run)):
        assert torch.isfinite(g).all() and torch.equal(g, w)


@pytest.mark.parametrize("mode", [0, 3])
def test_gather_table_of_the_node_kernels(mode):
    """The two kernels with the gather table (meshes without a grid numbering) against the dof CSR."""
    from goosefem_gb300 import batch

    gf.set_strict(False)
    bv = batch.BatchedVerlet(batch.seeded_instances(4, 7, nmin=8, nmax=40), eta=0.1)
    bv.mode = mode
    d = bv.vv.desc
    d.tiles = None
    assert d.ell and d.reg_nx == 0
    out = []
    for ell in (d.ell, None):
        d.ell = ell
        s = bv.state()
        bv.run_direct(*s, 30)
        out.append(s)
    for g, w in zip(*out):
        assert torch.isfinite(g).all() and torch.equal(g, w)


def test_partition_across_the_switch():
    """Three ranks whose meshes take the one kernel, of a mesh that takes two: the single-domain bits."""
    from goosefem_gb300 import partition as P

    nx, ny, world, nsteps = 200, 190, 3, 12
    vv, s0 = _mesh(nx, ny, False, False)
    assert tiles(nx, ny, 8) > FEW
    m = gf.Mesh.Quad4.Regular(nx, ny)
    K, G = vv.K.cpu().numpy(), vv.G.cpu().numpy()
    want = _run(vv, s0, nsteps)
    runs = []
    for r in range(world):
        part = P.RowBlockPartition(nx, ny, world, r)
        assert tiles(nx, part.local_ny, 8) <= FEW
        coor, conn, dofs, Kl, Gl, iip, _ = P.local_problem(part, K, G)
        lv = VelocityVerlet(coor, conn, dofs, Kl, Gl, dt=vv.dt, eta=vv.eta, iip=iip)
        run = P.RankRun(part, P.FP64Engine(lv))
        rows = torch.as_tensor(part.node_rows(), device="cuda")
        run.begin(*(t[rows].clone() for t in s0))
        runs.append(run)
    for it in range(nsteps):
        for run in runs:
            run.increment(it, it + 1 == nsteps)
        if it + 1 < nsteps:
            outs = [run.halo_out(it) for run in runs]
            for r, run in enumerate(runs):
                run.halo_in(it, outs[r - 1][1].clone() if r else None, outs[r + 1][0].clone() if r + 1 < world else None)
    W = nx + 1
    assert m.nnode() == W * (ny + 1)
    for run in runs:
        lo, hi = run.part.owned()
        for g, w in zip(run.end(nsteps - 1), want):
            assert torch.equal(g[lo * W:hi * W], w[run.part.r0 * W:run.part.r1 * W])
