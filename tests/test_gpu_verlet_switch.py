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
