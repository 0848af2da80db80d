"""The pair stiffness action of the Jacobi-PCG where its blocks end. Hex8: warps of 31 node columns, rows
of 1 to 63 elements, one and several warps per row, rows shared by a warp. Quad4: tiles of 15 nodes, and a
mesh of more tiles than the one-kernel operator takes."""

import ctypes as C

import numpy as np
import pytest
import torch

import goosefem_gb300 as gf
import goosefem_gb300.statics  # noqa: F401

from _common import seeded_material, to_np

pytestmark = pytest.mark.gpu


def _check(st, iip, nnode, nd, seed):
    """q = A p0 within 1e-12 of max |A p0| of the FP64 operator (pairs carry ~48 bits), 0 on prescribed."""
    from goosefem_gb300 import _dev, _lib

    assert st.arithmetic == "pair"
    n = nnode * nd
    x = torch.tensor(np.random.default_rng(seed).uniform(-1, 1, n), device="cuda")
    stream = _dev.stream()
    _lib.call("gfgpu_pcg_begin", C.addressof(st.desc), st.diag.data_ptr(), None, x.data_ptr(), st.ws.data_ptr(), stream)

    def vec(which):
        p = C.c_void_p(None)
        _lib.call("gfgpu_pcg_vector", C.addressof(st.desc), st.ws.data_ptr(), which, C.addressof(p))
        off = (p.value - st.ws.data_ptr()) // 8
        return st.ws[off:off + n]

    p0 = vec(2).clone()
    _lib.call("gfgpu_pcg_iterate", C.addressof(st.desc), 1, x.data_ptr(), st.ws.data_ptr(), stream)
    q = to_np(vec(3))
    f = to_np(st.force(p0.view(-1, nd))).ravel()
    free = np.setdiff1d(np.arange(n), iip)
    assert np.max(np.abs(q[iip])) == 0.0
    err = np.max(np.abs(q[free] - f[free])) / np.max(np.abs(f[free]))
    assert err <= 1e-12, err


@pytest.mark.parametrize("nx,ny,nz", [(1, 4, 5), (5, 7, 2), (30, 2, 3), (31, 1, 2), (32, 3, 1), (61, 2, 2), (63, 2, 1)])
def test_pair_action_hex8(oracle, nx, ny, nz):
    coor, conn = oracle.hex8_regular(nx, ny, nz)
    K, G = seeded_material(conn.shape[0], 48)
    nxy = (nx + 1) * (ny + 1)
    front = np.arange(nxy)
    back = front + nz * nxy
    iip = np.unique(np.concatenate([(front[:, None] * 3 + np.arange(3)).ravel(), back * 3 + 2]))
    nnode = coor.shape[0]
    st = gf.statics.ElasticStatic(coor, conn, np.arange(nnode * 3).reshape(-1, 3), K, G, iip, arithmetic="pair")
    _check(st, iip, nnode, 3, nx)


@pytest.mark.parametrize("nx,ny", [(1, 2), (13, 14), (14, 15), (15, 13), (29, 31), (254, 249), (270, 275)])
def test_pair_action_quad4(oracle, nx, ny):
    coor, conn = oracle.quad4_regular(nx, ny)
    K, G = seeded_material(conn.shape[0], 49)
    bot = np.arange(nx + 1)
    top = bot + ny * (nx + 1)
    iip = np.unique(np.concatenate([(bot[:, None] * 2 + np.arange(2)).ravel(), top * 2 + 1]))
    nnode = coor.shape[0]
    st = gf.statics.ElasticStatic(coor, conn, np.arange(nnode * 2).reshape(-1, 2), K, G, iip, arithmetic="pair")
    _check(st, iip, nnode, 2, nx)
