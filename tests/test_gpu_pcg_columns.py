"""The pair stiffness action of the Hex8 Jacobi-PCG where its warps of 31 node columns end: rows of 1 to
63 elements, one and several warps per row, rows shared by a warp."""

import ctypes as C

import numpy as np
import pytest
import torch

import goosefem_gb300 as gf
import goosefem_gb300.statics  # noqa: F401

from _common import seeded_material, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(1, 4, 5), (5, 7, 2), (30, 2, 3), (31, 1, 2), (32, 3, 1), (61, 2, 2), (63, 2, 1)])
def test_pair_action(oracle, nx, ny, nz):
    """q = A p0 within 1e-12 of max |A p0| of the FP64 operator (pairs carry ~48 bits), 0 on prescribed."""
    from goosefem_gb300 import _dev, _lib

    coor, conn = oracle.hex8_regular(nx, ny, nz)
    K, G = seeded_material(conn.shape[0], 48)
    nxy = (nx + 1) * (ny + 1)
    front = np.arange(nxy)
    back = front + nz * nxy
    iip = np.unique(np.concatenate([(front[:, None] * 3 + np.arange(3)).ravel(), back * 3 + 2]))
    nnode = coor.shape[0]
    st = gf.statics.ElasticStatic(coor, conn, np.arange(nnode * 3).reshape(-1, 3), K, G, iip, arithmetic="pair")
    assert st.arithmetic == "pair"
    x = torch.tensor(np.random.default_rng(nx).uniform(-1, 1, nnode * 3), device="cuda")
    stream = _dev.stream()
    _lib.call("gfgpu_pcg_begin", C.addressof(st.desc), st.diag.data_ptr(), None, x.data_ptr(), st.ws.data_ptr(), stream)

    def vec(which):
        p = C.c_void_p(None)
        _lib.call("gfgpu_pcg_vector", C.addressof(st.desc), st.ws.data_ptr(), which, C.addressof(p))
        off = (p.value - st.ws.data_ptr()) // 8
        return st.ws[off:off + nnode * 3]

    p0 = vec(2).clone()
    _lib.call("gfgpu_pcg_iterate", C.addressof(st.desc), 1, x.data_ptr(), st.ws.data_ptr(), stream)
    q = to_np(vec(3))
    f = to_np(st.force(p0.view(-1, 3))).ravel()
    free = np.setdiff1d(np.arange(nnode * 3), iip)
    assert np.max(np.abs(q[iip])) == 0.0
    err = np.max(np.abs(q[free] - f[free])) / np.max(np.abs(f[free]))
    assert err <= 1e-12, err
