"""Infinities and NaN in the inputs: fast arithmetic puts NaN and infinities where the oracle has them."""

import numpy as np
import pytest

from _common import seeded_field, to_np

pytestmark = pytest.mark.gpu

SPECIAL = (np.inf, -np.inf, np.nan)


@pytest.fixture(scope="module")
def gf():
    import goosefem_gb300 as gf

    gf.set_strict(False)
    return gf


def _same_kind(got, ref):
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], ref[inf])


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("nip", [1, 3, 4])
@pytest.mark.parametrize("nd", [2, 3])
def test_stress(gf, oracle, nd, nip, symmetric):
    ne = 97
    eps = seeded_field((ne, nip, nd, nd), 1)
    if symmetric:
        eps = eps + eps.swapaxes(2, 3)
    n = 0
    for i in range(nd):
        for j in range(nd):
            for s in SPECIAL:
                eps[5 * n % ne, n % nip, i, j] = s
                if symmetric:
                    eps[5 * n % ne, n % nip, j, i] = s
                n += 1
    K, G = np.abs(seeded_field((2, ne), 2)) + 0.2
    with np.errstate(invalid="ignore"):
        ref = oracle.elastic_stress(eps, K, G)
    _same_kind(to_np(gf.elastic_stress(eps, K, G)), ref)
    assert np.isnan(ref).any() and np.isinf(ref).any()


@pytest.mark.parametrize("nd,dims", [(2, (9, 7)), (3, (5, 4, 3))])
def test_general_element_forces(gf, oracle, nd, dims):
    from goosefem_gb300 import ElasticStatic

    R = oracle
    mesh = (gf.Mesh.Quad4 if nd == 2 else gf.Mesh.Hex8).Regular(*dims)
    conn, dofs = mesh.conn(), mesh.dofs()
    coor = mesh.coor() + seeded_field((mesh.nnode(), nd), 3, amp=0.15)
    K, G = np.abs(seeded_field((2, mesh.nelem()), 4)) + 0.2
    st = ElasticStatic(coor, conn, dofs, K, G, np.arange(nd, dtype=np.int32), uniform=False)
    dNx, vol = R.compute_dN(R.as_element(conn, coor), *(R.quad4_gauss() if nd == 2 else R.hex8_gauss()))
    for k, s in enumerate(SPECIAL):
        u = seeded_field((mesh.nnode(), nd), 5)
        u[mesh.nnode() // 2, k % nd] = s
        with np.errstate(invalid="ignore"):
            sig = R.elastic_stress(R.sym_grad_n_vector(dNx, R.as_element(conn, u)), K, G)
            ref = R.assemble_node(conn, dofs, R.int_grad_n_dot_tensor2_dv(dNx, vol, sig))
        got = to_np(st.force(u))
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and not np.isinf(got).any()


@pytest.mark.parametrize("where", [(0, 0, 34), (1, 34, 0), (0, 20, 17), (1, 34, 34), (0, 16, 15), (0, 31, 31)])
def test_network_gradients(gf, where):
    """A NaN in a crop whose edge is no multiple of the tiles' 16 pixels. The ReLU after the first layer (a
    maximum with 0) turns what it makes of it into 0, so NaN is left in the first layer's weight gradient,
    for the channel and the taps that bring a pixel of the image to it, and nowhere else."""
    import torch
    from goosefem_gb300 import _lib

    layers = ((4, 32), (32, 32), (32, 32), (32, 2))
    rng = np.random.default_rng(1)
    flat = np.concatenate([a for ci, co in layers for a in (rng.normal(0.0, np.sqrt(2.0 / (9 * ci)), 9 * ci * co),
                                                           rng.normal(0.0, 0.1, co))]).astype(np.float32)
    B, S, ch = 2, 35, 1
    X = rng.normal(size=(B, S, S, 4)).astype(np.float32)
    T = rng.normal(size=(B, S, S, 2)).astype(np.float32)
    X[where + (ch,)] = np.nan
    flat, Xd, Td = (torch.tensor(a, device="cuda") for a in (flat, X, T))
    ws = torch.empty(int(_lib.lib().gfgpu_nn_train_workspace_bytes(B, S, S)) // 4 + 1, dtype=torch.float32, device="cuda")
    g, loss = torch.empty_like(flat), torch.empty(1, dtype=torch.float32, device="cuda")
    wb = flat.to(torch.bfloat16)
    _lib.call("gfgpu_nn_train_step", wb.data_ptr(), flat.data_ptr(), Xd.data_ptr(), Td.data_ptr(), None, None, B, S,
              4, g.data_ptr(), loss.data_ptr(), ws.data_ptr(), torch.cuda.current_stream().cuda_stream)
    want = np.zeros(flat.numel(), dtype=bool)
    first = want[:9 * 4 * 32].reshape(9, 4, 32)
    for t in range(9):
        y, x = where[1] - (t // 3 - 1), where[2] - (t % 3 - 1)
        first[t, ch] = 0 <= y < S and 0 <= x < S
    assert np.array_equal(np.isnan(g.cpu().numpy()), want) and bool(torch.isfinite(g[~g.isnan()]).all())
