"""The fast forms of the element operators at the edges of their blocks and at every number of
integration points they stage apart, against the CPU oracle (the reference's loops).

Tolerance: the operators reorder sums of at most 24 products of FP64 values (72 for the stiffness
integral, two factors deep); 1e-12 of the largest value is the project's bound for fast mode, about
4500 units of 2^-52.
"""

import numpy as np
import pytest

from _common import RTOL, rel_err, seeded_field, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gf():
    import goosefem_gb300 as gf

    gf.set_strict(False)
    return gf


def _rule(nd, nip, seed):
    """`nip` points inside the element with positive weights."""
    rng = np.random.default_rng(seed)
    return rng.uniform(-0.8, 0.8, (nip, nd)), rng.uniform(0.5, 1.5, nip)


def _elements(nelem, nd, seed):
    """`nelem` separate distorted unit elements, as an elemvec."""
    s = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], dtype=np.float64)
    if nd == 3:
        s = np.concatenate([np.c_[s, np.zeros(4)], np.c_[s, np.ones(4)]])
    return s[None] + seeded_field((nelem,) + s.shape, seed, amp=0.15)


@pytest.mark.parametrize("planar", [False, True])
@pytest.mark.parametrize("nip", [1, 3, 4, 9])
@pytest.mark.parametrize("nelem", [1, 15, 16, 17, 250])
def test_stiffness_quad4(gf, oracle, nelem, nip, planar):
    R, td = oracle, 3 if planar else 2
    x = _elements(nelem, 2, nelem)
    xi, w = _rule(2, nip, nip)
    quad = (gf.Element.Quad4.QuadraturePlanar if planar else gf.Element.Quad4.Quadrature)(x, xi, w)
    C = seeded_field((nelem, nip) + (td,) * 4, 3)
    dNx, vol = R.quad4_planar_compute_dN(x, xi, w, thick=1.0) if planar else R.compute_dN(x, xi, w)
    ref = (R.int_grad_n_dot_tensor4_dot_grad_nt_dv_planar if planar
           else R.int_grad_n_dot_tensor4_dot_grad_nt_dv)(dNx, vol, C)
    assert rel_err(to_np(quad.Int_gradN_dot_tensor4_dot_gradNT_dV(C)), ref) <= RTOL


@pytest.mark.parametrize("nip", [1, 7, 8, 11])
@pytest.mark.parametrize("nelem", [1, 3, 4, 5, 61])
def test_stiffness_hex8(gf, oracle, nelem, nip):
    R = oracle
    x = _elements(nelem, 3, nelem)
    xi, w = _rule(3, nip, nip)
    quad = gf.Element.Hex8.Quadrature(x, xi, w)
    C = seeded_field((nelem, nip, 3, 3, 3, 3), 4)
    dNx, vol = R.compute_dN(x, xi, w)
    ref = R.int_grad_n_dot_tensor4_dot_grad_nt_dv(dNx, vol, C)
    assert rel_err(to_np(quad.Int_gradN_dot_tensor4_dot_gradNT_dV(C)), ref) <= RTOL


@pytest.mark.parametrize("nip", [1, 3, 8])
@pytest.mark.parametrize("nelem,nd", [(1, 2), (127, 2), (129, 2), (1, 3), (33, 3), (257, 3)])
def test_gradients_stress_and_forces(gf, oracle, nelem, nip, nd):
    """The operator chain on separate elements, and the fused element forces of the same elements."""
    R = oracle
    x = _elements(nelem, nd, 10 + nelem)
    xi, w = _rule(nd, nip, nip)
    quad = (gf.Element.Quad4 if nd == 2 else gf.Element.Hex8).Quadrature(x, xi, w)
    dNx, vol = R.compute_dN(x, xi, w)
    ue = seeded_field(x.shape, 11)
    K, G = np.abs(seeded_field((2, nelem), 12)) + 0.2
    eps = R.sym_grad_n_vector(dNx, ue)
    sig = R.elastic_stress(eps, K, G)
    assert rel_err(to_np(quad.GradN_vector(ue)), R.grad_n_vector(dNx, ue)) <= RTOL
    assert rel_err(to_np(quad.GradN_vector_T(ue)), R.grad_n_vector_T(dNx, ue)) <= RTOL
    assert rel_err(to_np(quad.SymGradN_vector(ue)), eps) <= RTOL
    assert rel_err(to_np(gf.elastic_stress(eps, K, G)), sig) <= RTOL
    # a strain that is not symmetric keeps its two off-diagonal parts
    h = R.grad_n_vector(dNx, ue)
    assert rel_err(to_np(gf.elastic_stress(h, K, G)), R.elastic_stress(h, K, G)) <= RTOL
    fe = R.int_grad_n_dot_tensor2_dv(dNx, vol, sig)
    assert rel_err(to_np(quad.Int_gradN_dot_tensor2_dV(sig)), fe) <= RTOL


@pytest.mark.parametrize("nd,dims", [(2, (1, 1)), (2, (43, 3)), (3, (1, 1, 1)), (3, (5, 9, 3))])
def test_element_forces_and_gather(gf, oracle, nd, dims):
    """AsElement and the general element kernel of a distorted mesh against the oracle's chain."""
    from goosefem_gb300 import ElasticStatic

    R = oracle
    mesh = (gf.Mesh.Quad4 if nd == 2 else gf.Mesh.Hex8).Regular(*dims)
    conn, dofs = mesh.conn(), mesh.dofs()
    coor = mesh.coor() + seeded_field((mesh.nnode(), nd), 20, amp=0.15)
    K, G = np.abs(seeded_field((2, mesh.nelem()), 21)) + 0.2
    u = seeded_field((mesh.nnode(), nd), 22)
    st = ElasticStatic(coor, conn, dofs, K, G, np.arange(nd, dtype=np.int32), uniform=False)
    dNx, vol = R.compute_dN(R.as_element(conn, coor), *(R.quad4_gauss() if nd == 2 else R.hex8_gauss()))
    ue = R.as_element(conn, u)
    assert np.array_equal(to_np(st.vector.AsElement(u)), ue)
    fe = R.int_grad_n_dot_tensor2_dv(dNx, vol, R.elastic_stress(R.sym_grad_n_vector(dNx, ue), K, G))
    assert rel_err(to_np(st.force(u)), R.assemble_node(conn, dofs, fe)) <= RTOL


def test_unaligned_vectors(gf):
    """2-d vectors and strains off the 16-byte boundary: the same bits as aligned ones."""
    import torch
    from goosefem_gb300 import _lib

    s = torch.cuda.current_stream().cuda_stream
    mesh = gf.Mesh.Quad4.Regular(19, 14)
    conn = torch.tensor(mesh.conn(), device="cuda")
    n, ne = mesh.nnode(), mesh.nelem()
    u = torch.tensor(seeded_field((n, 2), 30), device="cuda")
    eps = torch.tensor(seeded_field((ne, 4, 2, 2), 31), device="cuda")
    K, G = torch.tensor(np.abs(seeded_field((2, ne), 32)), device="cuda")

    def off(t):
        o = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:]
        o.copy_(t.reshape(-1))
        return o

    for shift in (False, True):
        a, e = (off(u), off(eps)) if shift else (u, eps)
        ue, sig = torch.empty(ne * 8 + 1, dtype=u.dtype, device="cuda"), torch.empty(ne * 16 + 1, dtype=u.dtype, device="cuda")
        ue, sig = (ue[1:], sig[1:]) if shift else (ue[:-1], sig[:-1])
        _lib.call("gfgpu_as_element", conn.data_ptr(), ne, 4, 2, a.data_ptr(), ue.data_ptr(), s)
        _lib.call("gfgpu_elastic_stress", e.data_ptr(), K.data_ptr(), G.data_ptr(), ne, 4, 2, sig.data_ptr(), s)
        if not shift:
            want = ue.clone(), sig.clone()
    assert torch.equal(ue, want[0]) and torch.equal(sig, want[1])
    assert torch.equal(ue.reshape(ne, 4, 2), u[conn.long()])


def _stiffness_bound(dNx, vol, C):
    """Sum of the magnitudes of an entry's terms: 2^-53 of it is one rounding."""
    a = np.abs
    t = np.einsum("eqmi,eqijkl->eqmjkl", a(dNx), a(C) * vol[..., None, None, None, None])
    k = dNx.shape[2] * dNx.shape[3]
    return np.einsum("eqmjkl,eqnl->emjnk", t, a(dNx)).reshape(-1, k, k)


@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("stretch,scale", [(1.0, "one"), (40.0, "one"), (1e5, "one"), (1.0, "wide"), (1.0, "blocks"),
                                           (1.0, "huge"), (1.0, "tiny"), (1e-3, "zero")])
def test_stiffness_scales(gf, oracle, nd, stretch, scale):
    """Thin elements and tensors whose entries or blocks lie far apart: every entry to within 64
    roundings of its terms (the oracle's own sum of 64 to 72 terms takes up to as many; integer sums
    and the FP64 form for what they do not cover)."""
    R = oracle
    x = _elements(37, nd, 5)
    x[..., 0] *= stretch
    quad = (gf.Element.Quad4 if nd == 2 else gf.Element.Hex8).Quadrature(x)
    dNx, vol = R.compute_dN(x, *(R.quad4_gauss() if nd == 2 else R.hex8_gauss()))
    C = seeded_field(vol.shape + (nd,) * 4, 6)
    if scale == "wide":
        C *= 10.0 ** (6.0 * seeded_field(C.shape, 7) - 6.0)
    elif scale == "blocks":
        C[:, :, :, 0, 1, :] *= 1e-14
        C[:, :, :, 1, 0, :] = 0.0
    elif scale in ("huge", "tiny"):
        C *= 1e300 if scale == "huge" else 1e-300
    elif scale == "zero":
        C[::2] = 0.0
    ref = R.int_grad_n_dot_tensor4_dot_grad_nt_dv(dNx, vol, C)
    err = np.abs(to_np(quad.Int_gradN_dot_tensor4_dot_gradNT_dV(C)) - ref)
    assert np.all(err <= 64 * 2.0 ** -53 * _stiffness_bound(dNx, vol, C))


@pytest.mark.parametrize("nd", [2, 3])
def test_stiffness_not_finite(gf, oracle, nd):
    """An infinite and a NaN tensor entry reach the entries that they take part in, and no others."""
    R = oracle
    x = _elements(21, nd, 8)
    quad = (gf.Element.Quad4 if nd == 2 else gf.Element.Hex8).Quadrature(x)
    dNx, vol = R.compute_dN(x, *(R.quad4_gauss() if nd == 2 else R.hex8_gauss()))
    C = seeded_field(vol.shape + (nd,) * 4, 9)
    C[3, 1, 0, 1, 0, 1] = np.inf
    C[17, 2, 1, 0, 0, 0] = np.nan
    ref = R.int_grad_n_dot_tensor4_dot_grad_nt_dv(dNx, vol, C)
    got = to_np(quad.Int_gradN_dot_tensor4_dot_gradNT_dV(C))
    assert np.array_equal(np.isfinite(got), np.isfinite(ref)) and not np.isfinite(ref).all()
    ok = np.isfinite(ref)
    assert rel_err(got[ok], ref[ok]) <= RTOL
