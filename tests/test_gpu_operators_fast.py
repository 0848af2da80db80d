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
