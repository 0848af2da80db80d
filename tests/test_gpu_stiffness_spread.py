"""The stiffness integral of rules with as many points as nodes where values of very different scale meet,
against the CPU oracle: integration points of different scale, sheared, thin and nearly collapsed elements,
the nodal rule (whose gradients hold zeros).

The oracle takes the gradients and volumes of the quadrature itself: those of a degenerate element depend
on the order of its determinant. Tolerance: 64 roundings of 2^-53 of the sum of the magnitudes of an entry's terms, as many as the oracle's
own sum of 64 to 72 terms may take."""

import numpy as np
import pytest

from _common import seeded_field, to_np

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gf():
    import goosefem_gb300 as gf

    gf.set_strict(False)
    return gf


def _elements(nelem, nd, seed):
    s = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], dtype=np.float64)
    if nd == 3:
        s = np.concatenate([np.c_[s, np.zeros(4)], np.c_[s, np.ones(4)]])
    return s[None] + seeded_field((nelem,) + s.shape, seed, amp=0.15)


def _bound(dNx, vol, C):
    a, nd = np.abs, dNx.shape[3]
    t = np.einsum("eqmi,eqijkl->eqmjkl", a(dNx), a(C[:, :, :nd, :nd, :nd, :nd]) * a(vol)[..., None, None, None, None])
    k = dNx.shape[2] * nd
    return np.einsum("eqmjkl,eqnl->emjnk", t, a(dNx)).reshape(-1, k, k)


def _check(gf, R, x, rule, C, planar=False):
    nd = x.shape[2]
    cls = gf.Element.Hex8 if nd == 3 else gf.Element.Quad4
    quad = (cls.QuadraturePlanar if planar else cls.Quadrature)(x, *rule)
    dNx, vol = to_np(quad.GradN()), to_np(quad.dV())
    ref = (R.int_grad_n_dot_tensor4_dot_grad_nt_dv_planar if planar
           else R.int_grad_n_dot_tensor4_dot_grad_nt_dv)(dNx, vol, C)
    err = np.abs(to_np(quad.Int_gradN_dot_tensor4_dot_gradNT_dV(C)) - ref)
    assert np.all(err <= 64 * 2.0 ** -53 * _bound(dNx, vol, C))


@pytest.mark.parametrize("nd,planar", [(2, False), (2, True), (3, False)])
@pytest.mark.parametrize("p", [3, 6, 12, 15, 40])
def test_points_of_different_scale(gf, oracle, nd, planar, p):
    """The tensor 10^p at a point with a weight of 10^-p: the point counts as much as the others."""
    nip = 2 ** nd
    rng = np.random.default_rng(p)
    xi, w = rng.uniform(-0.8, 0.8, (nip, nd)), rng.uniform(0.5, 1.5, nip)
    x = _elements(37, nd, 1)
    C = seeded_field((37, nip) + (3 if planar else nd,) * 4, 2)
    for q in range(nip // 2):
        w[2 * q] *= 10.0 ** -p
        C[:, 2 * q] *= 10.0 ** p
    _check(gf, oracle, x, (xi, w), C, planar)


@pytest.mark.parametrize("nd", [2, 3])
@pytest.mark.parametrize("rule", ["gauss", "nodal"])
@pytest.mark.parametrize("shape", ["plain", "sheared", "thin", "collapsed"])
@pytest.mark.parametrize("tensor", ["full", "isotropic"])
def test_shapes(gf, oracle, nd, rule, shape, tensor):
    R = oracle
    x = _elements(61, nd, 3)
    if shape == "sheared":
        x[..., 0] += 1e3 * x[..., 1]
    elif shape == "thin":
        x[..., 0] *= 1e-6
    elif shape == "collapsed":  # two nodes of an edge 2^-20 to 2^-40 apart
        x[:, 1] = x[:, 0] + (x[:, 1] - x[:, 0]) * 2.0 ** -np.linspace(20, 40, 61)[:, None]
    name = ("quad4" if nd == 2 else "hex8") + "_" + rule
    xi, w = getattr(R, name)()
    eye = np.eye(nd)
    C = seeded_field((61, 2 ** nd) + (nd,) * 4, 4)
    if tensor == "isotropic":
        iso = 1.7 * np.einsum("ij,kl->ijkl", eye, eye) + np.einsum("ik,jl->ijkl", eye, eye) + \
            np.einsum("il,jk->ijkl", eye, eye)
        C = np.broadcast_to(iso, C.shape).copy()
    _check(gf, R, x, (xi, w), C)
