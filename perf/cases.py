"""Performance cases of the framework: what its users run, from the smallest call to the largest.

Families (the field ``kind`` of a case):

* ``chain``: the internal force of a displacement through the operators of the GooseFEM API, one call
  at a time (AsElement, SymGradN_vector, elastic_stress, Int_gradN_dot_tensor2_dV, AssembleNode): the
  loop of a user's own material model or time integrator;
* ``stiffness``: the element stiffness of a tangent tensor, its assembly into the partitioned sparse
  matrix and one product with it: a Newton step's set-up;
* ``explicit``: velocity-Verlet increments of one mesh (VelocityVerlet);
* ``batch``: velocity-Verlet increments of many periodic meshes in one schedule (BatchedVerlet);
* ``static``: the matrix-free static solve with prescribed displacements (ElasticStatic);
* ``learned``: the two-level static solve with the network as its post-smoother;
* ``train``: one gradient step of that network (crops, forward, loss, backward).

``exact`` restates each of them in plain torch FP64.
"""

import math

import numpy as np
import torch

import goosefem_gb300 as gf
from goosefem_gb300 import _lib, batch, learned

DEV = "cuda"
F64 = torch.float64
G0 = 1.0 / math.sqrt(3.0)
SIGN2 = np.array([[-1, -1], [1, -1], [1, 1], [-1, 1]], dtype=np.float64)
SIGN3 = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                  [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.float64)


# ---------------------------------------------------------------------------------- the cases

def listed():
    return [
        # a unit test or a tutorial mesh: launches and host time count
        dict(name="chain_quad4_small", kind="chain", elem="quad4", nx=33, ny=29, nz=0),
        # a million distorted elements: the operators' throughput in 2-d
        dict(name="chain_quad4_large", kind="chain", elem="quad4", nx=1031, ny=997, nz=0),
        # the same in 3-d, where an element carries 8 nodes and 8 integration points
        dict(name="chain_hex8", kind="chain", elem="hex8", nx=61, ny=53, nz=47),
        # tangent assembly of a 2-d and of a 3-d mesh
        dict(name="stiffness_quad4", kind="stiffness", elem="quad4", nx=257, ny=191, nz=0),
        dict(name="stiffness_hex8", kind="stiffness", elem="hex8", nx=23, ny=21, nz=19),
        # a small wave-propagation mesh with the default arithmetic: two launches per increment
        dict(name="explicit_small", kind="explicit", elem="quad4", nx=48, ny=40, nz=0, distort=False,
             arithmetic="fp64", nsteps=20),
        # the headline workload: a Regular mesh of 2048^2 squares in float-float arithmetic
        dict(name="explicit_regular_large", kind="explicit", elem="quad4", nx=2048, ny=2048, nz=0,
             distort=False, arithmetic="pair", nsteps=20),
        # a distorted mesh with the default arithmetic
        dict(name="explicit_distorted", kind="explicit", elem="quad4", nx=509, ny=491, nz=0,
             distort=True, arithmetic="fp64", nsteps=10),
        # a parameter study: many periodic meshes of uneven sizes, one schedule for all
        dict(name="batch_uneven", kind="batch", n=24, nmin=32, nmax=256, nsteps=50),
        # a 3-d static solve, matrix-free, pair stiffness action
        dict(name="static_hex8", kind="static", elem="hex8", nx=64, ny=64, nz=64, arithmetic="pair"),
        # the two-level solve with the network on a two-phase material
        dict(name="learned_solve", kind="learned", nx=193, ny=161, hc=12),
        # the network's training step at the batch and crop of the learned workload
        dict(name="train_step", kind="train", B=32, S=96, margin=8, loss="energy"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "chain", "stiffness", "explicit", "explicit", "batch", "static", "learned",
                       "train"])
    elem = rng.choice(["quad4", "hex8"])
    if kind == "chain":
        if elem == "quad4":
            return dict(kind=kind, elem=elem, nx=_logint(rng, 8, 1000), ny=_logint(rng, 8, 1000), nz=0)
        return dict(kind=kind, elem=elem, nx=_logint(rng, 3, 56), ny=_logint(rng, 3, 56), nz=_logint(rng, 3, 48))
    if kind == "stiffness":
        if elem == "quad4":
            return dict(kind=kind, elem=elem, nx=_logint(rng, 8, 240), ny=_logint(rng, 8, 200), nz=0)
        return dict(kind=kind, elem=elem, nx=_logint(rng, 2, 22), ny=_logint(rng, 2, 22), nz=_logint(rng, 2, 19))
    if kind == "explicit":
        ar = rng.choice(["fp64", "pair"])
        distort = rng.random() < 0.5
        nsteps = rng.randint(1, 20)
        if ar == "fp64" and elem == "hex8":
            return dict(kind=kind, elem=elem, nx=_logint(rng, 3, 48), ny=_logint(rng, 3, 48), nz=_logint(rng, 3, 40),
                        distort=distort, arithmetic=ar, nsteps=nsteps)
        return dict(kind=kind, elem="quad4", nx=_logint(rng, 8, 800), ny=_logint(rng, 8, 800), nz=0,
                    distort=distort, arithmetic=ar, nsteps=nsteps)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(2, 24), nmin=rng.randint(8, 32), nmax=rng.randint(48, 256),
                    nsteps=rng.randint(5, 50))
    if kind == "static":
        n = _logint(rng, 8, 48)
        ar = rng.choice(["pair", "fp64"])
        if elem == "hex8":
            return dict(kind=kind, elem=elem, nx=n + rng.randint(0, 5), ny=n + rng.randint(0, 5), nz=n, arithmetic=ar)
        return dict(kind=kind, elem=elem, nx=2 * n + rng.randint(0, 9), ny=2 * n + rng.randint(0, 9), nz=0, arithmetic=ar)
    if kind == "learned":
        return dict(kind=kind, nx=_logint(rng, 49, 190), ny=_logint(rng, 49, 160), hc=rng.choice([12, 16]))
    return dict(kind=kind, B=rng.randint(2, 32), S=rng.randint(33, 96), margin=8, loss=rng.choice(["energy", "mse"]))


# ---------------------------------------------------------------------------------- inputs

def _dims(case):
    return (case["nx"], case["ny"]) if case["elem"] == "quad4" else (case["nx"], case["ny"], case["nz"])


def _mesh(case):
    if case["elem"] == "quad4":
        return gf.Mesh.Quad4.Regular(case["nx"], case["ny"])
    return gf.Mesh.Hex8.Regular(case["nx"], case["ny"], case["nz"])


def _grid(dims):
    """(coordinates, connectivity) of a Regular mesh of unit elements: nodes x fastest, then y, then z."""
    n = [np.arange(d + 1) for d in dims]
    if len(dims) == 2:
        y, x = np.meshgrid(n[1], n[0], indexing="ij")
        num = np.arange(x.size).reshape(x.shape)
        a = num[:-1, :-1].ravel()
        w = dims[0] + 1
        conn = np.stack([a, a + 1, a + w + 1, a + w], 1)
        return np.stack([x.ravel(), y.ravel()], 1).astype(np.float64), conn
    z, y, x = np.meshgrid(n[2], n[1], n[0], indexing="ij")
    num = np.arange(x.size).reshape(x.shape)
    a = num[:-1, :-1, :-1].ravel()
    w = dims[0] + 1
    p = w * (dims[1] + 1)
    conn = np.stack([a, a + 1, a + w + 1, a + w, a + p, a + p + 1, a + p + w + 1, a + p + w], 1)
    return np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.float64), conn


def _moved(coor, dims, rng):
    """Interior nodes moved by up to 0.15 of an element."""
    move = rng.uniform(-0.15, 0.15, coor.shape)
    inner = np.all((coor > 0) & (coor < np.asarray(dims)), axis=1)
    return coor + move * inner[:, None]


def _moduli(n, rng):
    return rng.uniform(0.5, 1.5, n), rng.uniform(0.25, 0.75, n)


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV)


def _chain_inputs(case, seed):
    rng = np.random.default_rng(seed)
    dims = _dims(case)
    coor, conn = _grid(dims)
    coor = _moved(coor, dims, rng)
    K, G = _moduli(conn.shape[0], rng)
    u = 1e-2 * coor @ rng.uniform(-1, 1, (len(dims), len(dims))) + rng.uniform(-1e-3, 1e-3, coor.shape)
    return coor, conn, K, G, u


def _stiff_inputs(case, seed):
    """Mesh, prescribed dofs (the first row or plane of nodes), the tangent tensor per integration point
    (isotropic, less a rank-one softening as a plastic tangent has) and a vector."""
    rng = np.random.default_rng(seed)
    dims = _dims(case)
    coor, conn = _grid(dims)
    coor = _moved(coor, dims, rng)
    K, G = _moduli(conn.shape[0], rng)
    nd = len(dims)
    nip = 2 ** nd
    first = np.flatnonzero(coor[:, nd - 1] == 0)
    iip = (first[:, None] * nd + np.arange(nd)).ravel()
    a = rng.uniform(-1, 1, (conn.shape[0], nip, nd, nd))
    a = _dev(a + a.swapaxes(2, 3)) * 0.5
    x = rng.uniform(-1e-2, 1e-2, coor.size)
    eye = torch.eye(nd, dtype=F64, device=DEV)
    K, G = _dev(K)[:, None, None, None, None, None], _dev(G)[:, None, None, None, None, None]
    ii = torch.einsum("ij,kl->ijkl", eye, eye)
    sy = torch.einsum("ik,jl->ijkl", eye, eye) + torch.einsum("il,jk->ijkl", eye, eye)
    C = (K - 2.0 * G / 3.0) * ii + G * (sy - 0.2 * torch.einsum("eqij,eqkl->eqijkl", a, a))
    return coor, conn, iip, C.contiguous(), x


def _explicit_inputs(case, seed):
    rng = np.random.default_rng(seed)
    dims = _dims(case)
    coor, conn = _grid(dims)
    if case["distort"]:
        coor = _moved(coor, dims, rng)
    K, G = _moduli(conn.shape[0], rng)
    fixed = np.flatnonzero(coor[:, len(dims) - 1] == 0)
    v = rng.uniform(-1e-3, 1e-3, coor.shape)
    v[fixed] = 0.0
    fext = rng.uniform(-1e-4, 1e-4, coor.shape)
    iip = (fixed[:, None] * len(dims) + np.arange(len(dims))).ravel()
    dt = 0.1 / math.sqrt(float(np.max(K + 4.0 * G / 3.0)))
    return coor, conn, K, G, iip, v, fext, dt


def _static_inputs(case, seed):
    """The first plane (3-d) or row (2-d) fixed, the last one pressed in along its normal."""
    rng = np.random.default_rng(seed)
    dims = _dims(case)
    coor, conn = _grid(dims)
    K, G = _moduli(conn.shape[0], rng)
    nd = len(dims)
    lo, hi = np.flatnonzero(coor[:, nd - 1] == 0), np.flatnonzero(coor[:, nd - 1] == dims[-1])
    x = np.zeros(coor.shape)
    x[hi, nd - 1] = -1e-2 * rng.uniform(0.9, 1.1, hi.size)
    iip = np.unique(np.concatenate([(lo[:, None] * nd + np.arange(nd)).ravel(), hi * nd + nd - 1]))
    return coor, conn, K, G, iip, x


def _batch_inputs(case, seed):
    """(nx, ny, K, G) of each instance; the sizes belong to the case, the moduli to the seed."""
    sizes = np.random.default_rng([case["n"], case["nmin"], case["nmax"]])
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["n"]):
        nx, ny = (int(k) for k in sizes.integers(case["nmin"], case["nmax"] + 1, 2))
        out.append((nx, ny) + _moduli(nx * ny, rng))
    return out


def _two_phase(nx, ny, seed):
    """Stiff circular inclusions in a soft matrix, 15 % of the area, ten times the moduli."""
    rng = np.random.default_rng(seed)
    cy, cx = np.meshgrid(np.arange(ny) + 0.5, np.arange(nx) + 0.5, indexing="ij")
    inside = np.zeros((ny, nx), dtype=bool)
    while inside.mean() < 0.15:
        r = rng.uniform(4.0, 12.0)
        inside |= (cx - rng.uniform(0, nx)) ** 2 + (cy - rng.uniform(0, ny)) ** 2 <= r * r
    f = np.where(inside, 10.0, 1.0).ravel()
    return f, 0.5 * f


def _learned_inputs(case, seed):
    nx, ny = case["nx"], case["ny"]
    K, G = _two_phase(nx, ny, seed)
    coor, conn = _grid((nx, ny))
    bot, top = np.arange(nx + 1), np.arange(nx + 1) + ny * (nx + 1)
    iip = np.unique(np.concatenate([(bot[:, None] * 2 + np.arange(2)).ravel(), top * 2 + 1]))
    x = np.zeros(coor.size)
    x[top * 2 + 1] = -1e-2
    return coor, conn, K, G, iip, x


_LAYERS = ((4, 32), (32, 32), (32, 32), (32, 2))


def _train_inputs(case, seed):
    """Parameters (He), a few stored pairs on a grid, its moduli and free dofs, and crop positions."""
    rng = np.random.default_rng(seed)
    H = W = 129
    npairs = 8
    par = []
    for layer, (ci, co) in enumerate(_LAYERS):
        std = math.sqrt(2.0 / (9 * ci)) * (0.1 if layer == 3 else 1.0)
        par += [rng.normal(0.0, std, 9 * ci * co), rng.normal(0.0, 0.01, co)]
    par = np.concatenate(par).astype(np.float32)
    R = rng.normal(0.0, 1.0, (npairs, H, W, 2)).astype(np.float32)
    T = (0.25 * (R + np.roll(R, 1, 1) + np.roll(R, 1, 2) + np.roll(R, (1, 1), (1, 2)))).astype(np.float32)
    E = rng.uniform(0.1, 1.0, (H - 1, W - 1, 2)).astype(np.float32)
    mat = rng.uniform(0.1, 1.0, (H, W, 2)).astype(np.float32)
    free = np.ones((H, W, 2), dtype=np.float32)
    free[0] = 0.0
    free[-1, :, 1] = 0.0
    m, S = case["margin"], case["S"]
    pos = np.stack([rng.integers(0, npairs, case["B"]), rng.integers(-m, H - S + m + 1, case["B"]),
                    rng.integers(-m, W - S + m + 1, case["B"])], 1).astype(np.int32)
    return dict(par=par, R=R, T=T, E=E, mat=mat, free=free, pos=pos, H=H, W=W)


# ---------------------------------------------------------------------------------- prepare and run

def prepare(case, seed):
    kind = case["kind"]
    if kind == "chain":
        coor, conn, K, G, u = _chain_inputs(case, seed)
        vector = gf.Vector(conn, _mesh(case).dofs())
        E = gf.Element.Quad4 if case["elem"] == "quad4" else gf.Element.Hex8
        return dict(kind=kind, vector=vector, quad=E.Quadrature(vector.AsElement(coor)), K=_dev(K), G=_dev(G),
                    u=_dev(u))
    if kind == "stiffness":
        coor, conn, iip, C, x = _stiff_inputs(case, seed)
        dofs = _mesh(case).dofs()
        vector = gf.Vector(conn, dofs)
        E = gf.Element.Quad4 if case["elem"] == "quad4" else gf.Element.Hex8
        return dict(kind=kind, quad=E.Quadrature(vector.AsElement(coor)), A=gf.MatrixPartitioned(conn, dofs, iip),
                    C=C, x=_dev(x))
    if kind == "explicit":
        coor, conn, K, G, iip, v, fext, dt = _explicit_inputs(case, seed)
        vv = gf.VelocityVerlet(coor, conn, _mesh(case).dofs(), K, G, dt=dt, eta=0.1, iip=iip, fext=fext,
                               arithmetic=case["arithmetic"])
        v = _dev(v)
        return dict(kind=kind, vv=vv, u=torch.zeros_like(v), v=v, a=torch.zeros_like(v), nsteps=case["nsteps"])
    if kind == "batch":
        # the schedule that BatchedVerlet.autotune picks for such instances
        bv = batch.BatchedVerlet([batch.Instance(nx, ny, K, G, 2e-3) for nx, ny, K, G in _batch_inputs(case, seed)],
                                 eta=0.1)
        bv.mode = 3
        u, v, a = bv.state()
        return dict(kind=kind, bv=bv, u=u, v=v, a=a, nsteps=case["nsteps"])
    if kind == "static":
        coor, conn, K, G, iip, x = _static_inputs(case, seed)
        st = gf.ElasticStatic(coor, conn, _mesh(case).dofs(), K, G, iip, arithmetic=case["arithmetic"])
        x0 = _dev(x)
        return dict(kind=kind, st=st, x0=x0, x=torch.empty_like(x0))
    if kind == "learned":
        coor, conn, K, G, iip, x = _learned_inputs(case, seed)
        lp = learned.LearnedPreconditioner(case["nx"], case["ny"], K, G, iip, seed=seed % 1000, arithmetic="pair")
        lp.coarse_setup(case["hc"])
        x0 = _dev(x)
        return dict(kind=kind, lp=lp, x0=x0, x=torch.empty_like(x0))
    t = _train_inputs(case, seed)
    B, S = case["B"], case["S"]
    f32 = dict(dtype=torch.float32, device=DEV)
    s = {k: _dev(t[k]) for k in ("par", "R", "T", "E", "mat", "free", "pos")}
    nb = int(_lib.lib().gfgpu_nn_train_workspace_bytes(B, S, S))
    energy = case["loss"] == "energy"
    s.update(kind="train", B=B, S=S, margin=case["margin"], H=t["H"], W=t["W"], wbf=s["par"].to(torch.bfloat16),
             X=torch.empty((B, S, S, 4), **f32), Tc=torch.empty((B, S, S, 2), **f32),
             Ec=torch.empty((B, S - 1, S - 1, 2), **f32) if energy else None,
             Fc=torch.empty((B, S, S, 2), **f32) if energy else None,
             grads=torch.empty_like(s["par"]), loss=torch.empty(1, **f32), ws=torch.empty(nb // 4 + 64, **f32))
    return s


def _ptr(t):
    return None if t is None else t.data_ptr()


def run(s):
    kind = s["kind"]
    if kind == "chain":
        ue = s["vector"].AsElement(s["u"])
        eps = s["quad"].SymGradN_vector(ue)
        sig = gf.elastic_stress(eps, s["K"], s["G"])
        fe = s["quad"].Int_gradN_dot_tensor2_dV(sig)
        return dict(eps=eps, sig=sig, fe=fe, f=s["vector"].AssembleNode(fe))
    if kind == "stiffness":
        Ke = s["quad"].Int_gradN_dot_tensor4_dot_gradNT_dV(s["C"])
        s["A"].assemble(Ke)
        return dict(Ke=Ke, val=s["A"].data()[2], b=s["A"].Dot(s["x"]))
    if kind == "explicit":
        s["vv"].step(s["u"], s["v"], s["a"], s["nsteps"])
        return dict(u=s["u"], v=s["v"], a=s["a"])
    if kind == "batch":
        s["bv"].run_graph(s["u"], s["v"], s["a"], s["nsteps"])
        return dict(u=s["u"], v=s["v"], a=s["a"])
    if kind == "static":
        s["x"].copy_(s["x0"])
        s["st"].solve(s["x"], tol=1e-12)  # in the place of a direct solver: its accuracy
        return s["x"]
    if kind == "learned":
        s["x"].copy_(s["x0"])
        s["lp"].solve(s["x"], tol=1e-11)
        return s["x"]
    st = torch.cuda.current_stream().cuda_stream
    _lib.call("gfgpu_nn_gather_crops", _ptr(s["R"]), _ptr(s["T"]), _ptr(s["mat"]), _ptr(s["E"]), _ptr(s["free"]),
              _ptr(s["pos"]), s["B"], s["S"], s["H"], s["W"], _ptr(s["X"]), _ptr(s["Tc"]), _ptr(s["Ec"]),
              _ptr(s["Fc"]), st)
    _lib.call("gfgpu_nn_train_step", _ptr(s["wbf"]), _ptr(s["par"]), _ptr(s["X"]), _ptr(s["Tc"]), _ptr(s["Ec"]),
              _ptr(s["Fc"]), s["B"], s["S"], s["margin"], _ptr(s["grads"]), _ptr(s["loss"]), _ptr(s["ws"]), st)
    return dict(grads=s["grads"], loss=s["loss"])


# ---------------------------------------------------------------------------------- work

def work(case):
    """Each input read and each output written once, in FP64 (FP32 for the network); operations of the
    formulas with the common factors taken out."""
    kind = case["kind"]
    if kind == "train":
        pix = case["B"] * case["S"] ** 2
        macs = sum(9 * ci * co for ci, co in _LAYERS)
        return dict(bytes=pix * 4 * 10.0 + 3 * 81032, flops=2.0 * pix * (3 * macs - 9 * 4 * 32))
    if kind == "batch":
        m = 0.5 * (case["nmin"] + case["nmax"])
        n = case["n"] * m * m * case["nsteps"]
        return dict(bytes=n * 128.0, flops=n * 110.0)
    if kind == "learned":
        n = case["nx"] * case["ny"]
        its = 200.0
        return dict(bytes=its * n * (2 * 112.0), flops=its * n * (2 * 110.0 + 2 * 20160))
    dims = _dims(case)
    nd, nne = len(dims), 2 ** len(dims)
    nelem = float(np.prod(dims))
    nnode = float(np.prod([d + 1 for d in dims]))
    nip = nne
    if kind == "chain":
        by = nelem * (nne * 4 + 8 * (nip * (nne * nd + 1) + 2 + 2 * nip * nd * nd + nne * nd)) + 16 * nnode * nd
        fl = nelem * nip * (2 * nne * nd * nd + 12 + 2 * nne * nd * nd)
        return dict(bytes=by, flops=fl)
    if kind == "stiffness":
        k = nne * nd
        nnz = nnode * nd * nd * 3 ** nd
        by = 8 * nelem * (nip * (nd ** 4 + nne * nd + 1) + k * k) + 12 * nnz + 16 * nnode * nd
        return dict(bytes=by, flops=nelem * nip * 2 * (nd ** 4 + nne * nd ** 4 + k * k * nd) + 2 * nnz)
    per = 8 * (7 * nd * nnode + 2 * nelem)
    ops = nelem * (110 if nd == 2 else 420)
    if kind == "explicit":
        if case["distort"]:
            per += 8 * nd * nnode
            ops = nelem * nip * (4 * nne * nd * nd + 12)
        return dict(bytes=per * case["nsteps"], flops=ops * case["nsteps"])
    its = 15.0 * max(dims)
    return dict(bytes=its * per, flops=its * (ops + 12 * nd * nnode))


# ---------------------------------------------------------------------------------- exact

def _quadrature(coor, conn):
    """(dNx [e, q, m, i], vol [e, q]) with 2-point Gauss rules; in 3-d the gradient is the row sum of the
    inverse Jacobian times dN/dxi, as the reference library defines it."""
    nd = coor.shape[1]
    sg = SIGN2 if nd == 2 else SIGN3
    xi = sg * G0
    one = 1.0 + xi[:, None, :] * sg[None, :, :]  # [q, m, i]
    dn = np.empty((len(xi), len(sg), nd))
    for i in range(nd):
        dn[:, :, i] = sg[None, :, i] / 2 ** nd * np.prod(np.delete(one, i, axis=2), axis=2)
    dn = _dev(dn)
    J = torch.einsum("qmi,emj->eqij", dn, _dev(coor)[_dev(conn)])
    Ji = torch.linalg.inv(J)
    if nd == 2:
        dNx = torch.einsum("eqij,qmj->eqmi", Ji, dn)
    else:
        dNx = Ji.sum(-1)[:, :, None, :] * dn[None]
    return dNx, torch.linalg.det(J)


def _stress(eps, K, G):
    nd = eps.shape[-1]
    tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
    eye = torch.eye(nd, dtype=F64, device=DEV)
    K, G = K[:, None], G[:, None]
    return ((K - 2.0 * G / 3.0) * tr)[..., None, None] * eye + 2.0 * G[..., None, None] * eps


class _Operator:
    """Element forces and their assembly for any mesh; `group` numbers the dofs' nodes."""

    def __init__(self, coor, conn, K, G, group=None):
        self.conn = _dev(conn)
        self.K, self.G = _dev(K), _dev(G)
        self.same = bool(np.all(coor == np.round(coor)))
        if self.same:  # congruent unit elements: one stiffness per modulus
            g, v = _quadrature(coor, conn[:1])
            self.k = [self._ke(g, v, *m) for m in ((1.0, 0.0), (0.0, 1.0))]
            self.vol = v.sum() / conn.shape[1]
        else:
            self.g, self.v = _quadrature(coor, conn)
        self.n, self.nd = coor.shape
        self.group = None if group is None else _dev(group)

    def _ke(self, g, v, K, G):
        nd, nne = g.shape[3], g.shape[2]
        one = torch.ones(1, dtype=F64, device=DEV)
        B = torch.zeros((1, g.shape[1], nne * nd, nd, nd), dtype=F64, device=DEV)
        for m in range(nne):
            for j in range(nd):
                B[:, :, m * nd + j, :, j] = g[:, :, m, :]
        e = 0.5 * (B + B.transpose(-1, -2))
        s = torch.stack([_stress(e[:, :, c], K * one, G * one) for c in range(nne * nd)], 2)
        return torch.einsum("eqrij,eqcij,eq->rc", B, s, v)

    def elem(self, u):
        ue = u[self.conn]
        if self.same:
            w = ue.reshape(ue.shape[0], -1)
            f = (w @ self.k[0].T) * self.K[:, None] + (w @ self.k[1].T) * self.G[:, None]
            return f.reshape(ue.shape)
        h = torch.einsum("eqmi,emj->eqij", self.g, ue)
        s = _stress(0.5 * (h + h.transpose(-1, -2)), self.K, self.G)
        return torch.einsum("eqmi,eqij,eq->emj", self.g, s, self.v)

    def gather(self, fe):
        tgt = self.conn if self.group is None else self.group[self.conn]
        f = torch.zeros((self.n, fe.shape[2]), dtype=F64, device=DEV)
        f.index_add_(0, tgt.reshape(-1), fe.reshape(-1, fe.shape[2]))
        return f if self.group is None else f[self.group]

    def __call__(self, u):
        return self.gather(self.elem(u))

    def diagonal(self):
        """diag A: the element stiffness applied to each unit vector."""
        ne, nne, nd = self.conn.shape[0], self.conn.shape[1], self.nd
        if self.same:
            d = self.k[0].diagonal()[None] * self.K[:, None] + self.k[1].diagonal()[None] * self.G[:, None]
        else:
            n2 = (self.g ** 2).sum(-1, keepdim=True)
            lam = (self.K - 2.0 * self.G / 3.0)[:, None, None, None]
            G = self.G[:, None, None, None]
            d = (self.v[..., None, None] * ((lam + G) * self.g ** 2 + G * n2)).sum(1)
        return self.gather(d.reshape(ne, nne, nd))


def _lumped(op, coor, conn):
    """Lumped mass per node (unit density, nodal quadrature: each node the volume at its own corner)."""
    nd = coor.shape[1]
    sg = SIGN2 if nd == 2 else SIGN3
    one = 1.0 + sg[:, None, :] * sg[None, :, :]
    dn = np.empty((len(sg), len(sg), nd))
    for i in range(nd):
        dn[:, :, i] = sg[None, :, i] / 2 ** nd * np.prod(np.delete(one, i, axis=2), axis=2)
    J = torch.einsum("qmi,emj->eqij", _dev(dn), _dev(coor)[_dev(conn)])
    return op.gather(torch.linalg.det(J)[:, :, None])


def _verlet(op, mass, free, fext, dt, eta, nsteps, u, v, a):
    for _ in range(nsteps):
        u = u + dt * v + 0.5 * dt * dt * a
        R = fext - op(u)
        new = lambda vv, old: torch.where(free, (R - eta * vv) / mass, old)  # noqa: E731
        a1 = new(v + dt * a, a)
        a2 = new(v + 0.5 * dt * (a + a1), a1)
        v = v + 0.5 * dt * (a + a2)
        a = new(v, a2)
    return dict(u=u, v=v, a=a)


def _cg(op, x, iip, tol=1e-14):
    """A_uu x_u = -A_up x_p by Jacobi-preconditioned CG, restarted from the true residual."""
    free = torch.ones(x.numel(), dtype=torch.bool, device=DEV)
    free[_dev(iip).long()] = False
    free = free.reshape(x.shape)
    zero = torch.zeros((), dtype=F64, device=DEV)
    minv = torch.where(free, 1.0 / op.diagonal(), zero)
    bn = torch.where(free, op(x), zero).norm()
    for _ in range(3):
        r = torch.where(free, -op(x), zero)
        p = minv * r
        rz = (r * p).sum()
        for k in range(4000):
            q = torch.where(free, op(p), zero)
            al = rz / (p * q).sum()
            x = x + al * p
            r = r - al * q
            z = minv * r
            new = (r * z).sum()
            p = z + new / rz * p
            rz = new
            if k % 50 == 49 and float(r.norm() / bn) < tol:
                break
    return x


def _net(par, X):
    """The network's output [B, 2, S, S] for X [B, 4, S, S] (dilations 1, 2, 4, 1, zero padding)."""
    h, o = X, 0
    for k, ((ci, co), dil) in enumerate(zip(_LAYERS, (1, 2, 4, 1))):
        w = par[o:o + 9 * ci * co].reshape(3, 3, ci, co).permute(3, 2, 0, 1)
        o += 9 * ci * co
        h = torch.nn.functional.conv2d(h, w, par[o:o + co], padding=dil, dilation=dil)
        o += co
        h = h if k == 3 else torch.relu(h)
    return h


def _exact_train(case, seed):
    t = _train_inputs(case, seed)
    B, S, m, H, W = case["B"], case["S"], case["margin"], t["H"], t["W"]

    def crop(a, h, w):  # zero outside
        out = np.zeros((B, h, w, a.shape[-1]))
        for b, (n, y, x) in enumerate(t["pos"]):
            src = a[n] if a.ndim == 4 else a
            ys, xs = max(0, y), max(0, x)
            ye, xe = min(src.shape[0], y + h), min(src.shape[1], x + w)
            out[b, ys - y:ye - y, xs - x:xe - x] = src[ys:ye, xs:xe]
        return _dev(out)

    X = torch.cat([crop(t["R"], S, S), crop(t["mat"], S, S)], -1).permute(0, 3, 1, 2)
    T, E, F = crop(t["T"], S, S), crop(t["E"], S - 1, S - 1), crop(t["free"], S, S)
    par = _dev(t["par"])
    o, keep = 0, torch.zeros_like(par, dtype=torch.bool)
    for ci, co in _LAYERS:  # weights act in BF16, biases in FP32
        keep[o + 9 * ci * co:o + 9 * ci * co + co] = True
        o += 9 * ci * co + co
    par = torch.where(keep, par, par.to(torch.bfloat16).float()).double().requires_grad_()
    Y = _net(par, X).permute(0, 2, 3, 1)
    M = torch.zeros((S, S, 1), dtype=F64, device=DEV)
    M[m:S - m, m:S - m] = 1.0
    if case["loss"] == "mse":
        loss = ((M * (Y - T)) ** 2).sum() / (B * (S - 2 * m) ** 2 * 2)
    else:
        coor, conn = _grid((1, 1))
        op = _Operator(coor, conn, np.ones(1), np.ones(1))

        def energy(w):
            c = torch.cat([w[:, :-1, :-1], w[:, :-1, 1:], w[:, 1:, 1:], w[:, 1:, :-1]], -1)
            return sum((E[..., k] * ((c @ op.k[k].T) * c).sum(-1)).sum() for k in range(2))

        loss = energy(M * F * (Y - T)) / energy(M * F * T)
    loss.backward()
    return dict(grads=par.grad, loss=loss.detach().reshape(1))


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "chain":
        coor, conn, K, G, u = _chain_inputs(case, seed)
        op = _Operator(coor, conn, K, G)
        h = torch.einsum("eqmi,emj->eqij", op.g, _dev(u)[op.conn])
        eps = 0.5 * (h + h.transpose(-1, -2))
        sig = _stress(eps, op.K, op.G)
        fe = torch.einsum("eqmi,eqij,eq->emj", op.g, sig, op.v)
        return dict(eps=eps, sig=sig, fe=fe, f=op.gather(fe))
    if kind == "stiffness":
        coor, conn, iip, C, x = _stiff_inputs(case, seed)
        g, v = _quadrature(coor, conn)
        t = torch.einsum("eqmi,eqijkl,eq->eqmjkl", g, C, v)
        nd, k = coor.shape[1], conn.shape[1] * coor.shape[1]
        Ke = torch.einsum("eqmjkl,eqnl->emjnk", t, g).reshape(-1, k, k)
        n = coor.size
        dof = (_dev(conn)[:, :, None] * nd + torch.arange(nd, device=DEV)).reshape(-1, k)
        b = torch.zeros(n, dtype=F64, device=DEV)
        b.index_add_(0, dof.reshape(-1), torch.einsum("erc,ec->er", Ke, _dev(x)[dof]).reshape(-1))
        fr = np.ones(n, dtype=bool)
        fr[iip] = False
        part = np.empty(n, dtype=np.int64)
        part[np.flatnonzero(fr)] = np.arange(fr.sum())
        part[iip] = fr.sum() + np.arange(iip.size)
        pd = _dev(part)[dof]
        key = (pd[:, :, None] * n + pd[:, None, :]).reshape(-1)
        uniq, inv = torch.unique(key, return_inverse=True)
        val = torch.zeros(uniq.numel(), dtype=F64, device=DEV).index_add_(0, inv, Ke.reshape(-1))
        return dict(Ke=Ke, val=val, b=b)
    if kind == "explicit":
        coor, conn, K, G, iip, v, fext, dt = _explicit_inputs(case, seed)
        op = _Operator(coor, conn, K, G)
        free = torch.ones(coor.size, dtype=torch.bool, device=DEV)
        free[_dev(iip).long()] = False
        v = _dev(v)
        return _verlet(op, _lumped(op, coor, conn), free.reshape(coor.shape), _dev(fext), dt, 0.1, case["nsteps"],
                       torch.zeros_like(v), v, torch.zeros_like(v))
    if kind == "batch":
        inst = _batch_inputs(case, seed)
        dt = 0.1 / math.sqrt(max(float(np.max(K + 4.0 * G / 3.0)) for _, _, K, G in inst))
        parts = []
        for nx, ny, K, G in inst:
            coor, conn = _grid((nx, ny))
            ix, iy = coor[:, 0].astype(np.int64) % nx, coor[:, 1].astype(np.int64) % ny
            op = _Operator(coor, conn, K, G, group=iy * (nx + 1) + ix)
            u = np.zeros(coor.shape)
            u[:, 0] = 2e-3 * coor[:, 1]
            u = _dev(u)
            parts.append(_verlet(op, _lumped(op, coor, conn), torch.ones_like(u, dtype=torch.bool), 0.0, dt, 0.1,
                                 case["nsteps"], u, torch.zeros_like(u), torch.zeros_like(u)))
        return {k: torch.cat([p[k] for p in parts]) for k in ("u", "v", "a")}
    if kind == "static":
        coor, conn, K, G, iip, x = _static_inputs(case, seed)
        return _cg(_Operator(coor, conn, K, G), _dev(x), iip)
    coor, conn, K, G, iip, x = _learned_inputs(case, seed)
    return _cg(_Operator(coor, conn, K, G), _dev(x).reshape(coor.shape), iip).reshape(-1)
