"""The training step's tiled convolutions at the edges of their 16 x 16 pixel tiles.

Gradients and forward output against the FP64 numpy network (oracle/nn.py). Tolerance: an output is
a chain of four layers of at most 288 FP32 products and a gradient a sum over at most 3 * 33^2
pixels; rounding errors of 2^-24 that add like a random walk give about 2^-24 (4 sqrt(288) +
sqrt(3267)) = 7e-6 of the largest value; the tests ask for 4e-5.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 4e-5
LAYERS = ((4, 32), (32, 32), (32, 32), (32, 2))
DILS = (1, 2, 4, 1)


@pytest.fixture(scope="module")
def L():
    from goosefem_gb300 import _lib

    return _lib


def _net(seed):
    """(flat FP32 parameters, BF16 weights on the device, oracle parameters with BF16 weights)."""
    rng = np.random.default_rng(seed)
    flat, par = [], []
    for ci, co in LAYERS:
        W = rng.normal(0.0, np.sqrt(2.0 / (9 * ci)), (9, ci, co)).astype(np.float32)
        b = rng.normal(0.0, 0.1, co).astype(np.float32)
        flat += [W.ravel(), b]
        par.append((torch.tensor(W).to(torch.bfloat16).double().numpy(), b.astype(np.float64)))
    flat = torch.tensor(np.concatenate(flat), device="cuda")
    return flat, flat.to(torch.bfloat16), par


def _step(L, flat, wb, X, T, E, F, S, margin, shift=0):
    """One gradient step; shift: X and the workspace moved by that many floats from alignment."""
    B = X.shape[0]
    Xd = torch.empty(X.size + 8, dtype=torch.float32, device="cuda")[shift:shift + X.size]
    Xd.copy_(torch.tensor(X.ravel()))
    dev = lambda a: None if a is None else torch.tensor(a, device="cuda")  # noqa: E731
    Td, Ed, Fd = dev(T), dev(E), dev(F)
    nb = int(L.lib().gfgpu_nn_train_workspace_bytes(B, S, S))
    ws = torch.empty(nb // 4 + 8, dtype=torch.float32, device="cuda")[shift:]
    g = torch.empty_like(flat)
    loss = torch.empty(1, dtype=torch.float32, device="cuda")
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    L.call("gfgpu_nn_train_step", wb.data_ptr(), flat.data_ptr(), Xd.data_ptr(), Td.data_ptr(), p(Ed), p(Fd), B, S,
           margin, g.data_ptr(), loss.data_ptr(), ws.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return g.cpu().numpy(), float(loss.item())


@pytest.mark.parametrize("B,S,margin,energy", [(1, 3, 0, False), (2, 15, 2, True), (1, 16, 3, False),
                                               (3, 17, 4, True), (2, 31, 8, False), (3, 33, 8, True)])
def test_gradients_at_tile_edges(L, B, S, margin, energy):
    from oracle import nn as N

    flat, wb, par = _net(S)
    rng = np.random.default_rng(100 + S)
    X = rng.normal(size=(B, S, S, 4)).astype(np.float32)
    T = rng.normal(size=(B, S, S, 2)).astype(np.float32)
    E = F = None
    if energy:
        E = rng.uniform(0.2, 1.0, (B, S - 1, S - 1, 2)).astype(np.float32)
        F = (rng.uniform(size=(B, S, S, 2)) > 0.1).astype(np.float32)
    got, loss = _step(L, flat, wb, X, T, E, F, S, margin)
    if energy:
        want, grads = N.energy_loss_and_grads(*(a.astype(np.float64) for a in (X, T, E, F)), margin, par, DILS)
    else:
        mask = np.zeros((B, S, S))
        mask[:, margin:S - margin, margin:S - margin] = 1.0
        want, grads = N.loss_and_grads(X.astype(np.float64), T.astype(np.float64), mask, par, DILS)
    assert abs(loss - want) <= TOL * abs(want)
    o = 0
    for (ci, co), (dW, db) in zip(LAYERS, grads):
        for ref in (dW.ravel(), db):
            g = got[o:o + ref.size]
            o += ref.size
            assert np.max(np.abs(g - ref)) <= TOL * np.max(np.abs(ref)), (ci, co)
    # inputs and workspace off the 16-byte boundary: the same bits
    again, loss2 = _step(L, flat, wb, X, T, E, F, S, margin, shift=1)
    assert np.array_equal(got, again) and loss == loss2


@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (2, 5, 48), (1, 34, 18), (1, 17, 1)])
def test_forward_of_rectangles(L, B, H, W):
    from oracle import nn as N

    flat, wb, par = _net(7)
    X = np.random.default_rng(H * 100 + W).normal(size=(B, H, W, 4)).astype(np.float32)
    nb = int(L.lib().gfgpu_nn_train_workspace_bytes(B, H, W))
    ws = torch.empty(nb // 4 + 1, dtype=torch.float32, device="cuda")
    Y = torch.empty((B, H, W, 2), dtype=torch.float32, device="cuda")
    Xd = torch.tensor(X, device="cuda")
    L.call("gfgpu_nn_forward", wb.data_ptr(), flat.data_ptr(), Xd.data_ptr(), B, H, W, Y.data_ptr(), ws.data_ptr(),
           torch.cuda.current_stream().cuda_stream)
    ref, _ = N.forward(X.astype(np.float64), par, DILS)
    assert np.max(np.abs(Y.cpu().numpy() - ref)) <= TOL * np.max(np.abs(ref))
