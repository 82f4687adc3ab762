"""The native training step (cl_b200_mlp_train_step) against the pass-by-pass one on the same network and batch.

Both take the same products with the same roundings to BF16; only the order of the FP32 sums over the rows differs, in
the weight gradients and the bias gradients. So a gradient may differ by the rounding of a sum of B terms in another
order: 8 sqrt(B) 2^-24 of the sum of the terms' magnitudes (a random walk of B roundings, eight deviations).
"""
from __future__ import annotations

import numpy as np
import pytest

from chaos_b200.mlp import MLP

pytestmark = pytest.mark.gpu


def _net(torch, dev):
    net = MLP(torch, dev, seed=3)
    g = torch.Generator(device=dev).manual_seed(5)
    for lay in net.layers:
        lay["b"].copy_(0.1 * torch.randn(lay["b"].shape, generator=g, device=dev))
        for p in ("W", "b"):
            m = 1e-3 * torch.randn(lay[p].shape, generator=g, device=dev)
            lay["m" + p].copy_(m)
            lay["v" + p].copy_(m * m + 1e-6)
    net.step = 100
    return net


# one tile; the pipeline's batch; row ranges that do not divide evenly; the wide tiles' rule (148 tiles of rows)
@pytest.mark.parametrize("rows", [128, 1152, 4096, 6784, 18816, 18944])
def test_step_equals_the_passes(rows):
    import torch
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(rows)
    X = torch.tensor(rng.standard_normal((rows, 64)).astype(np.float32), device=dev).to(torch.bfloat16)
    label = torch.tensor((rng.random(rows) < 0.5).astype(np.float32), device=dev)
    target = torch.tensor(rng.standard_normal(rows).astype(np.float32), device=dev)
    a, b = _net(torch, dev), _net(torch, dev)
    loss = a.train_step(X, label, target, w_reg=0.7, lr=2e-3)
    out = b.forward(X, keep=True)
    loss_b, g32, gb = b.loss_and_grad(out, label, target, 0.7)
    b.backward(g32, gb)
    assert torch.equal(loss, loss_b)
    # magnitudes of the sums: |dZ|^T |A| per layer, from the passes' own BF16 operands
    dZ, slack = gb, 8 * rows ** 0.5 * 2.0 ** -24
    for li in range(3, -1, -1):
        lay, lb = a.layers[li], b.layers[li]
        A = b._acts[li]
        scale = dZ.double().abs().T @ A.double().abs()
        assert bool(((lay["gW"].double() - lb["gW"].double()).abs() <= slack * scale + 1e-30).all()), f"gW[{li}]"
        colscale = dZ.double().abs().sum(0)
        assert bool(((lay["gb"].double() - lb["gb"].double()).abs() <= slack * colscale * 1.01 + 1e-30).all()), f"gb[{li}]"
        if li:
            dA = dZ.double() @ lb["Wb"].double()
            pre = b._pres[li - 1].double().requires_grad_()
            torch.nn.functional.gelu(pre, approximate="tanh").backward(dA)
            dZ = pre.grad.to(torch.bfloat16)
    # Adam and the copies the next step reads: the pass-by-pass kernel on the step's own gradients, bit for bit
    for lay, lb in zip(a.layers, b.layers):
        lb["gW"].copy_(lay["gW"])
        lb["gb"].copy_(lay["gb"])
    b.adam(lr=2e-3)
    for lay, lb in zip(a.layers, b.layers):
        for key in ("W", "b", "mW", "vW", "mb", "vb", "Wb", "Wbt"):
            assert torch.equal(lay[key], lb[key]), key
    assert a.step == b.step == 101


class _Own(MLP):
    def adam(self, lr=1e-3, b1=0.9, b2=0.999, eps=1e-8):
        super().adam(lr=0.0, b1=b1, b2=b2, eps=eps)


# what the native step does not take runs pass by pass, with those passes' result
@pytest.mark.parametrize("form", ["wide", "ragged", "bias off 16 bytes", "subclass"])
def test_other_calls_take_the_passes(form):
    import torch
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(11)
    rows, cols = 200 if form == "ragged" else 256, 72 if form == "wide" else 64
    X = torch.tensor(rng.standard_normal((rows, cols)).astype(np.float32), device=dev).to(torch.bfloat16)
    label = torch.tensor((rng.random(rows) < 0.5).astype(np.float32), device=dev)
    target = torch.tensor(rng.standard_normal(rows).astype(np.float32), device=dev)
    a, b = _net(torch, dev), _net(torch, dev)
    if form == "subclass":
        a.__class__ = b.__class__ = _Own
    if form == "bias off 16 bytes":
        for n in (a, b):
            n.layers[1]["b"] = torch.cat([n.layers[1]["b"][:1], n.layers[1]["b"]])[1:]
    loss = a.train_step(X, label, target, w_reg=0.7, lr=2e-3)
    out = b.forward(X, keep=True)
    loss_b, g32, gb = b.loss_and_grad(out, label, target, 0.7)
    b.backward(g32, gb)
    b.adam(lr=2e-3)
    assert torch.equal(loss, loss_b) and a.step == b.step == 101
    for lay, lb in zip(a.layers, b.layers):
        for key in ("W", "b", "mW", "vW", "mb", "vb", "Wb", "Wbt"):   # one partial sum at these sizes: bit for bit
            assert torch.equal(lay[key], lb[key]), key
