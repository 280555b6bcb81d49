"""The FP32 cache's tensor-core inference (three-way BF16 splits) and its training step against the FP64 oracle, at the edges of
their tiles and dispatch: one row, a row short of and past a 128-row tile, a second tile on an SM (the
grid is one CTA of two tiles per SM), 1 to 8 hidden layers, 1 to 16 outputs (4 and 16 wide variants), the
workload's frequency table and another one.

Tolerance: a layer's piece products are exact down to 2^-24 of the product and its accumulations cut at
most 2^-23 of a partial sum, ~6 times; with |w||h| summing to at most ~8 times a layer's result, a
layer adds < 8 * 8 * 2^-23 ~ 8e-6 of the output scale in the worst case and ~1e-6 in the mean. 2e-5
of the output's (gradient's) scale, in the maximum (norm), holds 8 layers with room; BF16 without the
split is off by 1e-2."""
import numpy as np
import pytest

import oracle.nrc as onrc

pytestmark = pytest.mark.gpu

FREQS = (4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2)
OTHER = (5, 1, 3, 0, 6, 2)
TOL = 2e-5


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def _net(sty, freqs, out, layers, batch=1024):
    return sty.nrc.NRC(sty.nrc.config(freqs, out, batch, layers, sty.nrc.STY_NRC_FP32, seed=17))


@pytest.mark.parametrize("rows,layers,out,freqs", [
    (1, 5, 3, FREQS), (127, 1, 1, FREQS), (129, 2, 4, OTHER), (128 * 152 + 1, 5, 3, FREQS), (128 * 304 + 77, 3, 5, OTHER),
    (300, 8, 16, FREQS), (513, 7, 3, FREQS),
])
def test_inference_matches_oracle(sty, cuda, rows, layers, out, freqs):
    net = _net(sty, freqs, out, layers)
    x = np.random.default_rng(rows).random((rows, len(freqs))).astype(np.float32)
    p = net.save_params().astype(np.float64)
    got = net.inference(_dev(x)).cpu().numpy()
    ref, _ = onrc.forward(p, x.astype(np.float64), freqs, layers, out)
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    assert (net.inference(_dev(x), ema=False).cpu().numpy() == got).all()
    q = (p * 0.7).astype(np.float32)  # loaded weights reach the operand images
    net.load_params(q)
    ref, _ = onrc.forward(q.astype(np.float64), x.astype(np.float64), freqs, layers, out)
    assert np.abs(net.inference(_dev(x)).cpu().numpy() - ref).max() <= TOL * np.abs(ref).max()
    assert sty.abi.device_status() == 0


@pytest.mark.parametrize("rows,layers,out,freqs", [
    (1, 5, 3, FREQS), (200, 1, 2, OTHER), (64 * 304 + 1, 2, 3, FREQS), (128 * 304 + 65, 2, 3, FREQS), (1000, 6, 16, FREQS),
    (777, 8, 5, FREQS),
])
def test_gradient_matches_oracle(sty, cuda, rows, layers, out, freqs):
    """The CUDA-core training kernels at 64- and 128-sample tiles (the wider ones past two tiles per SM, where
    the weights leave room), 32-row groups and quadrants of the weight gradient cut short."""
    net = _net(sty, freqs, out, layers)
    rng = np.random.default_rng(rows)
    x, t = rng.random((rows, len(freqs))).astype(np.float32), (rng.random((rows, out)) + 0.1).astype(np.float32)
    g, loss = net.gradient(_dev(x), _dev(t))
    rl, rg = onrc.loss_and_grad(net.save_params().astype(np.float64), x.astype(np.float64), t.astype(np.float64), freqs,
                                layers, out)
    assert np.linalg.norm(g.cpu().numpy() - rg) <= TOL * np.linalg.norm(rg)
    assert abs(loss - rl) <= TOL * abs(rl)
    assert sty.abi.device_status() == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_sampled_batch_is_the_gathered_one(sty, cuda, precision):
    """A training step on rows the kernel gathers itself gives the weights of a step on the one row there is to
    draw, repeated: count = 1, so every sample is that row (the first optimiser step is lr * sign)."""
    import torch
    x, t = _dev(np.random.default_rng(1).random((1, 11))), _dev([[0.3, 0.5, 0.9]])
    nets = [sty.nrc.NRC(sty.nrc.config(FREQS, 3, 256, 3, precision, seed=4)) for _ in range(2)]
    nets[0].train(x, t, 1)
    nets[1].train(x.expand(256, 11).contiguous(), t.expand(256, 3).contiguous(), 1)
    assert (nets[0].save_params() == nets[1].save_params()).all()
    torch.cuda.synchronize()
    assert sty.abi.device_status() == 0


def test_training_keeps_the_operand_images_current(sty, cuda):
    """After optimiser steps inference reads the new weights: the training weights exactly as a network
    loaded with them, and a BF16 network of 7 layers (which trains in FP32) still reduces its loss."""
    rng = np.random.default_rng(3)
    x, t = _dev(rng.random((4000, 11))), _dev(rng.random((4000, 3)) + 0.1)
    net = _net(sty, FREQS, 3, 4)
    net.train(x, t, 3)
    other = _net(sty, FREQS, 3, 4)
    other.load_params(net.save_params())
    assert (net.inference(x, ema=False) == other.inference(x, ema=False)).all()
    deep = sty.nrc.NRC(sty.nrc.config(FREQS, 3, 1024, 7, sty.nrc.STY_NRC_BF16, learning_rate=3e-3, seed=2))
    first = deep.train(x, t, 1)
    for _ in range(4):
        last = deep.train(x, t, 25)
    assert last < 0.7 * first
