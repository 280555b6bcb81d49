"""FP32 inference of networks whose weights leave the range in which the three-piece split adds up: infinities, NaNs and sums
that overflow come out as FP32 arithmetic gives them (a chain of fused multiply-adds over the 64 units, then max(., 0),
which turns a NaN into 0), and the ordinary path is taken again when the weights are back in range."""
import numpy as np
import pytest

FREQS = (4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2)
OTHER = (5, 1, 3, 0, 6, 2)


def _chain(p, x, freqs, layers, out):
    """The network in FP32, every sum over k in order (FP64 products and one rounding per step: an FMA's, but for double
    roundings that the tolerance covers)."""
    cols = []
    for d, f in enumerate(freqs):
        for k in range(f):
            a = np.pi * x[:, d].astype(np.float64) * 2.0 ** k
            cols += [np.sin(a), np.cos(a)]
    h = np.zeros((x.shape[0], 64), np.float32)
    h[:, :len(cols)] = np.stack(cols, 1)
    for l in range(layers + 1):
        w = p[l * 4096:(l + 1) * 4096].reshape(-1, 64)
        s = np.zeros((h.shape[0], w.shape[0]), np.float32)
        with np.errstate(all="ignore"):
            for k in range(64):
                s = (w[:, k].astype(np.float64) * h[:, k:k + 1].astype(np.float64) + s.astype(np.float64)).astype(np.float32)
        h = s if l == layers else np.where(s > 0, s, np.float32(0))
    return h


def _wild(p, layers, kind):
    q = p.copy()
    if kind == "inf":
        q[3 * 64 + 5], q[4096 + 7 * 64 + 9], q[layers * 4096 + 1] = np.inf, -np.inf, np.inf
    elif kind == "nan":
        q[2 * 64 + 1] = np.nan
    elif kind == "overflow":  # hidden sums of 1e38 and beyond
        q[:4096] *= 1e20
        q[4096:8192] *= 1e18
    elif kind == "near":  # finite throughout, pieces round to infinity
        q[0:64] = np.where(np.arange(64) == 1, 3.395e38, 0)
        q[4096:8192] *= 1e-30
    elif kind == "output":
        q[layers * 4096:] *= 1e38
    return q.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["inf", "nan", "overflow", "near", "output"])
@pytest.mark.parametrize("rows,layers,out,freqs", [(1, 2, 3, FREQS), (129, 2, 1, OTHER), (700, 5, 16, FREQS), (300, 8, 4, OTHER)])
def test_wide_weights(sty, cuda, rows, layers, out, freqs, kind):
    import torch
    net = sty.nrc.NRC(sty.nrc.config(freqs, out, 128, layers, sty.nrc.STY_NRC_FP32, seed=5))
    p = net.save_params()
    x = np.random.default_rng(rows).random((rows, len(freqs))).astype(np.float32)
    dx = torch.from_numpy(x).cuda()
    plain = net.inference(dx).cpu().numpy()
    q = _wild(p, layers, kind)
    net.load_params(q)
    ref = _chain(q, x, freqs, layers, out)
    for ema in (True, False):
        got = net.inference(dx, ema=ema).cpu().numpy()
        assert (np.isnan(got) == np.isnan(ref)).all() and (np.isposinf(got) == np.isposinf(ref)).all()
        assert (np.isneginf(got) == np.isneginf(ref)).all()
        fin = np.isfinite(ref)
        if fin.any():  # 9 chains of 64 roundings of 2^-24, and the angles' 2^-20 of the highest octave
            scale = np.abs(ref[fin].astype(np.float64)).max()
            assert np.abs(got[fin].astype(np.float64) - ref[fin]).max() <= 1e-5 * scale
    net.load_params(p)
    assert (net.inference(dx).cpu().numpy() == plain).all()


@pytest.mark.gpu
def test_training_counts_wide_weights(sty, cuda):
    """Optimiser steps of 1e6 carry weights past the bound of a 5-layer network (2^14): what inference gives is what a
    network loaded with the same weights gives."""
    import torch
    rng = np.random.default_rng(2)
    x, t = torch.from_numpy(rng.random((500, 11), np.float32)).cuda(), torch.from_numpy(rng.random((500, 3), np.float32) + 0.1).cuda()
    net = sty.nrc.NRC(sty.nrc.config(FREQS, 3, 128, 5, sty.nrc.STY_NRC_FP32, learning_rate=1e-3, seed=4))
    other = sty.nrc.NRC(sty.nrc.config(FREQS, 3, 128, 5, sty.nrc.STY_NRC_FP32, seed=4))
    seen = set()
    for lr in (1e-3, 1e6, 1e-3, 1e6):
        sty.check(sty.lib().sty_nrc_set_learning_rate(net.h, lr))
        net.train(x, t, 1)
        p = net.save_params()
        seen.add(bool((np.abs(p) > 2.0 ** 14).any()))
        other.load_params(p)
        a, b = net.inference(x, ema=False).cpu().numpy(), other.inference(x, ema=False).cpu().numpy()
        assert np.array_equal(a, b, equal_nan=True)
    assert seen == {False, True}
