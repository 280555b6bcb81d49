"""How exact the FP32 network's inference is, at a grain that shows every part of its three-way BF16 split.

Inputs are multiples of 1/2, whose frequency encoding is exact (0 and +-1), so what is measured is the layers alone.
Bounds: a dropped piece product costs 2^-17 (a2w2, a1w3, a3w1: of a product, ~64 to a sum, a layer; 2e-6 and more of
the output scale), all six leave 2^-25; an accumulation in the tensor core cuts at most 2^-23 of a partial sum, ~6 times a layer,
half of that on average and given back by the third piece (nrc.cuh). So 1.5e-6 of the output scale in the maximum, no more
than FMA chains in the norm (each of their 64 steps rounds by up to 2^-25), and 1e-7 in the mean, where the cuts
of 5 layers alone would leave 2e-7."""
import numpy as np
import pytest

FREQS = (4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2)
MAX, NORM, MEAN = 1.5e-6, 1.0, 1e-7


def _case(layers, out, rows):
    rng = np.random.default_rng(100 * layers + out)
    p = (rng.standard_normal(layers * 4096 + out * 64) * np.sqrt(2.0 / 64)).astype(np.float32)
    x = (rng.integers(0, 4, (rows, 11)) * 0.5).astype(np.float32)
    cols = []
    for d, f in enumerate(FREQS):
        for k in range(f):
            a = np.pi * x[:, d].astype(np.float64) * 2.0 ** k
            cols += [np.round(np.sin(a)), np.round(np.cos(a))]
    h = np.zeros((rows, 64))
    h[:, :len(cols)] = np.stack(cols, 1)
    return p, x, h


def _layers(p, h, product):
    n = p.size // 4096
    for l in range(n):
        h = np.maximum(product(h, p[l * 4096:(l + 1) * 4096].reshape(64, 64)), 0)
    return h @ p[n * 4096:].reshape(-1, 64).T.astype(np.float64)


def _exact(p, h):
    return _layers(p, h, lambda a, w: a @ w.T.astype(np.float64))


def _chain(p, h):
    """FP32 FMA chains over k = 0 .. 63, the output layer's too."""
    def dot(a, w):
        s = np.zeros((a.shape[0], w.shape[0]), np.float32)
        for k in range(64):
            s = (w[:, k].astype(np.float64) * a[:, k:k + 1].astype(np.float64) + s).astype(np.float32)
        return s
    n = p.size // 4096
    for l in range(n):
        h = np.maximum(dot(h, p[l * 4096:(l + 1) * 4096].reshape(64, 64)), 0)
    return dot(h, p[n * 4096:].reshape(-1, 64)).astype(np.float64)


def _pieces(v):
    import torch
    r, got = torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)), []
    for _ in range(3):
        b = r.bfloat16().float()
        got.append(b.numpy().astype(np.float64))
        r = r - b
    return got


def _split(p, h, used):
    def product(a, w):
        pa, pw = _pieces(a), _pieces(w)
        return sum(pa[i] @ pw[j].T for i, j in used).astype(np.float32).astype(np.float64)
    return _layers(p, h, product)


SIX = ((0, 0), (0, 1), (1, 0), (1, 1), (0, 2), (2, 0))


@pytest.mark.parametrize("drop", [None, (0, 1), (1, 0), (1, 1), (0, 2), (2, 0)])
@pytest.mark.parametrize("layers,out", [(1, 3), (2, 16), (5, 3), (8, 4)])
def test_the_bounds_show_a_dropped_product(layers, out, drop):
    p, _, h = _case(layers, out, 500)
    ref, got = _exact(p, h), _split(p, h, [u for u in SIX if u != drop])
    err = np.abs(got - ref).max() / np.abs(ref).max()
    # (a first layer of 0 and +-1 has nothing in its activations' lower pieces)
    if drop is None or (layers == 1 and drop[0] > 0):
        assert err <= MAX / 4
    else:
        assert err > MAX


@pytest.mark.gpu
@pytest.mark.parametrize("layers,out,rows", [(1, 3, 4096), (2, 16, 1000), (3, 1, 129), (5, 3, 40000), (8, 4, 5000)])
def test_inference_error(sty, cuda, layers, out, rows):
    import torch
    p, x, h = _case(layers, out, rows)
    net = sty.nrc.NRC(sty.nrc.config(FREQS, out, 128, layers, sty.nrc.STY_NRC_FP32, seed=1))
    net.load_params(p)
    ref, chain = _exact(p, h), _chain(p, h)
    for ema in (True, False):
        err = net.inference(torch.from_numpy(x).cuda(), ema=ema).cpu().numpy().astype(np.float64) - ref
        assert np.abs(err).max() <= MAX * np.abs(ref).max()
        assert np.linalg.norm(err) <= NORM * np.linalg.norm(chain - ref)
        assert abs((err * np.sign(ref)).mean()) <= MEAN * np.abs(ref).mean()
