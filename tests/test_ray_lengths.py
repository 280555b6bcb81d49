"""Rays whose directions are far from unit length: a direction times 2^e meets the same triangles at 2^-e times the
distance. Against the brute-force oracle in the same rounded arithmetic, bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-124, -100, -80, -50, -20, 0, 20, 60, 100, 124, 126])
def test_direction_lengths(sty, cuda, e):
    import torch
    rng = np.random.default_rng(200 + e)
    n, m = 300, 3000
    pos = (rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(scale=0.2, size=(n, 3, 3))).astype(np.float32).reshape(n, 9)
    _, _, mats, cam = sty.scene.cornell_box(8, 8)
    sc = sty.scene.Scene(pos, np.zeros(n, np.uint32), mats, cam)
    r = np.zeros((m, 8), np.float32)
    r[:, :3] = rng.uniform(-1.5, 1.5, (m, 3))
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[: m // 6, 0] = 0.0
    d[m // 6: m // 3, 1:] = 0.0
    d[m // 3: m // 2, 2] *= 1e-26  # (nearly) 0 beside the others
    r[:, 3:6] = (d * 2.0 ** e).astype(np.float32)
    r[:, 7] = 1e20 if e >= 0 else min(1e20 * 2.0 ** -e, 3e38)
    prim, t, b = sc.closest_hit(torch.from_numpy(r).cuda())
    rp, rt, rb = oracle.closest_hit(pos, r)
    hit = rp != 0xFFFFFFFF
    assert hit.sum() > m // 10
    assert (prim.cpu().numpy().view(np.uint32) == rp).all()
    assert (t.cpu().numpy()[hit] == rt[hit]).all() and (b.cpu().numpy()[hit] == rb[hit]).all()
    sc.close()
