"""The quantised 4-wide tree and its walks against the brute-force oracle: hits are the least (t, id) of all
triangles in the same rounded arithmetic, so ids, distances and barycentrics are compared bit for bit."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _soup(n, rng, kind):
    if kind == "flat":  # unit quads of the plane y = 0.5: boxes without extent along y
        k = int(np.ceil(np.sqrt((n + 1) // 2)))
        out = []
        for i in range((n + 1) // 2):
            x, z = float(i % k), float(i // k)
            a, b, c, d = (x, 0.5, z), (x + 1, 0.5, z), (x + 1, 0.5, z + 1), (x, 0.5, z + 1)
            out += [a + b + c, a + c + d]
        return np.array(out[:n], np.float32)
    c = rng.uniform(-1, 1, (n, 1, 3))
    t = (c + rng.normal(scale=0.2, size=(n, 3, 3))).astype(np.float32)
    if kind == "far":
        t += np.float32(5000.0)
    elif kind == "tiny":
        t *= np.float32(1e-5)
    elif kind == "twice":  # every triangle a second time: the lower id wins
        t[n // 2: n // 2 * 2] = t[: n // 2]
    return t.reshape(n, 9)


def _rays(pos, rng, m=6000):
    v = pos.reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    ext = np.maximum(hi - lo, (hi - lo).max() * 0.1).astype(np.float32)
    r = np.zeros((m, 8), np.float32)
    r[:, 0:3] = (lo - 0.5 * ext) + rng.random((m, 3), np.float32) * (2 * ext)
    d = rng.normal(size=(m, 3))
    r[:, 3:6] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 1e20
    k = m // 6
    for a in range(3):  # one component +0 / -0
        r[a * k // 2:(a + 1) * k // 2, 3 + a] = np.where(np.arange((a + 1) * k // 2 - a * k // 2) % 2, 0.0, -0.0)
    r[2 * k:3 * k, 3:6] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, k)] * rng.choice([-1, 1], (k, 1))
    s = rng.integers(0, v.shape[0], (k, 3))  # origins in the planes of vertices
    r[3 * k:4 * k, 0] = v[s[:, 0], 0]
    r[2 * k:4 * k:2, 1] = v[rng.integers(0, v.shape[0], k), 1]
    r[4 * k:5 * k, 7] = rng.random(k, np.float32) * np.linalg.norm(ext)  # a far limit
    r[5 * k:, 6] = rng.random(m - 5 * k, np.float32) * 0.3 * np.linalg.norm(ext)  # a near limit
    return r


@pytest.mark.parametrize("kind", ["soup", "flat", "far", "tiny", "twice"])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 17, 300])
def test_hits_match_the_oracle(sty, cuda, n, kind):
    import torch
    rng = np.random.default_rng(n)
    pos = _soup(n, rng, kind)
    _, _, mats, cam = sty.scene.cornell_box(8, 8)
    sc = sty.scene.Scene(pos, np.zeros(n, np.uint32), mats, cam)
    rays = _rays(pos, rng)
    prim, t, b = sc.closest_hit(torch.from_numpy(rays).cuda())
    rp, rt, rb = oracle.closest_hit(pos, rays)
    assert (prim.cpu().numpy().view(np.uint32) == rp).all()
    hit = rp != 0xFFFFFFFF
    assert hit.any() and (t.cpu().numpy()[hit] == rt[hit]).all() and (b.cpu().numpy()[hit] == rb[hit]).all()
    sc.close()


@pytest.mark.parametrize("size,inner", [((1, 1), (1,)), ((1, 1), (33,)), ((3, 1), (11, 1)), ((5, 3), (9, 2)), ((1, 9), (64,))])
def test_branches_of_small_films(sty, cuda, size, inner):
    """Ray counts below, at and above a warp and a block of the walk. FP32 against the FP64 oracle from the same
    random numbers: ~1e-5, and 1e-3 of the reference scale is allowed (a ray that grazes an edge moves a
    pixel by more; of these few hundred rays none is expected to)."""
    W, H = size
    pos, mids, mats, cam = sty.scene.cornell_box(W, H)
    sc = sty.scene.Scene(pos, mids, mats, cam)
    film, st = sc.brpt_render(sty.scene.brpt_config(max_depth=3, inner_samples=inner, repeats=1, vram_mb=64, seed=5), ())
    camv = list(cam.eye) + list(cam.target) + list(cam.up) + [cam.fov_y, cam.width, cam.height, cam.filter_radius]
    ref = oracle.brpt(pos, mids, (sty.scene.SceneMaterial * len(mats))(*mats), camv, (), 3, inner, repeats=1, seed=5)
    img = film.cpu().numpy()
    assert st.vertices > 0 and ref.max() > 0
    assert np.abs(img - ref).max() <= 1e-3 * ref.max(), (img, ref)
    sc.close()
