"""Scenes with closure materials are traced by several kernels per depth from a size on, others by one. A closure material
that no triangle has chooses the kernels and changes nothing else, so records and films have to be the same with and
without it, bit for bit, on both sides of the line (a block of 256 paths per SM) and at sizes that cut a block short."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scenes(sty, w, h):
    pos, ids, mats, cam = sty.scene.cornell_box(w, h)
    return [sty.scene.Scene(pos, ids, list(mats) + extra, cam) for extra in ([], [sty.scene.principled()], [sty.scene.glass()])]


@pytest.mark.parametrize("w,h,branch,depth", [(1, 1, 1, 3), (48, 48, 16, 4), (50, 49, 16, 4), (64, 65, 16, 0), (131, 77, 8, 5)])
def test_records(sty, cuda, w, h, branch, depth):
    cfg = sty.scene.screen_render_config(max_depth=depth, branch=branch, radius=1, sigma_pixel=0.0, screen_style=-1, seed=5)
    got = []
    for sc in _scenes(sty, w, h):
        rs, prim, vc = sc.trace_records(cfg, (), with_prim=True)
        got.append((rs.planes.cpu().numpy(), rs.valid.cpu().numpy(), prim.cpu().numpy(), vc))
        sc.close()
    assert got[0][3] > 0
    for other in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.parametrize("w,h", [(1, 1), (17, 15), (200, 199)])
def test_final_gather(sty, cuda, w, h):
    films = []
    for sc in _scenes(sty, w, h):
        net = sty.nrc.NRC(sty.nrc.config(sty.nrc.C4_FREQS, 3, 128, 2, sty.nrc.STY_NRC_FP32, seed=3))
        film, _ = sc.nrc_render(net, sty.scene.nrc_render_config(max_depth=4, training_iters=1, batches_per_iter=1, final_gather=3), ())
        films.append(film.cpu().numpy())
        sc.close()
    assert np.isfinite(films[0]).all() and (w * h == 1 or films[0].max() > 0)
    assert (films[1] == films[0]).all() and (films[2] == films[0]).all()
