"""The device memory a scene keeps between calls: never above a later call's budget, and given back when asked for."""
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _render(sty, sc, vram_mb):
    film, st = sc.brpt_render(sty.scene.brpt_config(max_depth=5, inner_samples=(64, 16), repeats=1, vram_mb=vram_mb, seed=2), ())
    return film.cpu(), st


def test_brpt_workspace(sty, cuda):
    """1.0 M vertex slots of 100 bytes per worst-case tree of 4161 slots a pixel: 48 x 27 pixels want 540 MB, of which a
    budget of 64 MB is an eighth. 32 MB for what else a call allocates or the driver rounds."""
    import torch
    sc = sty.scene.Scene(*sty.scene.cornell_box(48, 27))
    small, _ = _render(sty, sc, 64)  # everything but the workspace is there from here on
    sc.trim()
    torch.cuda.empty_cache()
    base = _free()
    big, st = _render(sty, sc, 4096)
    kept = base - _free()
    assert st.passes == 1 and kept > 256 * MB
    again, st = _render(sty, sc, 64)
    assert st.passes > 1 and base - _free() <= (64 + 32) * MB
    assert (again == big).all() and (small == big).all()
    _render(sty, sc, 4096)
    sc.trim()
    assert base - _free() <= 32 * MB
    after, _ = _render(sty, sc, 4096)
    assert (after == big).all()
    sc.close()


def test_trim_gives_render_buffers_back(sty, cuda):
    import torch
    sc = sty.scene.Scene(*sty.scene.cornell_box(256, 256))
    cfg = sty.scene.screen_render_config(max_depth=5, branch=16, radius=1, screen_style=-1, seed=1)
    film = torch.zeros((256, 256, 3), dtype=torch.float64, device="cuda")
    base = _free()
    sc.render(cfg, (), film=film)
    assert base - _free() > 256 * MB
    first = film.cpu()
    sc.trim()
    assert base - _free() <= 32 * MB
    film.zero_()
    sc.render(cfg, (), film=film)
    assert (film.cpu() == first).all()
    sc.close()
