"""The work that users of this library have it do, as measurable cases.

Every case goes through the package's public calls, with the sizes of the repository's own workloads
(the 1080p x 4 spp filter, the Cornell box and interior renders, the adjoint of the 512 x 512 image,
the neural cache's 2^16 / 2^14 training batches and 1080p query frames) and smaller, ragged ones.

Where a case styles its result it uses the smoothed ramp, and only the branching path tracer's case
the hard toon steps too: a quantising node turns the last bit of a value that lies on a band edge into
a whole step, so images styled with it can be compared with each other only bit for bit.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import __graft_entry__

sty = __graft_entry__.package()

L2E = 1.4426950408889634
DEV = "cuda:0"
# the ramp of the interior workload
RAMP = (30.0, (0.02, 0.15, 0.6), ((0.08, 0.1, 0.2), (0.55, 0.45, 0.35), (1.3, 1.2, 1.0)))
#: pair evaluations of the largest filter case; a drawn one stays under it (and under a quarter of it
#: where the samples per pixel are not 4, whose kernels do fewer pairs a second)
MOST_PAIRS = 5 * 1920 * 1080 * 16 * 33 * 33


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # the filter's headline workload: a whole backward pass over five path depths of a 1080p frame
        dict(name="filter_1080p", kind="filter", width=1920, height=1080, spp=4, depths=5, radius=16, sigma_pixel=8.0, sigma_pos=0.5, sigma_nrm=0.2, style=True),
        # an interactive preview of odd size, one depth with the depth below as child: few tiles, a short launch
        dict(name="filter_preview", kind="filter_depth", width=321, height=181, spp=4, depths=1, radius=8, sigma_pixel=4.0, sigma_pos=0.5, sigma_nrm=0.2, style=True),
        # the Cornell box end to end, traced, filtered with the bilateral filter and splatted (16 paths a pixel)
        dict(name="render_screen_cornell", kind="render_screen", scene="cornell", width=256, height=256, branch=16, depth=5, radius=8),
        # the same render with the reference's world-space hash-grid filter (SMIS, reservoirs of 64)
        dict(name="render_ref_cornell", kind="render_ref", scene="cornell", width=256, height=256, branch=16, depth=5, radius_scale=5.0, reuse=64, smis=True, cluster=False),
        # one gradient of the filter's and the ramp's 36 parameters, the inverse-stylization step
        dict(name="adjoint_512", kind="adjoint", width=512, height=512, spp=4, radius=8, steps=8),
        # the cache's training burst of a frame: four steps of 2^16 samples on the tensor cores
        dict(name="nrc_train_bf16", kind="nrc_train", precision="bf16", batch=1 << 16, rows=100000, layers=5, iters=4),
        # the same loop in FP32 at the online render's batch
        dict(name="nrc_train_fp32", kind="nrc_train", precision="fp32", batch=1 << 14, rows=30000, layers=5, iters=4),
        # one cache query per pixel of a 1080p frame
        dict(name="nrc_infer_bf16_1080p", kind="nrc_infer", precision="bf16", rows=1920 * 1080, layers=5),
        # a quarter-resolution frame of an odd row count through the FP32 cache
        dict(name="nrc_infer_fp32", kind="nrc_infer", precision="fp32", rows=480 * 270 + 1, layers=5),
        # a frame with the reference's network (hash grid, one-blob, 5 x 128): one training step and a query per pixel
        dict(name="grid_frame_1080p", kind="grid_frame", width=1920, height=1080, batch=1 << 16, fp16=False),
        # forward and backward of the reference's network on one online batch, the tables' gradients among the result
        dict(name="grid_gradient", kind="grid_gradient", batch=1 << 14, fp16=False),
        # the branching path tracer on the tessellated interior
        dict(name="brpt_interior", kind="brpt", scene="room", width=160, height=90, depth=8, inner="16,8,4", repeats=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter_depth", "render_screen", "render_ref", "adjoint", "nrc_train", "nrc_infer", "nrc_infer", "grid_frame", "grid_gradient", "brpt"])
    if kind in ("filter", "filter_depth"):
        spp = rng.choice([4, 4, 4, 16, 1, 2, 8])
        while True:
            c = dict(kind=kind, width=_log(rng, 40, 1920), height=_log(rng, 24, 1080), spp=spp, depths=rng.randint(1, 5) if kind == "filter" else 1, radius=rng.randint(3, 16),
                     sigma_pixel=rng.choice([0.0, 4.0, 8.0]), sigma_pos=rng.choice([0.5, 0.7]), sigma_nrm=rng.choice([0.2, 0.3]), style=rng.random() < 0.5)
            if _pairs(c) <= MOST_PAIRS // (1 if spp == 4 else 4):
                return c
    if kind == "render_screen":
        return dict(kind=kind, scene=rng.choice(["cornell", "room"]), width=_log(rng, 64, 256), height=_log(rng, 48, 256), branch=rng.choice([4, 8, 16]), depth=rng.randint(2, 5), radius=rng.randint(4, 8))
    if kind == "render_ref":
        return dict(kind=kind, scene=rng.choice(["cornell", "room"]), width=_log(rng, 64, 256), height=_log(rng, 48, 192), branch=rng.randint(2, 12), depth=rng.randint(2, 5),
                    radius_scale=rng.choice([1.0, 2.0, 4.0]), reuse=rng.choice([16, 32, 64]), smis=rng.random() < 0.75, cluster=rng.random() < 0.25)
    if kind == "adjoint":
        return dict(kind=kind, width=_log(rng, 48, 512), height=_log(rng, 32, 512), spp=rng.choice([4, 4, 1]), radius=rng.randint(4, 8), steps=rng.randint(2, 8))
    if kind == "nrc_train":
        return dict(kind=kind, precision=rng.choice(["bf16", "fp32"]), batch=128 * _log(rng, 8, 512), rows=_log(rng, 5000, 200000), layers=rng.randint(2, 6), iters=rng.randint(1, 4))
    if kind == "nrc_infer":
        return dict(kind=kind, precision=rng.choice(["bf16", "fp32"]), rows=_log(rng, 500, 1920 * 1080), layers=rng.randint(2, 6))
    if kind == "grid_frame":
        return dict(kind=kind, width=_log(rng, 96, 1920), height=_log(rng, 54, 1080), batch=128 * _log(rng, 32, 512), fp16=rng.random() < 0.25)
    if kind == "grid_gradient":
        return dict(kind=kind, batch=128 * _log(rng, 16, 512), fp16=rng.random() < 0.25)
    return dict(kind="brpt", scene=rng.choice(["room", "cornell"]), width=_log(rng, 48, 160), height=_log(rng, 27, 90), depth=rng.randint(4, 8), inner=rng.choice(["8,4", "16,8,4", "1", "32,4"]), repeats=rng.randint(1, 2))


def _pairs(c):
    return c["depths"] * c["width"] * c["height"] * c["spp"] ** 2 * (2 * c["radius"] + 1) ** 2


# ---- inputs ---------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _records(c, g):
    """The synthetic path-vertex records of practical-stylized_gb300/synth.py (uniform positions about a smooth
    per-pixel offset, von Mises-Fisher normals about 8 x 8-tile means, lognormal radiance, 10 % invalid), made
    on the GPU. The offset's slope per pixel is that of the 1920-pixel frame at every size."""
    w, h, s, d = c["width"], c["height"], c["spp"], c["depths"]
    n = w * h * s
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32), torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    u, v = (x + 0.5) / 1920.0, (y + 0.5) / 1080.0
    off = 4.0 * torch.stack([2 * u - 1, 2 * v - 1, 0.5 * torch.sin(2 * math.pi * u) * torch.cos(2 * math.pi * v)]).reshape(3, h * w)
    off = off.repeat_interleave(s, 1)
    tw, th = (w + 7) // 8, (h + 7) // 8
    tile = ((y // 8).long() * tw + (x // 8).long()).reshape(-1).repeat_interleave(s)
    planes = torch.empty((12, d, n), device=DEV)
    valid = torch.empty((d, n), dtype=torch.int32, device=DEV)
    for k in range(d):
        planes[0:3, k] = torch.rand((3, n), generator=g, device=DEV) * 2 - 1 + off
        mu = torch.randn((3, tw * th), generator=g, device=DEV)
        mu = (mu / mu.norm(dim=0))[:, tile]
        xi = torch.rand(n, generator=g, device=DEV)
        cw = 1 + torch.log(xi + (1 - xi) * math.exp(-40.0)) / 20.0
        phi = 2 * math.pi * torch.rand(n, generator=g, device=DEV)
        r = torch.sqrt((1 - cw * cw).clamp_min(0))
        a = torch.where(mu[:1].abs() > 0.9, torch.tensor([[0.0], [1.0], [0.0]], device=DEV), torch.tensor([[1.0], [0.0], [0.0]], device=DEV))
        t = torch.linalg.cross(a, mu, dim=0)
        t = t / t.norm(dim=0)
        b = torch.linalg.cross(mu, t, dim=0)
        nr = r * torch.cos(phi) * t + r * torch.sin(phi) * b + cw * mu
        planes[3:6, k] = nr / nr.norm(dim=0)
        planes[6:9, k] = torch.exp(torch.randn((3, n), generator=g, device=DEV) * 1.5 - 1.0)
        planes[9:12, k] = torch.rand((3, n), generator=g, device=DEV)
        valid[k] = (torch.rand(n, generator=g, device=DEV) >= 0.1).int()
    return planes.reshape(12, d * n), valid.reshape(d * n)


def _ramp_program(depth_mask):
    return sty.abi.style_program([sty.abi.ramp_smooth(*RAMP, depth_mask=depth_mask)])


def _scene(c, seed):
    if c["scene"] == "cornell":
        return sty.scene.cornell_box(c["width"], c["height"], style=(0, -1, -1, -1))
    return sty.scene.room_with_door(c["width"], c["height"], cell=0.05, seed=seed)


def _surface_records(c, g):
    """Records as a traced depth 0 leaves them: points on a few smooth surfaces that change at object edges,
    each path jittered inside its pixel, radiance smooth with path noise."""
    w, h, s = c["width"], c["height"], c["spp"]
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32), torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    jx, jy = (torch.rand((h, w, s), generator=g, device=DEV) for _ in range(2))
    u, v = (x[..., None] + jx) / max(w, h), (y[..., None] + jy) / max(w, h)
    box = ((u * 5).floor() + (v * 4).floor()) % 3  # which surface the path hits
    k = box.long()
    nrm = torch.tensor([[0.0, 0.0, 1.0], [0.6, 0.0, 0.8], [0.0, -0.8, 0.6]], device=DEV)[k]
    p = torch.stack([u, v, 0.3 * box + 0.05 * torch.sin(9 * u) * nrm[..., 0]], -1)
    rad = torch.stack([(0.3 + 0.25 * torch.sin(7 * u + i) * torch.cos(5 * v)) for i in range(3)], -1)
    rad = rad * torch.exp(0.5 * torch.randn((h, w, s, 1), generator=g, device=DEV))
    thr = torch.rand((h, w, s, 3), generator=g, device=DEV)
    planes = torch.cat([p, nrm, rad, thr], -1).reshape(-1, 12).t().contiguous()
    valid = (torch.rand(h * w * s, generator=g, device=DEV) >= 0.02).int()
    child = torch.exp(torch.randn((3, h * w * s), generator=g, device=DEV) - 1.5)
    return planes, valid, child


def _adjoint_params(c, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(36)
    p[0] = 50.0
    p[1:9] = np.sort(rng.uniform(0.02, 0.8, 8))
    p[9:33] = np.sort(rng.uniform(0.0, 1.0, 24))
    p[33:36] = [4.0, 0.05, 0.2]
    return p.astype(np.float32)


def _mlp_params(layers, seed, width=64, out=3):
    """Weights of a small cache part-way through training (He-scaled)."""
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(layers * width * width + out * width) * math.sqrt(2.0 / width)).astype(np.float32)


def _cache_rows(n, seed):
    """Rows of the frequency-encoded cache (11 inputs in [0, 1)) with smooth positive targets and path noise."""
    g = _gen(seed)
    x = torch.rand((n, 11), generator=g, device=DEV)
    t = torch.exp(torch.sin(6 * x[:, :3]) + 0.5 * torch.cos(4 * x[:, 3:6]) + 0.5 * torch.randn((n, 3), generator=g, device=DEV) - 1.0)
    return x, t.contiguous()


GRID_DEPTH, GRID_LEVELS, GRID_ENC, GRID_WIDTH = 8, 22, 144, 128


def _grid_net(c):
    return sty.nrc.NRC(sty.nrc.grid_config(max_depth=GRID_DEPTH, batch_size=c["batch"], learning_rate=1e-3, seed=1, fp16=c["fp16"]))


def _grid_levels():
    """(scale, resolution, table entries) of the 22 levels: base resolution 16, doubled from level to level, tables of at most 2^19 entries."""
    got = []
    for lev in range(GRID_LEVELS):
        res = 16 * 2 ** lev
        got.append((float(np.float32(res - 1)), res, min((res ** 3 + 7) // 8 * 8, 1 << 19)))
    return got


def _grid_params(seed):
    """Weights of the hash-grid network part-way through training: He-scaled layers, features of about 0.05."""
    n_mlp = GRID_WIDTH * GRID_ENC + 4 * GRID_WIDTH * GRID_WIDTH + 3 * GRID_WIDTH
    g = _gen(seed)
    p = torch.empty(n_mlp + 4 * sum(s for _, _, s in _grid_levels()), device=DEV)
    p[:n_mlp] = torch.randn(n_mlp, generator=g, device=DEV) * math.sqrt(2.0 / GRID_WIDTH)
    p[n_mlp:] = (torch.rand(p.numel() - n_mlp, generator=g, device=DEV) * 2 - 1) * 0.05
    return p


def _room_hits(o, d, seed):
    """First hits of rays inside a 6 x 3 x 4 room with 12 spheres: position in [0, 1]^3, normal."""
    rng = np.random.default_rng(seed)
    size = torch.tensor([6.0, 3.0, 4.0], device=DEV)
    t = torch.where(d > 0, (size - o) / d, -o / d).nan_to_num(1e9)
    best, axis = t.min(1)
    n = torch.zeros_like(d).scatter_(1, axis[:, None], -torch.sign(d.gather(1, axis[:, None])))
    for _ in range(12):
        r = float(rng.uniform(0.15, 0.5))
        c = torch.tensor([rng.uniform(1.0, 5.5), rng.uniform(r, 1.6), rng.uniform(0.5, 3.5)], device=DEV, dtype=torch.float32)
        b = ((o - c) * d).sum(1)
        disc = b * b - ((o - c) ** 2).sum(1) + r * r
        ts = -b - disc.clamp_min(0).sqrt()
        hit = (disc > 0) & (ts > 1e-3) & (ts < best)
        best = torch.where(hit, ts, best)
        n = torch.where(hit[:, None], (o + ts[:, None] * d - c) / r, n)
    return ((o + best[:, None] * d) / size).clamp(0, 1), n


def _grid_rows(o, d, depth, seed):
    """Rows of the reference's layout (20 + max depth inputs) at the first hits of the given rays."""
    p, n = _room_hits(o, d, seed)
    k = o.shape[0]
    rough = 0.3 + 0.7 * (p[:, 1:2] > 0.01)
    albedo = 0.5 + 0.3 * torch.sin(torch.stack([p[:, 0], p[:, 1] + 1, p[:, 2] + 2], 1) * 9).sign() * 0.5
    flags = torch.tensor([0.0, 1.0, 1.0, 0.0, 0.0, 0.0], device=DEV).expand(k, 6)
    hot = torch.zeros((k, GRID_DEPTH + 1), device=DEV).scatter_(1, depth[:, None], 1.0)
    return torch.cat([p, n * 0.5 + 0.5, -d * 0.5 + 0.5, rough, albedo, flags, hot], 1).contiguous()


def _view_rows(w, h, seed):
    """One row per pixel of a w x h view into the room, in the order of the pixels."""
    g = _gen(seed)
    y, x = torch.meshgrid(torch.arange(h, device=DEV, dtype=torch.float32), torch.arange(w, device=DEV, dtype=torch.float32), indexing="ij")
    j = torch.rand((2, h, w), generator=g, device=DEV)
    f = 1.15 / h
    d = torch.stack([torch.ones_like(x), -(y + j[0] - h / 2) * f, (x + j[1] - w / 2) * f], -1).reshape(-1, 3)
    o = torch.tensor([0.4, 1.6, 2.0], device=DEV).expand_as(d)
    return _grid_rows(o, d / d.norm(dim=1, keepdim=True), torch.zeros(w * h, dtype=torch.long, device=DEV), seed)


def _path_rows(n, seed):
    """Training rows: vertices of paths through the room at mixed depths, with noisy targets."""
    g = _gen(seed)
    o = torch.rand((n, 3), generator=g, device=DEV) * torch.tensor([5.0, 2.0, 3.0], device=DEV) + 0.5
    d = torch.randn((n, 3), generator=g, device=DEV)
    x = _grid_rows(o, d / d.norm(dim=1, keepdim=True), torch.randint(0, GRID_DEPTH + 1, (n,), generator=g, device=DEV), seed)
    t = torch.exp(torch.sin(5 * x[:, :3]) + 0.5 * torch.randn((n, 3), generator=g, device=DEV) - 1.0)
    return x, t.contiguous()


# ---- one state and one pass ------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(c)
    if kind in ("filter", "filter_depth"):
        planes, valid = _records(c, _gen(seed))
        n = c["width"] * c["height"] * c["spp"]
        st["rs"] = sty.RecordSet(planes, valid, c["width"], c["height"], c["spp"], c["depths"])
        st["params"] = sty.ScreenParams(c["radius"], c["sigma_pixel"], c["sigma_pos"], c["sigma_nrm"])
        if kind == "filter":  # the ramp at the first bounce (depth 0 where there is one depth only)
            st["style"] = _ramp_program(1 << min(1, c["depths"] - 1)) if c["style"] else None
            st["out"] = torch.empty((c["depths"], 3, n), device=DEV)
        else:
            st["style"] = _ramp_program(1) if c["style"] else None
            st["child"] = torch.exp(torch.randn((3, n), generator=_gen(seed + 1), device=DEV) - 1.5)
            st["out"], st["filtered"] = torch.empty((3, n), device=DEV), torch.empty((3, n), device=DEV)
    elif kind in ("render_screen", "render_ref"):
        st["scene"] = sty.scene.Scene(*_scene(c, seed))
        st["progs"] = [_ramp_program(0b11)]
        if kind == "render_screen":
            st["cfg"] = sty.scene.screen_render_config(max_depth=c["depth"], branch=c["branch"], radius=c["radius"], sigma_pixel=0.0, sigma_pos=0.05, sigma_nrm=0.2, screen_style=0, seed=seed)
        else:
            st["cfg"] = sty.scene.render_config(max_depth=c["depth"], branch=c["branch"], radius_scale=(c["radius_scale"],), reuse=(c["reuse"],), smis=c["smis"], cluster=c["cluster"], seed=seed)
    elif kind == "adjoint":
        st["planes"], st["valid"], st["child"] = _surface_records(c, _gen(seed))
        st["rs"] = sty.RecordSet(st["planes"], st["valid"], c["width"], c["height"], c["spp"], 1)
        st["prm"] = (C.c_float * 36)(*_adjoint_params(c, seed))
        st["target"] = 0.2 + 0.6 * torch.rand((c["height"], c["width"], 3), generator=_gen(seed + 1), device=DEV)
        st["grad"] = torch.empty(36, device=DEV)
    elif kind == "nrc_train":
        prec = sty.nrc.STY_NRC_BF16 if c["precision"] == "bf16" else sty.nrc.STY_NRC_FP32
        st["net"] = sty.nrc.NRC(sty.nrc.config(sty.nrc.C4_FREQS, 3, c["batch"], c["layers"], prec, learning_rate=1e-2, seed=1))
        st["x"], st["t"] = _cache_rows(c["rows"], seed)
    elif kind == "nrc_infer":
        prec = sty.nrc.STY_NRC_BF16 if c["precision"] == "bf16" else sty.nrc.STY_NRC_FP32
        st["net"] = sty.nrc.NRC(sty.nrc.config(sty.nrc.C4_FREQS, 3, 1 << 14, c["layers"], prec, seed=1))
        st["net"].load_params(_mlp_params(c["layers"], seed))
        st["x"], _ = _cache_rows(c["rows"], seed)
        st["out"] = torch.empty((c["rows"], 3), device=DEV)
    elif kind in ("grid_frame", "grid_gradient"):
        st["net"] = _grid_net(c)
        st["net"].load_params(_grid_params(seed).cpu().numpy())
        st["x"], st["t"] = _path_rows(2 * c["batch"] if kind == "grid_frame" else c["batch"], seed)
        if kind == "grid_frame":
            st["q"] = _view_rows(c["width"], c["height"], seed)
            st["out"] = torch.empty((st["q"].shape[0], 3), device=DEV)
    else:
        st["scene"] = sty.scene.Scene(*_scene(c, seed))
        st["progs"] = [sty.abi.style_program([sty.abi.toon(0.2, depth_mask=0b11), sty.abi.ramp_smooth(*RAMP, depth_mask=0b11)])]
        inner = tuple(int(v) for v in c["inner"].split(","))
        st["cfg"] = sty.scene.brpt_config(max_depth=c["depth"], inner_samples=inner, repeats=c["repeats"], vram_mb=16384, seed=seed)
    return st


def run(state):
    s, kind = state, state["kind"]
    if kind == "filter":
        return list(sty.pf_screen_filter(s["rs"], s["params"], s["style"], out=s["out"]).unbind(0))
    if kind == "filter_depth":
        out = sty.pf_screen_filter_depth(s["rs"], 0, s["params"], s["style"], out_next=s["child"], out=s["out"], filtered=s["filtered"])
        return [out, s["filtered"]]
    if kind in ("render_screen", "render_ref"):
        film, vertices = s["scene"].render(s["cfg"], s["progs"])
        return [film, vertices]
    if kind == "adjoint":
        rec = s["rs"].c()
        sty.check(sty.lib().sty_pf_adjoint(C.byref(rec), 0, s["radius"], s["prm"], s["steps"], s["child"].data_ptr(), s["target"].data_ptr(), s["grad"].data_ptr(), None,
                                           torch.cuda.current_stream().cuda_stream or None))
        return [s["grad"]]
    if kind == "nrc_train":
        loss = s["net"].train(s["x"], s["t"], s["iters"])
        return [loss, s["net"].save_params()]
    if kind == "nrc_infer":
        return [s["net"].inference(s["x"], s["out"])]
    if kind == "grid_frame":
        s["net"].train(s["x"], s["t"], 1, want_loss=False)
        return [s["net"].inference(s["q"], s["out"])]
    if kind == "grid_gradient":
        grad, loss = s["net"].gradient(s["x"], s["t"])
        return [loss, grad]
    film, stats = s["scene"].brpt_render(s["cfg"], s["progs"])
    return [film, int(stats.vertices)]


# ---- what a pass cannot do without -----------------------------------------------------------
# Operations of one filter pair: 7 fused multiply-adds of the exponent's position and normal products,
# one exponential, 4 accumulations. A traced vertex: about 40 box and 8 triangle tests for its two rays.
PAIR_FLOPS, VERTEX_FLOPS = 21.0, 2.0 * (40 * 12 + 8 * 50)


def _mlp_flops(layers, width=64, inp=64, out=3):
    return 2.0 * (inp * width + (layers - 1) * width * width + width * out)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("filter", "filter_depth"):
        n = c["width"] * c["height"] * c["spp"] * c["depths"]
        extra = 24 if kind == "filter_depth" else 0
        return {"bytes": n * (52.0 + 12.0 + extra), "flops": _pairs(c) * PAIR_FLOPS}
    if kind in ("render_screen", "render_ref"):
        vertices = c["width"] * c["height"] * c["branch"] * (c["depth"] + 1)
        film = c["width"] * c["height"] * 48.0
        if kind == "render_screen":
            pairs = vertices * c["branch"] * (2 * c["radius"] + 1) ** 2
            return {"bytes": vertices * 64.0 + film, "flops": pairs * PAIR_FLOPS + vertices * VERTEX_FLOPS}
        per = c["reuse"] * (c["reuse"] if c["smis"] else 1) * 8.0
        return {"bytes": vertices * 132.0 + film, "flops": vertices * (VERTEX_FLOPS + per)}
    if kind == "adjoint":
        n = c["width"] * c["height"] * c["spp"]
        return {"bytes": n * 64.0 + c["width"] * c["height"] * 12.0, "flops": n * c["spp"] * (2 * c["radius"] + 1) ** 2 * 2 * PAIR_FLOPS}
    if kind == "nrc_train":
        np_ = c["layers"] * 4096 + 192
        return {"bytes": c["iters"] * (c["batch"] * 56.0 + np_ * 40.0), "flops": c["iters"] * c["batch"] * (3 * _mlp_flops(c["layers"]) - 2 * 64 * 64)}
    if kind == "nrc_infer":
        return {"bytes": c["rows"] * 56.0, "flops": c["rows"] * _mlp_flops(c["layers"])}
    fwd = _mlp_flops(5, GRID_WIDTH, GRID_ENC)
    table = GRID_LEVELS * 8 * 8.0  # FP16 corner entries of one row
    if kind == "grid_frame":
        q = c["width"] * c["height"]
        return {"bytes": q * (4.0 * (20 + GRID_DEPTH) + 12 + 4) + c["batch"] * (4.0 * (20 + GRID_DEPTH) + 12 + 3 * table), "flops": q * fwd + c["batch"] * 3 * fwd}
    if kind == "grid_gradient":
        return {"bytes": c["batch"] * (4.0 * (20 + GRID_DEPTH) + 12 + 3 * table) + 41.1e6 * 4, "flops": c["batch"] * 3 * fwd}
    inner = [int(v) for v in c["inner"].split(",")]
    level, slots = 1.0, 1.0
    for k in range(c["depth"]):
        level *= inner[k] if k < len(inner) else 1
        slots += level
    slots *= c["width"] * c["height"] * c["repeats"]
    return {"bytes": slots * 100.0, "flops": slots * VERTEX_FLOPS}


# ---- the same in 64 bits ---------------------------------------------------------------------
def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "filter":
        planes, valid = _records(c, _gen(seed))
        n, budget, child, out = c["width"] * c["height"] * c["spp"], 6e10, None, [None] * c["depths"]
        for d in range(c["depths"] - 1, -1, -1):  # the deepest depths, as many as the time allows
            budget -= _pairs(c) / c["depths"]
            if budget < 0:
                break
            f = _exact_filter(c, planes.reshape(12, c["depths"], n)[:, d], valid.reshape(c["depths"], n)[d], child)
            out[d] = child = _exact_ramp(f) * (valid.reshape(c["depths"], n)[d] != 0) if c["style"] and d == min(1, c["depths"] - 1) else f
        return None if out[-1] is None else out
    if kind == "filter_depth":
        if _pairs(c) > 6e10:
            return None
        planes, valid = _records(c, _gen(seed))
        child = torch.exp(torch.randn((3, planes.shape[1]), generator=_gen(seed + 1), device=DEV) - 1.5).double()
        f = _exact_filter(c, planes, valid, child)
        return [_exact_ramp(f) * (valid != 0) if c["style"] else f, f]
    if kind == "adjoint":
        return [_exact_adjoint(c, seed)]
    if kind == "nrc_infer":
        x, _ = _cache_rows(c["rows"], seed)
        p = torch.from_numpy(_mlp_params(c["layers"], seed)).to(DEV).double()
        return [torch.cat([_exact_mlp(p, b.double(), c["layers"]) for b in x.split(1 << 18)])]
    if kind == "grid_gradient":
        return _exact_grid_gradient(c, seed)
    return None  # Monte Carlo renders and trained networks: what they return depends on the sampler's draws


def _exact_ramp(f):
    s, th, col = RAMP
    lum = (f.clamp(0, 1e5) * torch.tensor([[0.2126], [0.7152], [0.0722]], device=DEV, dtype=torch.float64)).sum(0)
    out, prev = torch.zeros_like(f), torch.zeros((3, 1), device=DEV, dtype=torch.float64)
    for t, cc in zip(np.float32(th).tolist(), np.float32(col).tolist()):
        cc = torch.tensor(cc, device=DEV, dtype=torch.float64)[:, None]
        out += torch.sigmoid(s * (lum - t)) * (cc - prev)
        prev = cc
    return out


def _windows(h, w, r):
    for dy in range(-r, r + 1):
        ys, yc = slice(max(0, -dy), min(h, h - dy)), slice(max(0, dy), min(h, h + dy))
        for dx in range(-r, r + 1):
            xs, xc = slice(max(0, -dx), min(w, w - dx)), slice(max(0, dx), min(w, w + dx))
            if ys.stop > ys.start and xs.stop > xs.start:
                yield dx, dy, (ys, xs), (yc, xc)


def _pair_weights(pos, nrm, ok, q, k, dx, dy, spix, spos, snrm):
    """Weights of one window offset, [rows, columns, query sample, candidate sample], and the two squared distances."""
    d2 = sum((pos[i][q][..., :, None] - pos[i][k][..., None, :]) ** 2 for i in range(3))
    nn = sum(nrm[i][q][..., :, None] * nrm[i][k][..., None, :] for i in range(3))
    rho = (dx * dx + dy * dy) / (2 * spix * spix) if spix > 0 else 0.0
    w = torch.exp(-d2 / (2 * spos * spos) - (1 - nn) / (snrm * snrm) - rho)
    return w * ok[k][..., None, :], d2, nn


def _exact_filter(c, planes, valid, child):
    h, w, s = c["height"], c["width"], c["spp"]
    p = planes.double().reshape(12, h, w, s)
    inc = p[6:9] + (p[9:12] * child.reshape(3, h, w, s) if child is not None else 0)
    ok = (valid != 0).double().reshape(h, w, s)
    spos, snrm = float(np.float32(c["sigma_pos"])), float(np.float32(c["sigma_nrm"]))
    acc = torch.zeros((4, h, w, s), device=DEV, dtype=torch.float64)
    for dx, dy, q, k in _windows(h, w, c["radius"]):
        wt, _, _ = _pair_weights(p[0:3], p[3:6], ok, q, k, dx, dy, c["sigma_pixel"], spos, snrm)
        acc[0][q] += wt.sum(-1)
        for i in range(3):
            acc[1 + i][q] += (wt * inc[i][k][..., None, :]).sum(-1)
    return torch.where(ok > 0, acc[1:] / acc[0], torch.zeros((), device=DEV, dtype=torch.float64)).reshape(3, -1)


def _exact_adjoint(c, seed):
    h, w, s, steps = c["height"], c["width"], c["spp"], c["steps"]
    planes, valid, child = _surface_records(c, _gen(seed))
    prm = torch.from_numpy(_adjoint_params(c, seed)).to(DEV).double()
    target = (0.2 + 0.6 * torch.rand((h, w, 3), generator=_gen(seed + 1), device=DEV)).double()
    spix, spos, snrm = (float(v) for v in prm[33:36])
    p = planes.double().reshape(12, h, w, s)
    inc = p[6:9] + p[9:12] * child.double().reshape(3, h, w, s)
    ok = (valid != 0).double().reshape(h, w, s)
    acc = torch.zeros((4, h, w, s), device=DEV, dtype=torch.float64)
    for dx, dy, q, k in _windows(h, w, c["radius"]):
        wt, _, _ = _pair_weights(p[0:3], p[3:6], ok, q, k, dx, dy, spix, spos, snrm)
        acc[0][q] += wt.sum(-1)
        for i in range(3):
            acc[1 + i][q] += (wt * inc[i][k][..., None, :]).sum(-1)
    wsum = torch.where(ok > 0, acc[0], 1.0)
    f = (acc[1:] / wsum * ok).requires_grad_(True)
    free = prm[:33].clone().requires_grad_(True)
    lum = (f.clamp(0, 1e5) * torch.tensor([0.2126, 0.7152, 0.0722], device=DEV, dtype=torch.float64)[:, None, None, None]).sum(0)
    out, prev = 0.0, torch.zeros(3, device=DEV, dtype=torch.float64)
    for k in range(steps):
        cc = free[9 + 3 * k:12 + 3 * k]
        out = out + torch.sigmoid(free[0] * (lum - free[1 + k])) * (cc - prev)[:, None, None, None]
        prev = cc
    img = (out * ok).mean(-1).permute(1, 2, 0)
    ((img - target) ** 2).sum().backward()
    df = f.grad * ok  # by the filtered radiance; the bandwidths follow by the chain rule through the weights
    fv, bw = f.detach(), torch.zeros(3, device=DEV, dtype=torch.float64)
    for dx, dy, q, k in _windows(h, w, c["radius"]):
        wt, d2, nn = _pair_weights(p[0:3], p[3:6], ok, q, k, dx, dy, spix, spos, snrm)
        e = sum(df[i][q][..., :, None] * (inc[i][k][..., None, :] - fv[i][q][..., :, None]) for i in range(3))
        e = e * wt / wsum[q][..., :, None]
        bw[0] += e.sum() * (dx * dx + dy * dy) / spix ** 3
        bw[1] += (e * d2).sum() / spos ** 3
        bw[2] += (e * (1 - nn)).sum() * 2 / snrm ** 3
    return torch.cat([free.grad, bw])


def _exact_mlp(p, x, layers):
    cols = []
    for d, f in enumerate((4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 2)):
        for k in range(f):
            a = math.pi * x[:, d] * 2.0 ** k
            cols += [torch.sin(a), torch.cos(a)]
    hid = torch.stack(cols, 1)
    for n in range(layers):
        hid = (hid @ p[n * 4096:(n + 1) * 4096].reshape(64, 64).t()).clamp_min(0)
    return hid @ p[layers * 4096:].reshape(3, 64).t()


def _exact_grid_gradient(c, seed):
    """Loss and gradient of the hash-grid network (22 levels of 4 features, one-blob of 7 inputs, identity, 5 x 128)."""
    x, t = _path_rows(c["batch"], seed)
    par = _grid_params(seed).double().requires_grad_(True)
    shapes = [(GRID_WIDTH, GRID_ENC)] + [(GRID_WIDTH, GRID_WIDTH)] * 4 + [(3, GRID_WIDTH)]
    mats, at = [], 0
    for a, b in shapes:
        mats.append(par[at:at + a * b].reshape(a, b))
        at += a * b
    cols, x3 = [], x[:, :3].clamp(0, 1)
    for scale, res, size in _grid_levels():
        tab = par[at:at + size * 4].reshape(size, 4)
        at += size * 4
        u = (x3.double() * scale + 0.5).float()  # the cell is found in 32 bits: the finest levels' scales exceed its 24 digits
        c0 = u.floor()
        wt, c0 = (u - c0).double(), c0.long()
        feat = 0.0
        for k in range(8):
            o = [(k >> i) & 1 for i in range(3)]
            cc = [c0[:, i] + o[i] for i in range(3)]
            if res ** 3 <= size:
                idx = (cc[0] + cc[1] * res + cc[2] * res * res) % size
            else:
                idx = (cc[0] ^ ((cc[1] * 2654435761) & 0xFFFFFFFF) ^ ((cc[2] * 805459861) & 0xFFFFFFFF)) % size
            kw = 1.0
            for i in range(3):
                kw = kw * (wt[:, i] if o[i] else 1 - wt[:, i])
            feat = feat + kw[:, None] * tab[idx]
        cols.append(feat)
    edges = torch.arange(5, device=DEV, dtype=torch.float64) / 4
    cdf = 0.5 * (1 + torch.erf((edges - x[:, 3:10].double()[..., None]) / (0.25 * math.sqrt(2.0))))
    cols += [(cdf[..., 1:] - cdf[..., :-1]).reshape(x.shape[0], -1), x[:, 10:].double()]
    hid = torch.cat(cols, 1)
    hid = torch.nn.functional.pad(hid, (0, GRID_ENC - hid.shape[1]))
    for m in mats[:-1]:
        hid = (hid @ m.t()).clamp_min(0)
    pred = hid @ mats[-1].t()
    loss = ((pred - t.double()) ** 2 / (pred.detach() ** 2 + 0.01)).mean()
    loss.backward()
    return [loss.detach(), par.grad]
