"""The adjoint at bandwidths far from the middle: so wide that a term of the weight vanishes (down to squares that overflow),
where invalid records have to stay invisible and a gradient is 0 and not a NaN; and narrow against the coordinates, where
the filtered radiance and the sums of the gradient have to come from the same rounded weights."""
import numpy as np
import pytest

import oracle
from test_adjoint import _case, _close, _gpu_adjoint, _target


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [2, 4])
@pytest.mark.parametrize("which", [33, 34, 35])
@pytest.mark.parametrize("wide", [1e8, 1e15, 1e20, 1e30])
def test_a_term_switched_off(sty, cuda, wide, which, spp):
    """One bandwidth without effect: its gradient is 0 to within FP32 of the others', which are those of the FP64
    oracle at a bandwidth as good as infinite."""
    W, H, R = 37, 11, 4
    planes, valid, rec, p, pt = _case(sty, W, H, spp, seed=3)
    p[which] = pt[which] = 1e8
    target = _target(oracle, rec, pt, R, W, H)
    loss_ref, ref = oracle.pf_adjoint(rec, 0, R, p, 8, target)
    p[which] = wide
    rs = sty.RecordSet.from_numpy(planes, valid, W, H, spp, 1)
    for fn in ("sty_pf_adjoint", "sty_pf_adjoint_noalloc"):
        loss, g = _gpu_adjoint(sty, rs, R, p, target, fn=fn)
        assert np.isfinite(g).all()
        assert abs(loss - loss_ref) <= 1e-4 * loss_ref
        keep = np.arange(36) != which
        assert _close(g[keep], ref[keep], 1e-4) < 1e-4
        assert abs(g[which]) <= 1e-6 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [1, 2, 4, 8])
@pytest.mark.parametrize("sigma_nrm", [0.05, 0.3])
def test_narrow_against_the_coordinates(sty, cuda, sigma_nrm, spp):
    """A surface 2000 sigma_pos from the origin. Tolerance: differences of nearby coordinates are exact, an exponent of up to 25
    (log2) then carries at most 3 roundings of 2^-24 of it, 5e-6 a weight, and the normal term 2^-24 / sigma_nrm^2 of
    1.44, 4e-5 at 0.05. They are independent over the ~100 to 1000 weights of a query and the ~1000 queries of a sum, so
    4e-6 is 10 times above what is left of them. (Positions scaled before they are subtracted: 2000 2^-24 of
    sigma_pos, 1e-4 a weight, the same for all weights of a record.)"""
    W, H, R = 40, 26, 5
    rng = np.random.default_rng(7)
    y, x, s = np.meshgrid(np.arange(H), np.arange(W), np.arange(spp), indexing="ij")
    jx, jy = (x + rng.random(x.shape)) * 0.01, (y + rng.random(x.shape)) * 0.01
    pos = np.stack([100 + jx, 50 + jy, 30 + 0.02 * np.sin(9 * jx)])
    nrm = np.stack([-0.18 * np.cos(9 * jx), 0.1 * np.sin(7 * jy), np.ones_like(jx)])
    nrm /= np.linalg.norm(nrm, axis=0)
    rad = np.stack([0.4 + 0.3 * np.sin(7 * jx + k) * np.cos(5 * jy) for k in range(3)]) * np.exp(0.3 * rng.normal(size=jx.shape))
    planes = np.concatenate([pos, nrm, rad, np.zeros_like(rad)]).reshape(12, -1).astype(np.float32)
    valid = (rng.random(planes.shape[1]) > 0.03).astype(np.int32)
    rec = sty.pf.host_records(planes, valid, W, H, spp, 1)
    p = np.zeros(36)
    p[0], p[1:9], p[9:33] = 20.0, np.linspace(0.1, 0.7, 8), np.sort(rng.uniform(0.0, 1.0, 24))
    p[33:36] = [3.0, 0.05, sigma_nrm]
    p = p.astype(np.float32).astype(np.float64)
    target = 0.2 + 0.6 * rng.random((H, W, 3))
    loss_ref, ref = oracle.pf_adjoint(rec, 0, R, p, 8, target)
    loss, g = _gpu_adjoint(sty, sty.RecordSet.from_numpy(planes, valid, W, H, spp, 1), R, p, target)
    assert abs(loss - loss_ref) <= 4e-6 * loss_ref
    assert np.linalg.norm(g[:33] - ref[:33]) <= 4e-6 * np.linalg.norm(ref[:33])
    assert _close(g[33:], ref[33:], 1e-4) < 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [1, 2, 4, 8])
def test_invalid_records_are_not_read_into_the_sums(sty, cuda, spp):
    """Other (finite) values in the invalid records change nothing, in all 36 entries; with every record valid they do."""
    W, H, R = 35, 9, 4
    planes, valid, rec, p, pt = _case(sty, W, H, spp, seed=6)
    p[33:36] = [50.0, 20.0, 5.0]  # every record of the window counts
    target = _target(oracle, rec, p * 1.05, R, W, H)
    assert 0 < (valid == 0).sum() < valid.size
    other = planes.copy()
    other[:, valid == 0] = np.random.default_rng(1).uniform(0.1, 3.0, (12, int((valid == 0).sum())))
    for fn in ("sty_pf_adjoint", "sty_pf_adjoint_noalloc"):
        got = [_gpu_adjoint(sty, sty.RecordSet.from_numpy(a, v, W, H, spp, 1), R, p, target, fn=fn)
               for a, v in ((planes, valid), (other, valid), (planes, np.ones_like(valid)))]
        assert got[0][0] == got[1][0] and (got[0][1] == got[1][1]).all()
        assert (got[0][1][33:] != got[2][1][33:]).all()
    loss_ref, ref = oracle.pf_adjoint(rec, 0, R, p, 8, target)
    assert _close(got[0][1], ref, 1e-4) < 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("spp,w,h,bandwidths", [(8, 96, 64, (4.0, 0.05, 0.2)), (8, 96, 64, (4.0, 0.05, 1.0)), (4, 128, 96, (4.0, 0.05, 0.05)),
                                                (4, 128, 96, (4.0, 0.05, 1.0))])
def test_sums_cancel_with_their_own_weights(sty, cuda, spp, w, h, bandwidths):
    """Positions up to 100 sigma_pos from the origin and from each other, so a record has few neighbours and its sums of
    w (in_j - f_i) are small against their terms. With f from the same weights an error of 2^-24 in each leaves 6e-8 of
    a term, 1e-6 of the gradient where the sums are a tenth of their terms; with f from others, of 2^-24 times 100 each, it
    does not cancel. (The image is the forward filter's; at 2 samples its own rounding, through the ramp's slope, is as large
    as that.) Parameters as the kernel takes them, in FP32, and a target away from the image."""
    planes, valid = sty.synth.records(w, h, spp, 1, seed=1)
    rec = sty.pf.host_records(planes, valid, w, h, spp, 1)
    rng = np.random.default_rng(1)
    p = np.zeros(36)
    p[0], p[1:9], p[9:33] = 50.0, np.sort(rng.uniform(0.02, 0.8, 8)), np.sort(rng.uniform(0.0, 1.0, 24))
    p[33:36] = bandwidths
    p = p.astype(np.float32).astype(np.float64)
    target = (0.2 + 0.6 * rng.random((h, w, 3))).astype(np.float32).astype(np.float64)
    loss_ref, ref = oracle.pf_adjoint(rec, 0, 6, p, 8, target)
    loss, g = _gpu_adjoint(sty, sty.RecordSet.from_numpy(planes, valid, w, h, spp, 1), 6, p, target)
    assert np.linalg.norm(g - ref) <= 1e-6 * np.linalg.norm(ref), np.linalg.norm(g - ref) / np.linalg.norm(ref)
