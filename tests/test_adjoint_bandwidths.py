"""The adjoint at bandwidths far from the middle: so wide that a term of the weight vanishes (down to squares that overflow),
where invalid records have to stay invisible and a gradient is 0 and not a NaN."""
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
