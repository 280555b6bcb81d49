"""The adjoint's single sweep at the edges of its 32 x 4 pixel blocks, for each sample count, against the FP64
analytic adjoint of the oracle with the 1e-4 that the repository's other comparisons of the two use."""
import numpy as np
import pytest

import oracle
from test_adjoint import _case, _close, _gpu_adjoint, _target


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [1, 2, 4, 8])
@pytest.mark.parametrize("size,radius", [((1, 1), 0), ((31, 4), 3), ((33, 5), 2), ((64, 9), 5), ((5, 41), 9)])
def test_block_edges(sty, cuda, size, radius, spp):
    W, H = size
    planes, valid, rec, p, pt = _case(sty, W, H, spp, seed=W + H)
    target = _target(oracle, rec, pt, radius, W, H)
    loss_ref, ref = oracle.pf_adjoint(rec, 0, radius, p, 8, target)
    rs = sty.RecordSet.from_numpy(planes, valid, W, H, spp, 1)
    for fn in ("sty_pf_adjoint", "sty_pf_adjoint_noalloc"):
        loss, g = _gpu_adjoint(sty, rs, radius, p, target, fn=fn)
        assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref) + 1e-12
        if np.abs(ref).max() > 0:
            assert _close(g, ref, 1e-4) < 1e-4, (fn, _close(g, ref, 1e-4))


@pytest.mark.gpu
def test_invalid_records_weigh_nothing_at_any_bandwidth(sty, cuda):
    """Bandwidths so wide that no distance could hide a record: only its validity can."""
    W, H, R = 37, 11, 4
    planes, valid, rec, p, pt = _case(sty, W, H, 4, seed=3)
    p[33:36] = [1e6, 1e6, 1e3]
    pt[33:36] = [1e6, 1e6, 1e3]
    target = _target(oracle, rec, pt, R, W, H)
    loss_ref, ref = oracle.pf_adjoint(rec, 0, R, p, 8, target)
    loss, g = _gpu_adjoint(sty, sty.RecordSet.from_numpy(planes, valid, W, H, 4, 1), R, p, target)
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    assert _close(g[:33], ref[:33], 1e-4) < 1e-4
    assert np.isfinite(g).all()
