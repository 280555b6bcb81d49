"""The grid network's gradient into a caller's buffer of any alignment: the tables' 16-byte atomics need a buffer that
starts on 16 bytes, others go through the network's own. Values beside the buffer stay as they are."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp16", [False, True])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_gradient_into_an_unaligned_buffer(sty, cuda, offset, fp16):
    import torch
    net = sty.nrc.NRC(sty.nrc.grid_config(max_depth=3, batch_size=256, seed=3, fp16=fp16))
    n = int(net.save_params().size)
    rng = np.random.default_rng(offset)
    x = torch.from_numpy(rng.random((256, 23), np.float32)).cuda()
    t = torch.from_numpy(rng.random((256, 3), np.float32) + 0.1).cuda()
    got = []
    for off in (0, offset):
        buf = torch.full((n + 8,), 7.0, device="cuda")
        loss = C.c_float()
        sty.check(sty.lib().sty_nrc_gradient(net.h, 256, x.data_ptr(), t.data_ptr(), buf.data_ptr() + 4 * off, C.byref(loss), None))
        torch.cuda.synchronize()
        assert (buf[:off] == 7).all() and (buf[off + n:] == 7).all()
        got.append((loss.value, buf[off:off + n].double()))
    # the loss and the tables' gradient are sums in any order: of at most 256 terms, 256 2^-24 of them
    assert abs(got[0][0] - got[1][0]) <= 2e-5 * got[0][0]
    assert got[0][1].norm() > 0 and (got[0][1] - got[1][1]).norm() <= 2e-5 * got[0][1].norm()
