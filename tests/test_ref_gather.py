"""The reference-mode filter's gather (128 candidates per step, queue of 32) and its pdf sums of flat diffuse frames
at the sizes where they can go wrong: cells that end inside a step, reservoirs around a warp, groups of
four frames that are or are not all flat. Counts and final draws bit for bit, radiance within the 1e-5 that
FP32 against the FP64 oracle keeps elsewhere."""
import numpy as np
import pytest

from conftest import rel_err
from test_pf_ref import TOL, _gpu, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flat", ["all", "some", "none"])
@pytest.mark.parametrize("reuse", [1, 7, 31, 33, 64])
@pytest.mark.parametrize("n", [1, 5, 127, 130, 900])
def test_gather_and_flat_frames(sty, orc, cuda, n, reuse, flat):
    arr, mats, progs, rng = _setup(sty, n=n, seed=n + reuse, p_active=1.0 if n < 10 else 0.9, p_flags=0.3)
    r = np.random.default_rng(n)
    pick = {"all": np.ones(n, bool), "some": r.random(n) < 0.8, "none": np.zeros(n, bool)}[flat]
    arr["ns"][:, pick] = arr["ng"][:, pick]
    if flat != "none":
        arr["material"][pick] %= 2  # the diffuse ones
    prm = sty.pf_ref.RefParams(depth=1, radius=0.7, reuse=reuse, smis=True, cluster=False)
    st, ref_out, ref_nb, _, ref_rng = orc.pf_ref_filter(arr, prm.c(), mats, progs, 2, rng, in_next=arr["in_next"])
    assert st == 0
    out, nb, _, g = _gpu(sty, arr, mats, progs, rng, prm)
    assert (nb == ref_nb).all() and (g == ref_rng).all()
    act = arr["active"].astype(bool)
    assert rel_err(out[:, act], ref_out[:, act], 1e-4).max() < TOL


@pytest.mark.parametrize("seed", [0, 1])
def test_positions_on_the_radius(sty, orc, cuda, seed):
    """Candidates whose distance rounds to the radius: which side they fall on depends on every rounding of the
    distance, so the counts show a contracted or reordered one."""
    n = 4000
    arr, mats, progs, rng = _setup(sty, n=n, seed=seed, p_flags=0.0, p_active=1.0)
    r = np.random.default_rng(seed)
    c = r.uniform(-0.5, 0.5, (n // 100, 3))
    d = r.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = np.repeat(c, 100, 0) + 0.25 * d * (1 + r.integers(-2, 3, (n, 1)) * 6e-8)
    p[::100] = c
    arr["p"] = np.ascontiguousarray(p.T.astype(np.float32))
    prm = sty.pf_ref.RefParams(depth=1, radius=0.25, reuse=16, smis=False, cluster=False)
    st, _, ref_nb, _, ref_rng = orc.pf_ref_filter(arr, prm.c(), mats, progs, 2, rng, in_next=arr["in_next"])
    assert st == 0
    _, nb, _, g = _gpu(sty, arr, mats, progs, rng, prm)
    assert (nb == ref_nb).all() and (g == ref_rng).all()
