"""The reference-mode filter on tables so small that several of a vertex's 27 cells share a bucket: each of them lists
the bucket's points, so a vertex meets more candidates than there are points. Neighbour counts, cluster ids and
reservoir draws bit for bit against the oracle, radiance within its 1e-5."""
import numpy as np
import pytest

from conftest import rel_err
from test_pf_ref import TOL, _gpu, _setup


def _case(sty, n, reuse, table, cluster=False):
    arr, mats, progs, rng = _setup(sty, n=n, seed=n + table, p_active=0.8, p_flags=0.2)
    prm = sty.pf_ref.RefParams(depth=1, radius=0.6, reuse=reuse, smis=True, cluster=cluster, table_size=table)
    return arr, mats, progs, rng, prm


@pytest.mark.parametrize("n", [20, 130, 900])
def test_candidates_outnumber_the_points(sty, orc, n):
    """What makes the cases below worth running: counts past the number of active vertices, at table size 1
    also past the number of vertices."""
    arr, mats, progs, rng, prm = _case(sty, n, 16, 1)
    st, _, nb, _, _ = orc.pf_ref_filter(arr, prm.c(), mats, progs, 2, rng, in_next=arr["in_next"])
    assert st == 0 and nb.max() > n > arr["active"].sum()


@pytest.mark.gpu
@pytest.mark.parametrize("reuse,cluster", [(1, False), (16, False), (64, False), (16, True), (64, True)])
@pytest.mark.parametrize("table", [1, 2, 7])
@pytest.mark.parametrize("n", [20, 130, 900])
def test_shared_buckets(sty, orc, cuda, n, table, reuse, cluster):
    arr, mats, progs, rng, prm = _case(sty, n, reuse, table, cluster)
    st, ref_out, ref_nb, ref_cid, ref_rng = orc.pf_ref_filter(arr, prm.c(), mats, progs, 2, rng, in_next=arr["in_next"])
    assert st == 0
    out, nb, cid, g = _gpu(sty, arr, mats, progs, rng, prm)
    assert (nb == ref_nb).all() and (g == ref_rng).all()
    if cluster:
        assert (cid == ref_cid).all()
    act = arr["active"].astype(bool)
    assert rel_err(out[:, act], ref_out[:, act], 1e-4).max() < TOL
