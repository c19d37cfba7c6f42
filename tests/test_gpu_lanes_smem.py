"""Lanes whose launches of one kernel differ in shared memory: the coarse level's products take 96 rows of A
a particle here (+-4 px at 1 px, half the band), the fine level's 160, one particle a pass, so that lanes
set out with both sizes at a time.  Every call succeeds and gives one lane's bits."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


def test_coarse_and_fine_sizes_side_by_side(built):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=4, T=2, step=4.0)
    many, q = np.tile(imgs, (75, 1, 1)), np.tile(parts, 75)
    kw = dict(origin_max=4.0, origin_step=0.5, topk=8, coarse=8, nbr_best=2, want_cands=True)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        ctx.set_batch(1)
        ctx.set_lanes(1)
        one = parts.copy()
        c = ctx.contract_search(imgs, one, **kw)
        ctx.set_lanes(6)
        for _ in range(4):
            qm = q.copy()
            cm = ctx.contract_search(many, qm, **kw)
            assert np.array_equal(qm, np.tile(one, 75))
            assert np.array_equal(cm, np.tile(c, (75, 1, 1)))
