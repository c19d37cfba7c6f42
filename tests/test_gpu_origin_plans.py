"""Origin grids in turn: a context holds the bases of its last grids, so that a search that alternates between
some gives each grid's results and takes no longer than one that stays with a grid."""
import time

import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [dict(), dict(precision="fp8"), dict(coarse=8)])
def test_grids_in_turn(built, form):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=2, step=4.0)
    grids = [(2.0, 0.5), (4.0, 0.5), (2.0, 1.0), (1.5, 0.25), (3.0, 1.0), (0.0, 0.5)]
    kw = dict(topk=4, nbr_best=2, want_cands=True, **form)

    def call(ctx, g):
        q = parts.copy()
        c = ctx.contract_search(imgs, q, origin_max=g[0], origin_step=g[1], **kw)
        return q, c

    want = []
    for g in grids:  # a context each
        with ci.Context(0, p) as ctx:
            ctx.load_templates(timgs, tmpl)
            ctx.set_reference_map(vol)
            want.append(call(ctx, g))
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        for k in (0, 1, 2, 3, 4, 5, 0, 5, 1, 4, 2, 3):  # (with the coarse levels' more than are held)
            q, c = call(ctx, grids[k])
            assert np.array_equal(q, want[k][0]) and np.array_equal(c, want[k][1])


def test_two_grids_cost_what_one_does(built):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=2, step=4.0)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)

        def time_of(omaxes, n):
            out = []
            for k in range(n):
                for om in omaxes:
                    t = time.perf_counter()
                    ctx.contract_search(imgs, parts.copy(), origin_max=om, origin_step=0.25, topk=4, coarse=8)
                    out.append(time.perf_counter() - t)
            return np.median(out)

        time_of((6.0, 5.5), 3)
        alone = max(time_of((6.0,), 15), time_of((5.5,), 15))
        turn = time_of((6.0, 5.5), 15)
    # (49 and 45 origins an axis: making either basis is 0.3 ms at the least, 4 ms with a cosine per term)
    assert turn < 1.1 * alone + 2.5e-4, (turn, alone)
