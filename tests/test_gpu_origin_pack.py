"""Exhaustive searches over few origins, whose rows of A share a unit of the contraction among particles:
the same bits for every particle alone, in whole and in ragged units, and in several sub-batches; and no more
rows than such a grid has."""
import time

import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step,omax,ostep,form", [
    (4.0, 0.0, 0.5, {}), (4.0, 0.5, 0.5, {}), (4.8, 0.5, 0.5, {}), (4.0, 1.0, 0.5, {}), (4.0, 1.0, 1.0, {}),
    (4.0, 1.5, 0.5, {}), (4.8, 2.0, 1.0, {}), (4.0, 0.0, 0.5, dict(precision="fp8")),
    (4.0, 1.0, 0.5, dict(precision="fp8")), (4.8, 2.0, 0.5, dict(precision="fp8")), (4.0, 2.0, 0.5, dict(coarse=2)),
    (4.8, 1.0, 0.5, dict(coarse=2, centred_origins=True))])
def test_together_as_alone(built, step, omax, ostep, form):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=9, T=2, step=step)
    kw = dict(origin_max=omax, origin_step=ostep, topk=4, nbr_best=2, want_cands=True, **form)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        q1 = parts.copy()
        one = np.concatenate([ctx.contract_search(imgs[i:i + 1], q1[i:i + 1], **kw) for i in range(9)])
        have = one[:, :, 5] > -1e38
        assert have[:, 0].all()
        assert np.abs(one[:, :, 5] - one[:, :, 6])[have].max() < (5e-2 if "precision" in form else 2e-2)
        for P, batch in ((2, 64), (9, 64), (9, 5), (64, 64), (63, 64), (130, 128)):
            ctx.set_batch(batch)
            idx = np.arange(P) * 7 % 9
            q = parts[idx].copy()
            c = ctx.contract_search(imgs[idx], q, **kw)
            assert np.array_equal(c, one[idx]) and np.array_equal(q, q1[idx])


def test_one_origin_costs_less_than_eighty_one(built):
    """64 particles: 2 rows of A each in place of 96."""
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=4, T=2, step=2.0)
    many, q = np.tile(imgs, (16, 1, 1)), np.tile(parts, 16)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)

        def time_of(omax):
            out = []
            for _ in range(12):
                t = time.perf_counter()
                ctx.contract_search(many, q.copy(), origin_max=omax, origin_step=0.5, topk=4, nbr_best=1)
                out.append(time.perf_counter() - t)
            return np.median(out)

        time_of(0.0), time_of(2.0)
        assert time_of(0.0) < 0.8 * time_of(2.0)
