"""The listed orientations' maxima over the origins with the origins of a tile shared by several blocks (a
few particles) and by one (a batch): each origin's maximum is one block's either way, so results are
the same bits."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("origin_max,precision", [(0.0, "bf16"), (1.0, "bf16"), (2.0, "fp8"), (4.0, "bf16"), (5.5, "fp8")])
def test_few_particles_as_in_a_batch(built, origin_max, precision):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=4, T=2, step=4.0)
    many, q = np.tile(imgs, (40, 1, 1)), np.tile(parts, 40)
    kw = dict(origin_max=origin_max, origin_step=0.5, topk=8, coarse=8, nbr_best=2, precision=precision, want_cands=True)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        ctx.set_batch(160)
        c = ctx.contract_search(many, q, **kw)
        for n in (1, 3, 4):
            some = parts[:n].copy()
            d = ctx.contract_search(imgs[:n], some, **kw)
            assert np.array_equal(d[:, :, :6], c[:n, :, :6])
            assert np.array_equal(some, q[:n])
