"""Coarse proposals over bands of one radius and a little more, where the coarse band is the search's
own: a particle's pick is formed, and does not depend on its neighbours in the batch (whose windows
samples beyond the band would read)."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu
F = ("theta", "phi", "omega", "x", "y", "pr")


@pytest.mark.parametrize("interp", ["trilinear", "gaussian"])
@pytest.mark.parametrize("r0,R", [(25, 25), (20, 21), (5, 5), (4, 12)])
def test_pick_is_the_particles_own(built, r0, R, interp):
    import cryoim_gb300 as ci
    p0, vol, tmpl, timgs, imgs, parts, truth = small_case(P=3, T=2)
    p = ci.default_params(64, apix=4.0, searchstep=10.0, ampwg=0.07, imgmask=120.0)
    p.min_r, p.max_r = r0, R
    kw = dict(origin_max=1.0, origin_step=0.5, topk=16, nbr=1, pick=1)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        if interp != "trilinear":
            ctx.set_interpolation(interp, 0.6)
        all3 = parts.copy()
        ctx.contract_search(imgs, all3, coarse=4, **kw)
        assert np.all(np.isfinite(all3["pr"])) and np.all(all3["pr"] > 0)
        for i in range(len(parts)):
            one = parts[i:i + 1].copy()
            ctx.contract_search(imgs[i:i + 1], one, coarse=4, **kw)
            for f in F:
                assert one[f][0] == all3[f][i], (i, f)
