"""Particle and template masks from a few pixels of the image to wider than the box, where the inner radius of
the soft edge lies beyond the outer one (which stops at the box's edge): scores against the FP64
oracle with the tolerances of the oracle comparisons of these cases, which allow a term within
rounding of its cut."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("px", [6.0, 20.0, 32.0, 34.5, 35.0, 35.5, 36.0, 64.0])
def test_scores_under_each_mask(built, orc, px):
    import cryoim_gb300 as ci
    p0, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=3)
    n = p0.fftsize
    p = ci.default_params(n, apix=4.0, minRes=60.0, maxRes=12.0, searchstep=6.0, ampwg=0.07, imgmask=4.0 * px)
    assert p.imgmask_px == px and n == 64
    tm, tf = orc.load_templates(timgs, tmpl, p, "f64")
    want = orc.globesearch(p, tm, tf, tmpl, imgs, parts.copy(), want_pr_array=True, fp="f64")
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        got = ctx.globesearch(imgs, parts.copy(), want_pr_array=True)
    assert np.array_equal(got >= 999, want >= 999)
    ok = want < 999
    assert ok.any()
    rel = np.abs(got[ok] - want[ok]) / want[ok]
    assert np.mean(rel < 1e-4) >= 0.995 and rel.max() < 5e-3, (np.mean(rel < 1e-4), rel.max())
