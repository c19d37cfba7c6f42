"""A view's omegas shared by several blocks (one particle, few views) against a block a view (a batch):
the same terms per line, the lines' sums in FP32 in other groups (60 partials: 60 x 2^-24)."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [4.0, 5.0, 7.5, 11.0, 20.0])
def test_one_particle_scores_as_in_a_batch(built, step):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=3, step=step)
    many, q = np.tile(imgs, (60, 1, 1)), np.tile(parts, 60)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        rows = ctx.globesearch(many, q, want_pr_array=True)
        for i in (0, 1):
            one = parts[i:i + 1].copy()
            r = ctx.globesearch(imgs[i:i + 1], one, want_pr_array=True)
            np.testing.assert_allclose(r[0], rows[i], rtol=60 * 2.0 ** -24)
            np.testing.assert_allclose(one["pr"], q["pr"][i:i + 1], rtol=60 * 2.0 ** -24)
