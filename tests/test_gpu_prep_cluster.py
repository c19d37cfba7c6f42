"""Preparation of images by 1, 2, 4 or 8 blocks to an image (by their number and side): a particle's
result does not depend on how many images are prepared together by more than the order of the
image sums."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 50, 64, 130])
def test_batches_of_all_sizes(built, n):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(n=n, P=2, T=2, max_res=4.0 * 4.0)
    many, q = np.tile(imgs, (100, 1, 1)), np.tile(parts, 100)
    q["theta"], q["phi"], q["omega"] = (np.tile(truth[:, i], 100) for i in range(3))
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_batch(200)
        want = None
        for B in (200, 1, 2, 19, 20, 38, 39, 76, 77):
            some = q[:B].copy()
            ctx.refine(many[:B], some)
            if want is None:
                want = some
            for f in ("theta", "phi", "omega", "x", "y", "pr"):
                # a residual is a mean of angles over amplitudes above a cut: 2e-5 is the FP32 bound of the
                # same terms from images whose mean and deviation round alike
                np.testing.assert_allclose(some[f], want[f][:B], rtol=2e-5, atol=2e-5)
