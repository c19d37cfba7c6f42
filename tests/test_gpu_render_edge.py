"""The training renderer at the largest band a box takes (maxR = n / 2 - 2): the frequencies of a smaller band
come out as they do at that band, and training and search run there."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64, 96])
def test_largest_band(built, n):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(n=n, P=3, T=2, step=6.0, max_res=4.0 * n / (n // 2 - 6))
    e = truth[:, :3].astype(np.float32)
    par = np.tile(np.array([1.5, 1.6, 20.0, 0.5, -0.5], np.float32), (3, 1))
    q = ci.default_params(n, apix=p.apix, minRes=60.0, maxRes=12.0, searchstep=6.0, ampwg=0.07, imgmask=4.0 * n)
    r = p.max_r
    assert 4 < r < n // 2 - 2
    with ci.Context(0, p) as ctx:
        want = ctx.learn_render(vol, e, par)
    q.max_r = n // 2 - 2
    with ci.Context(0, q) as ctx:
        got = ctx.learn_render(vol, e, par)
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        st = ctx.learn_train(vol, samples=128, batch=32, seed=3, snr=1.0, df_min=1.0, df_max=3.0, origin_max=2.0)
        assert np.isfinite(st["loss"])
        s = parts.copy()
        ctx.contract_search(imgs, s, origin_max=1.0, origin_step=0.5, topk=4, learned=8)
        assert np.all(s["pr"] < 999)
    ky, hx = np.meshgrid(np.arange(n) - n // 2, np.arange(n) - n // 2, indexing="ij")
    disc = hx ** 2 + ky ** 2 <= r * r
    for a, b in zip(got, want):
        fa, fb = np.fft.fftshift(np.fft.fft2(a))[disc], np.fft.fftshift(np.fft.fft2(b))[disc]
        # the same samples of the same map: FP32 transforms there and back
        assert np.linalg.norm(fa - fb) < 2e-5 * np.linalg.norm(fb)
