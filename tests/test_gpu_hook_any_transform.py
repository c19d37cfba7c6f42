"""cryoim_prscore_omega takes any transform, as the routine it replaces does: one that is not a real
image's (a half plane weighted, a phase that is not odd) against the oracle, on a grid whose omegas come
in pairs half a turn apart and on one whose do not."""
import numpy as np
import pytest

from _data import small_case
from test_gpu_parity import check_scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [4.0, 4.8])
@pytest.mark.parametrize("kind", ["weight", "phase", "half"])
def test_scores_of_a_transform_without_symmetry(built, orc, step, kind):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(step=step)
    tm, tf = orc.load_templates(timgs, tmpl, p, "f64")
    a, b, f = orc.prep_particle(imgs[0], 1, p.imgmask_px, parts["x"][0], parts["y"][0], 1, p.min_r, p.max_r, "f64")
    ctf = orc.ctf2d(p.fftsize, parts["df1"][0], parts["df2"][0], parts["astigang"][0], p.apix, p.vol, p.cs, p.ampwg,
                    "f64")
    n = p.fftsize
    ky, hx = np.meshgrid(np.arange(n) - n // 2, np.arange(n) - n // 2, indexing="ij")
    if kind == "weight":
        w = 1.0 + 0.4 * np.tanh(hx / 8.0)
    elif kind == "phase":
        w = np.exp(0.5j * np.cos(ky / 6.0))
    else:
        w = np.where(hx >= 0, 1.0, 0.0)
    z = (a + 1j * b) * w
    a, b = np.ascontiguousarray(z.real), np.ascontiguousarray(z.imag)
    tort = np.stack([tmpl["theta"], tmpl["phi"], tmpl["omega"]], 1)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        rel = []
        for th, ph in [(81.0, 8.0), (73.0, -12.0)]:
            want = orc.pr_omega(a, b, f, tm, tort, tf, ctf, p.min_r, p.max_r, p.searchstep, th, ph, fp="f64")
            got = ctx.prscore_omega(a, b, f, ctf, th, ph)
            ok = want < 999
            assert np.array_equal(got < 999, ok) and ok.sum() > 10
            rel.append(np.abs(got[ok] - want[ok]) / want[ok])
        check_scores(np.concatenate(rel))
