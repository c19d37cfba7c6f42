"""The descent's scoring kernel over batches that take other numbers of blocks per candidate (one
particle to a whole batch) and a band too large for shared memory: each particle ends where it
does alone, and its residual is cal_crosslin_PR's at that end."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctf", [1, 0])
@pytest.mark.parametrize("T", [1, 5])
def test_batches_equal_single_particles(built, T, ctf):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=5, T=T, step=4.0, apply_ctf=ctf)
    q = np.tile(parts, 8)
    rng = np.random.default_rng(3)
    for f in ("theta", "phi", "omega"):
        q[f] += rng.uniform(-2, 2, len(q)).astype(np.float32)
    im = np.tile(imgs, (8, 1, 1))
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        many = q.copy()
        ctx.refine(im, many)
        for n in (1, 2, 13):
            some = q[:n].copy()
            ctx.refine(im[:n], some)
            for f in ("theta", "phi", "omega", "x", "y", "pr"):
                # the same terms, summed to 2^-48 in another order: the same FP32 score
                assert np.array_equal(some[f], many[f][:n]), (n, f)


def test_band_beyond_shared_memory(built, orc):
    """maxR 94 (a 190 x 190 band, 289 KB) takes the other kernel; one cycle from the truth."""
    import cryoim_gb300 as ci
    import synth
    n = 200
    p = ci.default_params(n, apix=2.0, minRes=60.0, maxRes=2.0 * n / 94.01, ampwg=0.07, apply_ctf=1, ncycle=1,
                          imgmask=(n // 2 - 2) * 2.0)
    assert p.max_r == 94
    rng = np.random.default_rng(5)
    vol = synth.phantom(n, 5)
    te = synth.random_asu_orientations(2, rng)
    proj = lambda v, e: synth.project_fourier(v, np.asarray(e))
    tmpl = ci.templates(2)
    tmpl["particle_id"] = [1, 2]
    tmpl["theta"], tmpl["phi"], tmpl["omega"] = te[:, 0], te[:, 1], te[:, 2]
    imgs, parts, truth = synth.make_particles(vol, 2, 6, proj, 2.0, origin_max=2.0, snr=0.0)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(proj(vol, te), tmpl)
        q = parts.copy()
        ctx.refine(imgs, q)
        tm, tf = orc.load_templates(proj(vol, te), tmpl, p, "f64")
        tort = np.stack([tmpl["theta"], tmpl["phi"], tmpl["omega"]], 1)
    for i in range(2):
        a, b, f = orc.prep_particle(imgs[i], 1, p.imgmask_px, parts["x"][i], parts["y"][i], 0, p.min_r, p.max_r, "f64")
        ctf = orc.ctf2d(n, parts["df1"][i], parts["df2"][i], parts["astigang"][i], p.apix, p.vol, p.cs, p.ampwg, "f64")
        want = orc.pr_single(a, b, f, tm, tort, tf, ctf, p.min_r, p.max_r, q["theta"][i], q["phi"][i], q["omega"][i],
                             q["x"][i], q["y"][i], fp="f64")
        assert abs(q["pr"][i] - want) / want < 5e-3  # (the bound test_gpu_parity.py holds scores to)
