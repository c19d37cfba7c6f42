"""The search's paired omegas against the same omegas from their own samples (cryoim_prscore_omega) in large
boxes, where positions round more: white noise, a ring, and lattice peaks that stand out of their rings.

A term moves by up to 1e-4 of its weight with its sample's position; one within rounding of a cut may count in
one and not in the other, one of some thousand of these bands."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def image(n, kind, rng):
    y, x = np.mgrid[:n, :n] - n // 2
    v = rng.normal(size=(n, n))
    if kind == "ring":
        v = 0.5 * v + 4.0 * np.exp(-((np.hypot(x, y) - 0.25 * n) / (0.03 * n)) ** 2)
    elif kind == "lattice":
        v += 2.0 * np.cos(2 * np.pi * (0.014 * x + 0.009 * y)) + 2.0 * np.cos(2 * np.pi * (0.007 * x - 0.016 * y))
    return v.astype(np.float32)


@pytest.mark.parametrize("n,kind", [(512, "noise"), (1024, "noise"), (1024, "ring"), (1024, "lattice")])
def test_pairs_as_singles(built, orc, n, kind):
    import cryoim_gb300 as ci
    R, step = 24, 10.0
    p = ci.default_params(n, apix=1.0, minRes=n / 4.01, maxRes=n / (R + 0.01), searchstep=step, apply_ctf=0,
                          imgmask=n // 2 - 2.0)
    rng = np.random.default_rng(n)
    tmpl = ci.templates(3)
    tmpl["particle_id"] = np.arange(1, 4)
    tmpl["theta"], tmpl["phi"], tmpl["omega"] = (81.0, 75.0, 88.0), (5.0, -9.0, 14.0), (20.0, 110.0, 250.0)
    timgs = np.stack([image(n, kind, rng) for _ in range(3)])
    parts = ci.particles(1)
    img = image(n, kind, rng)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        nth, nph, nom, V = ctx.search_grid()
        rows = ctx.globesearch(img[None], parts.copy(), want_pr_array=True)[0].reshape(nth + 1, 2 * nph + 1, nom)
        a, b, f = orc.prep_particle(img, 1, p.imgmask_px, 0.0, 0.0, 1, p.min_r, p.max_r, "f64")
        assert nom % 2 == 0
        rel = []
        for it in range(nth + 1):
            for ip in range(2 * nph + 1):
                if rows[it, ip, 0] >= 999:
                    continue
                single = ctx.prscore_omega(a, b, f, None, 69.0 + step * it, step * (ip - nph))
                rel.append(np.abs(rows[it, ip] - single) / single)
    rel = np.array(rel)
    assert rel.size >= 5 * nom and rel.max() < 5e-3 and np.mean(rel < 1e-4) >= 0.98
