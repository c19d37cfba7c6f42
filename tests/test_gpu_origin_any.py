"""Origin grids of more functions than the register kernels hold: every candidate's correlation and origin
against FP64 at its orientation, at the edges of the sums held at a time (16 pairs of x: 31, 32, 33, 65
origins an axis), with one and two shares of K, with the functions in one and in several chunks, with the
table of q too large for shared memory and with the maxima of a list too large for it; and no more
time than the rows that they add."""
import time

import numpy as np
import pytest

from _data import small_case
from test_gpu_contract import cc_fp64, map_cube_full

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_res,step,omax,ostep,form", [
    (12.0, 4.0, 5.0, 0.5, {}), (12.0, 4.0, 7.5, 0.5, {}), (12.0, 4.8, 15.5, 1.0, {}), (12.0, 4.0, 16.0, 1.0, {}),
    (12.0, 4.0, 16.0, 0.5, dict(precision="fp8")),
    (8.6, 4.0, 16.0, 0.5, {}), (8.6, 4.8, 12.0, 0.5, {}),              # several chunks
    (12.0, 4.0, 7.5, 0.5, dict(coarse=3)), (12.0, 4.8, 16.0, 1.0, dict(coarse=3, centred_origins=True)),
    (8.6, 4.0, 20.0, 0.5, dict(coarse=2)), (12.0, 4.0, 7.0, 0.5, dict(coarse=3, precision="fp8")),
    (12.0, 6.0, 20.0, 0.125, dict(coarse=2)), (12.0, 6.0, 20.0, 0.125, {}),  # q's table where it is
    (12.0, 6.0, 2.0, 1 / 64, dict(coarse=2)),   # a fixed layout, 257 origins an axis
    (12.0, 6.0, 8.0, 1 / 32, dict(coarse=2))])  # a list's maxima where the result goes
def test_candidates_against_fp64(built, orc, max_res, step, omax, ostep, form):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=2, step=step, max_res=max_res)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        q = parts.copy()
        cands = ctx.contract_search(imgs, q, origin_max=omax, origin_step=ostep, topk=2, want_cands=True, **form)
    n1 = int(2 * omax / ostep + 0.5) + 1
    vft = map_cube_full(vol)
    # (the bounds of test_gpu_origin_basis.py)
    tol = 5e-2 if form.get("precision") == "fp8" else 2e-2
    for i in range(len(parts)):
        c = cands[i, 0].astype(np.float64)
        cx, cy = (parts["x"][i], parts["y"][i]) if form.get("centred_origins") else (0.0, 0.0)
        gx, gy = cx - omax + ostep * np.arange(n1), cy - omax + ostep * np.arange(n1)
        assert np.abs(gx - c[3]).min() < 1e-4 and np.abs(gy - c[4]).min() < 1e-4
        want = cc_fp64(orc, p, vft, imgs[i], parts[i], c[:5])
        assert abs(c[5] - want) < tol and abs(c[6] - want) < 2e-5
        # some 17 x 17 of the grid's origins, and those around the found one
        near = [(c[3] + a * ostep, c[4] + b * ostep) for a in (-1, 0, 1) for b in (-1, 0, 1)]
        some = [(x, y) for x in gx[::max(1, n1 // 16)] for y in gy[::max(1, n1 // 16)]]
        inside = [(x, y) for x, y in near + some if abs(x - cx) <= omax + 1e-4 and abs(y - cy) <= omax + 1e-4]
        scan = max(cc_fp64(orc, p, vft, imgs[i], parts[i], [*c[:3], x, y]) for x, y in inside)
        assert want > scan - 2 * tol


@pytest.mark.parametrize("form,P", [(dict(), 16), (dict(precision="fp8"), 16), (dict(coarse=8, nbr_best=2), 1)])
def test_no_cliff_past_the_fixed_layouts(built, form, P):
    """+-5 px at maxR 22 of 64 takes 320 rows of A in place of 160 at +-4 px (e4m3: +-6 in place of +-5), and
    has 1.5 times the origins."""
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=4, T=2, step=2.0)
    k = (P + 3) // 4
    many, q = np.tile(imgs, (k, 1, 1))[:P], np.tile(parts, k)[:P]
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)

        def time_of(omax):
            out = []
            for _ in range(12):
                t = time.perf_counter()
                ctx.contract_search(many, q.copy(), origin_max=omax, origin_step=0.5, topk=4, **form)
                out.append(time.perf_counter() - t)
            return np.median(out)

        inside, past = (5.0, 6.0) if "precision" in form else (4.0, 5.0)
        time_of(past), time_of(inside)
        assert time_of(past) < 2.0 * time_of(inside)
