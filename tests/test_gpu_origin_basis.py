"""The contraction over the origin grid's basis: every candidate's correlation and origin
against an FP64 scan of the whole origin grid at its orientation, for origin grids of one
origin, even, odd and many origins per axis, ranges beyond the register kernels, grids with and
without a half turn to share, both operand types, exhaustive and listed."""
import numpy as np
import pytest

from _data import small_case
from test_gpu_contract import cc_fp64, map_cube_full

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step,omax,ostep,form", [
    (4.0, 2.0, 0.5, {}), (4.0, 0.0, 0.5, {}), (4.0, 2.5, 1.0, {}), (4.8, 2.0, 0.5, {}), (4.0, 7.0, 0.5, {}),
    (4.0, 2.0, 0.5, dict(precision="fp8")), (4.8, 2.5, 0.5, dict(precision="fp8")),
    (4.0, 2.0, 0.5, dict(coarse=8)), (4.8, 3.0, 0.5, dict(coarse=8, centred_origins=True)),
    (4.0, 7.0, 0.5, dict(coarse=4, precision="fp8"))])
def test_candidates_against_a_scan(built, orc, step, omax, ostep, form):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=3, T=4, step=step)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        q = parts.copy()
        cands = ctx.contract_search(imgs, q, origin_max=omax, origin_step=ostep, topk=4, want_cands=True, **form)
    n1 = int(2 * omax / ostep + 0.5) + 1
    vft = map_cube_full(vol)
    # BF16 operands: 2^-9 each, of products whose absolute sum is at most 1; the sections' texture
    # weights, 2^-9 per axis of differences up to twice the sample; e4m3: 2^-4 each in quadrature
    # over thousands of samples.  The bounds test_gpu_contract.py holds the same scores to.
    tol = 5e-2 if form.get("precision") == "fp8" else 2e-2
    for i in range(len(parts)):
        c = cands[i, 0].astype(np.float64)
        cx, cy = (parts["x"][i], parts["y"][i]) if form.get("centred_origins") else (0.0, 0.0)
        gx = cx - omax + ostep * np.arange(n1)
        gy = cy - omax + ostep * np.arange(n1)
        assert np.abs(gx - c[3]).min() < 1e-4 and np.abs(gy - c[4]).min() < 1e-4
        sub = slice(None, None, 1 if n1 < 12 else 3)  # (every origin, or every third of a large grid)
        scan = max(cc_fp64(orc, p, vft, imgs[i], parts[i], [*c[:3], x, y]) for x in gx[sub] for y in gy[sub])
        want = cc_fp64(orc, p, vft, imgs[i], parts[i], c[:5])
        assert abs(c[5] - want) < tol and abs(c[6] - want) < 2e-5
        assert want > scan - 2 * tol
