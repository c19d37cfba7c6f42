"""The search's omegas taken in pairs half a turn apart against the same omegas scored one at a
time (the rescoring's scorer at the search's own particle origin): grids whose omegas pair up
over several groups and warps, one with an odd number of omegas, and a single pair.

The scores are sums over thousands of terms whose samples round differently by 2e-5 px: a term
moves by up to 1e-4 of its weight in either direction, the sum by far less than 1e-4 of itself; a
term whose amplitude is within rounding of a cut may count in one and not in the other (one in
the ~1,500 terms of these boxes)."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1.25, 1.6, 4.0, 7.5, 20.0])
def test_rows_match_single_scores(built, step):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=2, T=3, step=step)
    with ci.Context(0, p) as ctx:
        ctx.load_templates(timgs, tmpl)
        ctx.set_reference_map(vol)
        nth, nph, nom, V = ctx.search_grid()
        q = parts.copy()
        rows = ctx.globesearch(imgs, q, want_pr_array=True)
        c = ctx.contract_search(imgs, parts.copy(), origin_max=2.0, topk=64, nbr=1, want_cands=True)
    assert nom == int(360.0 / np.float32(step))
    off = 0
    for i in range(2):
        flat = rows[i].reshape(nth + 1, 2 * nph + 1, nom)
        assert np.isclose(flat[flat < 999].min(), q["pr"][i], rtol=1e-6)
        for th, ph, om, pr in c[i][:, [0, 1, 2, 7]]:
            if pr <= 0:
                continue  # an empty place of the list
            it, ip, io = round((th - 69.0) / step), round(ph / step) + nph, round(om / step)
            off += abs(flat[it, ip, io] - pr) > 1e-4 * pr
            assert abs(flat[it, ip, io] - pr) < 5e-3 * pr
    assert off <= 0.02 * 128 + 1
