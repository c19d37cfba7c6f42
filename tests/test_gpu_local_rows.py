"""Rows of the local grids at every number of samples a thread holds (2, 4, 6, 7, 8), with a last
group of 1, 2 or 3 of the four rows that are normalised together: the BF16 score of every candidate
follows its FP64 score (the bound of the other local tests: BF16 rows of a few hundred samples)."""
import numpy as np
import pytest

from _data import small_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,m", [(48, 12, 2), (64, 21, 3), (96, 29, 1), (96, 32, 2), (96, 34, 4)])
def test_scores_follow_fp64(built, n, R, m):
    import cryoim_gb300 as ci
    p, vol, tmpl, timgs, imgs, parts, truth = small_case(n=n, P=3, T=2, step=4.0, min_res=60.0,
                                                         max_res=4.0 * n / (R + 0.01))
    assert p.max_r in (R, R + 1)
    q = parts.copy()
    rng = np.random.default_rng(R)
    for i, f in enumerate(("theta", "phi", "omega")):
        q[f] = truth[:, i] + 2.0 * rng.integers(-(m - 1), m, size=3)
    with ci.Context(0, p) as ctx:
        ctx.set_reference_map(vol)
        c = ctx.contract_search(imgs, q, origin_max=2.0, origin_step=0.5, topk=16, pick=1, want_cands=True,
                                local_range=2.0 * m, local_step=2.0)
    have = c[:, :, 5] > -1e38  # slots beyond the distinct orientations stay empty
    assert have[:, 0].all() and np.abs(c[:, :, 5] - c[:, :, 6])[have].max() < 2e-2
    assert np.array_equal(q["pr"], np.where(have, c[:, :, 6], -1).max(axis=1).astype(np.float32))
